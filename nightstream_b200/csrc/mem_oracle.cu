// mem_oracle.cu -- Twist / Shout time-lane sum-check oracles on dense tables.
//
// Every time-lane oracle of crates/neo-memory/src/twist_oracle.rs is a sum over
// the time hypercube of a product of multilinear factors (bitness: χ times a
// weighted sum of b(b-1)).  The reference walks sparse columns pair by pair and
// recomputes χ_{r_cycle} children, eq-bit factors and, for Twist, Val_pre by a
// quadratic sum over all increments at every pair of every round
// (twist_oracle.rs:163-185, 311-379, 684-749).  Here each factor is a dense
// K table in HBM, built once:
//   * χ_{r_cycle} as a table, folded like any factor: folding variable 0 at c
//     multiplies by eq(c, r_0), which is the reference's prefix_eq update;
//   * eq_bit_affine(bit(t), r_b) per address bit: affine in the column, so
//     folding the factor equals the factor of the folded column;
//   * Val_pre(t) = init + Σ_{u<t} inc_terms(u): LT(u, ·) is the multilinear
//     extension of [u < t], so the reference's Σ inc_u·LT(u, point) is the
//     folded exclusive prefix sum (one scan here);
//   * LT(t, r_time) for the val-evaluation oracle.
// A round evaluates Σ_pairs Π_f (f0 + x (f1 - f0)) at x = 0..deg, the pending
// fold of every factor inside the same launch, and interpolates the requested
// points on the host.
// All arithmetic is exact in F_q / K, so values equal the reference's.
#include "internal.cuh"
#include <algorithm>

using gl::K;

namespace {

constexpr int MEM_MAX_DEG = 31;

__device__ __forceinline__ K shfl_xor_km(K a, int o) {
    K r;
    r.re = __shfl_xor_sync(0xffffffffu, a.re, o);
    r.im = __shfl_xor_sync(0xffffffffu, a.im, o);
    return r;
}

// eq(bit, u) = bit·(2u − 1) + (1 − u)   (neo-memory/src/bit_ops.rs:5-9)
__device__ __forceinline__ K eq_bit_affine(K bit, K u) {
    return gl::kadd(gl::kmul(bit, gl::ksub(gl::kdbl(u), gl::kone())), gl::ksub(gl::kone(), u));
}

// columns b = blockIdx.y of [A][len]: out_b[t] = eq_bit_affine(cols_b[t], u_b)
// (out may be cols).  Bound by HBM: 32 bytes an entry, and the columns are read
// where they are instead of copied first (12 columns of 2^16: 12 copies and
// 10.3 us of this kernel, now the latter alone).
__global__ void eqbit_kernel(const K* cols, uint64_t len, const __grid_constant__ KPoint u, K* out) {
    const uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (t >= len) return;
    const uint64_t i = blockIdx.y * len + t;
    out[i] = eq_bit_affine(cols[i], u.x[blockIdx.y]);
}

// inc_terms(t) = has_write(t)·inc(t)·Π_b eq_bit_affine(wa_b(t), r_addr_b)
// (build_inc_terms_at_r_addr, twist_oracle.rs:351-378)
__global__ void inc_terms_kernel(const K* __restrict__ has_w, const K* __restrict__ inc, const K* __restrict__ wa,
                                 uint32_t A, const __grid_constant__ KPoint r_addr, uint64_t len, K* __restrict__ out) {
    uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (t >= len) return;
    K v = has_w[t];
    if (!gl::kiszero(v)) v = gl::kmul(v, inc[t]);
    // rows without a write (most of the time domain) read no address bits
    for (uint32_t b = 0; b < A && !gl::kiszero(v); b++) v = gl::kmul(v, eq_bit_affine(wa[(uint64_t)b * len + t], r_addr.x[b]));
    out[t] = v;
}

// exclusive prefix sum over K in three passes: per-block sums, a scan of the
// block sums (one block), and the per-element scan with the block offset.
constexpr int SCAN_T = 256, SCAN_E = 4, SCAN_BLK = SCAN_T * SCAN_E;

__device__ K block_excl_scan(K v, K* s_warp, K* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    K inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        K n;
        n.re = __shfl_up_sync(0xffffffffu, inc.re, o);
        n.im = __shfl_up_sync(0xffffffffu, inc.im, o);
        if (lane >= o) inc = gl::kadd(inc, n);
    }
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        const int nw = blockDim.x >> 5;
        K w = lane < nw ? s_warp[lane] : gl::kzero();
        K wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            K n;
            n.re = __shfl_up_sync(0xffffffffu, wi.re, o);
            n.im = __shfl_up_sync(0xffffffffu, wi.im, o);
            if (lane >= o) wi = gl::kadd(wi, n);
        }
        if (lane < nw) s_warp[lane] = gl::ksub(wi, w);  // exclusive warp offsets
        if (lane == nw - 1) *total = wi;
    }
    __syncthreads();
    K r = gl::kadd(s_warp[warp], gl::ksub(inc, v));
    __syncthreads();
    return r;
}

__global__ void __launch_bounds__(SCAN_T) scan_sums_kernel(const K* __restrict__ in, uint64_t len, K* __restrict__ sums) {
    __shared__ K s_warp[32];
    __shared__ K s_tot;
    uint64_t base = blockIdx.x * (uint64_t)SCAN_BLK + threadIdx.x * SCAN_E;
    K v = gl::kzero();
#pragma unroll
    for (int e = 0; e < SCAN_E; e++)
        if (base + e < len) v = gl::kadd(v, in[base + e]);
    block_excl_scan(v, s_warp, &s_tot);
    if (threadIdx.x == 0) sums[blockIdx.x] = s_tot;
}

// one block scans up to SCAN_T * chunk block sums, in place, exclusive, plus init
__global__ void __launch_bounds__(SCAN_T) scan_top_kernel(K* __restrict__ sums, uint32_t n, K init) {
    __shared__ K s_warp[32];
    __shared__ K s_tot;
    K carry = init;
    for (uint32_t base = 0; base < n; base += SCAN_T) {
        uint32_t i = base + threadIdx.x;
        K v = i < n ? sums[i] : gl::kzero();
        K ex = block_excl_scan(v, s_warp, &s_tot);
        if (i < n) sums[i] = gl::kadd(carry, ex);
        carry = gl::kadd(carry, s_tot);
        __syncthreads();
    }
}

// out = prefix(in) combined per kind:
//   combine 0: out = VP                      (plain exclusive prefix + init)
//   combine 1: out = VP − a                  (read check:  Val_pre − rv)
//   combine 2: out = a − VP − b              (write check: wv − Val_pre − inc)
__global__ void __launch_bounds__(SCAN_T) scan_final_kernel(const K* __restrict__ in, uint64_t len,
                                                            const K* __restrict__ offs, int combine,
                                                            const K* __restrict__ a, const K* __restrict__ b,
                                                            K* __restrict__ out) {
    __shared__ K s_warp[32];
    __shared__ K s_tot;
    uint64_t base = blockIdx.x * (uint64_t)SCAN_BLK + threadIdx.x * SCAN_E;
    K v[SCAN_E];
    K s = gl::kzero();
#pragma unroll
    for (int e = 0; e < SCAN_E; e++) {
        v[e] = base + e < len ? in[base + e] : gl::kzero();
        s = gl::kadd(s, v[e]);
    }
    K run = gl::kadd(offs[blockIdx.x], block_excl_scan(s, s_warp, &s_tot));
#pragma unroll
    for (int e = 0; e < SCAN_E; e++) {
        uint64_t t = base + e;
        if (t < len) {
            K o = run;
            if (combine == 1) o = gl::ksub(run, a[t]);
            else if (combine == 2) o = gl::ksub(gl::ksub(a[t], run), b[t]);
            out[t] = o;
        }
        run = gl::kadd(run, v[e]);
    }
}

// LT(t, r) for Boolean t (twist_oracle.rs:320-334): from the top bit down,
// acc += suffix r_i where t_i = 0, suffix *= chi_i.  The low 8 bits' (acc, suffix = 1)
// is a thread's, the high bits' a warp leader's, and LT = acc_hi + suffix_hi acc_lo
// (2^18 entries: 51 us with every bit in every thread, now 9).
__device__ __forceinline__ void lt_bits(const KPoint& r, int hi, int lo, uint64_t t, K& acc, K& suffix) {
    acc = gl::kzero();
    suffix = gl::kone();
#pragma unroll 1
    for (int i = hi - 1; i >= lo; i--) {
        const K x = gl::kmul(r.x[i], suffix);
        if (((t >> i) & 1) == 0) {
            acc = gl::kadd(acc, x);
            suffix = gl::ksub(suffix, x);
        } else {
            suffix = x;
        }
    }
}
constexpr uint32_t LT_HIGH = 8;
__global__ void __launch_bounds__(256) lt_table_kernel(const __grid_constant__ KPoint r, uint32_t ell, K* __restrict__ out) {
    __shared__ K s_acc[LT_HIGH], s_suf[LT_HIGH];
    const uint32_t low = min(ell, 8u), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t n_hi = 1ull << (ell - low), h0 = blockIdx.x * (uint64_t)LT_HIGH;
    K acc, suffix;
    if (lane == 0) {
        lt_bits(r, (int)ell, (int)low, (h0 + warp) << low, acc, suffix);
        s_acc[warp] = acc;
        s_suf[warp] = suffix;
    }
    lt_bits(r, (int)low, 0, threadIdx.x, acc, suffix);
    __syncthreads();
    if (threadIdx.x >> low) return;
#pragma unroll
    for (uint32_t v = 0; v < LT_HIGH; v++)
        if (h0 + v < n_hi) out[((h0 + v) << low) + threadIdx.x] = gl::kadd(s_acc[v], gl::kmul(s_suf[v], acc));
}

// fold every factor on variable 0: dst[f][p] = src[f][2p] + r (src[f][2p+1] − src[f][2p])
// (host, unless null: page-locked copy of the last entries, one per factor)
__global__ void mem_fold_kernel(const K* __restrict__ src, uint64_t src_len, K* __restrict__ dst, uint32_t nf, K r,
                                K* host) {
    const uint64_t half = src_len >> 1;
    uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i >= half * nf) return;
    uint64_t f = i / half, p = i - f * half;
    const K* s = src + f * src_len + 2 * p;
    const K v = gl::klerp(s[0], s[1], r);
    dst[f * half + p] = v;
    if (host) host[f] = v;
}

// vals[x] = Σ_b partials[x][b]; one block per x
__global__ void __launch_bounds__(256) mem_reduce_kernel(const K* __restrict__ partials, uint32_t nblocks,
                                                         K* __restrict__ vals) {
    __shared__ K s_red[8];
    const uint32_t x = blockIdx.x;
    K v = gl::kzero();
    for (uint32_t b = threadIdx.x; b < nblocks; b += blockDim.x) v = gl::kadd(v, partials[(uint64_t)x * nblocks + b]);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = gl::kadd(v, shfl_xor_km(v, o));
    if (lane == 0) s_red[warp] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        K s = gl::kzero();
        for (int w = 0; w < 8; w++) s = gl::kadd(s, s_red[w]);
        vals[x] = s;
    }
}

// AddressLookupOracle weight table (twist_oracle.rs:1671-1724):
// w[addr(t)] += χ_{r_cycle}(t)·has_lookup(t), addr from bit columns equal to 1.
// Exact order-free accumulation: each u64 component is summed with a 64-bit
// atomic and its carries are counted separately (sum = lo + 2^64·carries).
__global__ void addr_weights_kernel(const K* __restrict__ chi, const K* __restrict__ has, const K* __restrict__ bits,
                                    uint32_t A, uint64_t len, unsigned long long* __restrict__ lo,
                                    unsigned long long* __restrict__ carry) {
    uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (t >= len) return;
    K g = has[t];
    if (gl::kiszero(g)) return;
    K wt = gl::kmul(chi[t], g);
    if (gl::kiszero(wt)) return;
    uint64_t addr = 0;
    for (uint32_t b = 0; b < A; b++) {
        K v = bits[(uint64_t)b * len + t];
        if (v.re == 1 && v.im == 0) addr |= 1ULL << b;
    }
    unsigned long long o = atomicAdd(&lo[2 * addr], (unsigned long long)wt.re);
    if (o + wt.re < o) atomicAdd(&carry[2 * addr], 1ULL);
    o = atomicAdd(&lo[2 * addr + 1], (unsigned long long)wt.im);
    if (o + wt.im < o) atomicAdd(&carry[2 * addr + 1], 1ULL);
}

__global__ void addr_weights_finish_kernel(const unsigned long long* __restrict__ lo,
                                           const unsigned long long* __restrict__ carry, uint64_t n, K* __restrict__ w) {
    uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    // lo + carry·2^64 with 2^64 = 2^32 − 1 (mod q)
    uint64_t re = gl::add(gl::canon(lo[2 * i]), gl::mul(gl::canon(carry[2 * i]), GL_EPS));
    uint64_t im = gl::add(gl::canon(lo[2 * i + 1]), gl::mul(gl::canon(carry[2 * i + 1]), GL_EPS));
    w[i] = gl::kmk(re, im);
}

// claim = Σ_a table[a]·w[a] (block partials, reduced by mem_reduce_kernel)
__global__ void __launch_bounds__(256) dot_kernel(const K* __restrict__ a, const K* __restrict__ b, uint64_t n,
                                                  K* __restrict__ partials) {
    __shared__ K s_red[8];
    K v = gl::kzero();
    for (uint64_t i = blockIdx.x * 256ULL + threadIdx.x; i < n; i += 256ULL * gridDim.x)
        v = gl::kadd(v, gl::kmul(a[i], b[i]));
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = gl::kadd(v, shfl_xor_km(v, o));
    if (lane == 0) s_red[warp] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        K s = gl::kzero();
        for (int w = 0; w < 8; w++) s = gl::kadd(s, s_red[w]);
        partials[blockIdx.x] = s;
    }
}

// ---- all memory claims of one sum-check round in one launch --------------
// A batched round (the Route-A time claims, the val-eval batch, the address
// pre-time batches) evaluates every claim's round polynomial at x = 0..deg
// before the transcript draws the next challenge.  One kernel folds (the
// pending challenge), evaluates and reduces the tables of up to MULTI_MAX claims
// together; the values land in page-locked memory.
constexpr int MULTI_MAX = 24;
// tiles of a launch below which a pair's factors are shared by more lanes: the active rows
// are often a quarter of all, so three times what two blocks per SM need (2^16 rows, 15
// factors, us per round 1 to 3: 28, 19, 15 with two tiles per SM, 20, 16, 14 with six)
constexpr uint32_t MULTI_TILES = 6 * 148;

struct MultiClaim {
    const K* tab;      // [nf][len] current tables (written by this launch when src is set)
    const K* src;      // a pending fold: [nf][2 len] tables before binding r, else null
    uint64_t len;
    uint32_t nf, npts;
    int bitness;
    const K* w;        // bitness weights [nf - 1]
    K r;               // fold challenge
    uint32_t blk0;     // first block of this claim
    uint32_t part0;    // first partial [npts][nblk]
    uint32_t nblk;     // blocks of this claim (tiles dealt out in turn)
    uint32_t hb;       // 1, 2, 4 or 8: warps per point set
    uint32_t fs;       // lanes that share a pair's factors (1, 2, 4, .. 16)
    uint32_t lpb;      // log2 of the pairs per tile, 32 hb / fs
    uint32_t small;    // few pairs: one block per point (multi_small)
    const uint64_t* vinv;  // null: out gets the values at x = 0..npts-1; else the polynomial's
                           // coefficients, through the npts x npts inverse Vandermonde matrix of 0..npts-1
    K* out;
    unsigned int* ticket;  // the claim's block counter (zero between launches)
    // [MULTI_COPIES][MEM_MAX_DEG + 1][4] sums of the tiles' values, as 32-bit halves of re
    // and im (zero between launches).  Blocks add to them without waiting; with a partial
    // per block and point, the last block read 592 x 17 of them, 10 us of a round.  The
    // blocks take turns over the copies, so that an address sees a quarter of the adds.
    unsigned long long* acc;
};
constexpr uint32_t MULTI_COPIES = 4;

// entries 2p, 2p + 1 of a table in one 32-byte load (read-only data, 32-byte aligned)
__device__ __forceinline__ void ldg_pair(const K* p, K& a, K& b) {
    asm("ld.global.nc.v4.u64 {%0, %1, %2, %3}, [%4];" : "=l"(a.re), "=l"(a.im), "=l"(b.re), "=l"(b.im) : "l"(p));
}
__device__ __forceinline__ K ldg_k(const K* p) {
    const ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2*>(p));
    return gl::kmk(v.x, v.y);
}

// The pending folds of the claims with at least FOLD_PAIRS pairs, as a launch of
// their own: most rows of the first rounds are outside the active trace, where the
// fold is all there is to do and streams (dst[p] = lerp(src[2p], src[2p+1], r),
// 48 bytes an entry; 100 factors of 2^16 entries: 20 us), while the evaluation's
// tiles wait on barriers (116 us with the fold inside).  blockIdx.y, z:
// a factor of one of the claims.
constexpr uint64_t FOLD_PAIRS = 4096;
constexpr uint32_t FOLD_PER = 2;
struct MultiFold {
    int n;
    const K* src[MULTI_MAX];
    K* dst[MULTI_MAX];
    uint64_t half[MULTI_MAX];   // entries of a folded factor
    uint32_t f0[MULTI_MAX + 1]; // first blockIdx.y
    K r[MULTI_MAX];
};
__global__ void __launch_bounds__(256) mem_multi_fold_kernel(const __grid_constant__ MultiFold a) {
    int c = 0;
    const uint32_t y = blockIdx.y + gridDim.y * blockIdx.z;  // a bitness claim may have more than 65535 columns
    if (y >= a.f0[a.n]) return;
    while (y >= a.f0[c + 1]) c++;
    const uint64_t half = a.half[c], f = y - a.f0[c];
    const uint64_t p0 = blockIdx.x * (uint64_t)(256 * FOLD_PER) + threadIdx.x;
    const K* s = a.src[c] + f * 2 * half;
    K* d = a.dst[c] + f * half;
    const K r = a.r[c];
    K lo[FOLD_PER], hi[FOLD_PER];
#pragma unroll
    for (uint32_t e = 0; e < FOLD_PER; e++)
        if (p0 + e * 256 < half) ldg_pair(s + 2 * (p0 + e * 256), lo[e], hi[e]);
#pragma unroll
    for (uint32_t e = 0; e < FOLD_PER; e++)
        if (p0 + e * 256 < half) {
            const K df = gl::ksub(hi[e], lo[e]);
            d[p0 + e * 256] = gl::kiszero(df) ? lo[e] : gl::kadd(lo[e], gl::kmul(df, r));  // constant runs cost no product
        }
}

struct MultiArgs {
    int n;
    MultiClaim c[MULTI_MAX];
    K* partials;
};

__device__ __forceinline__ int multi_claim_of(const MultiArgs& a, uint32_t blk) {
    int c = 0;
    while (c + 1 < a.n && blk >= a.c[c + 1].blk0) c++;
    return c;
}

// Factor f of pair p in the current round: (f0, f1) = the entries 2p, 2p+1; with
// a pending fold lerp(src[4p], src[4p+1], r) and lerp(src[4p+2], src[4p+3], r),
// written to the tables when `own`.
__device__ __forceinline__ void multi_factor(const MultiClaim& c, uint32_t f, uint64_t p, bool own, K& f0, K& f1) {
    if (c.src) {
        const K* o = c.src + (uint64_t)f * (2 * c.len) + 4 * p;
        K o0, o1, o2, o3;
        ldg_pair(o, o0, o1);
        ldg_pair(o + 2, o2, o3);
        f0 = gl::klerp(o0, o1, c.r);
        f1 = gl::klerp(o2, o3, c.r);
        if (own) {
            K* t = const_cast<K*>(c.tab) + (uint64_t)f * c.len + 2 * p;
            t[0] = f0;
            t[1] = f1;
        }
        return;
    }
    ldg_pair(c.tab + (uint64_t)f * c.len + 2 * p, f0, f1);
}

// The round polynomial from its values s_v[0..npts), by the whole block: eight
// lanes per coefficient.  The sum-check driver absorbs coefficients; interpolating
// 16 to 20 points on the host cost 60 to 100 us per claim and round.
__device__ __forceinline__ void multi_coeffs(const MultiClaim& c, const K* s_v) {
    const uint32_t n = c.npts, l = threadIdx.x & 7;
    for (uint32_t d0 = 0; d0 < n; d0 += 32) {
        const uint32_t d = d0 + (threadIdx.x >> 3);
        K acc = gl::kzero();
        if (d < n)
            for (uint32_t x = l; x < n; x += 8) acc = gl::kadd(acc, gl::kscale(s_v[x], __ldg(c.vinv + d * n + x)));
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) acc = gl::kadd(acc, shfl_xor_km(acc, o));
        if (l == 0 && d < n) c.out[d] = acc;
    }
}

// A claim with at most SMALL_PAIRS pairs (its last rounds): one block per point x
// does every pair (coefficients: the last block takes them from all points' values).  fs lanes share a
// pair's factors and multiply (bitness: add) their parts with shuffles: the launch
// is one dependent chain, and a thread walking 15 factors took 22 to 30 us where
// this takes 8.  Block 0 writes the folded tables.
constexpr uint32_t SMALL_PAIRS = 16;
__device__ __noinline__ void multi_small(const MultiClaim& c, uint32_t x, K* s_sum, K* s_v, K* partials) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t fs = c.fs, sub = threadIdx.x & (fs - 1), p = threadIdx.x / fs;
    const bool live = p < (uint32_t)(c.len >> 1);
    auto value = [&](uint32_t f) {  // factor f at x
        K f0, f1;
        multi_factor(c, f, p, x == 0, f0, f1);
        return gl::kadd(f0, gl::kscale_tiny(gl::ksub(f1, f0), x));
    };
    K acc;
    if (!c.bitness) {
        acc = gl::kone();
        if (live) {
#pragma unroll 2
            for (uint32_t f = sub; f < c.nf; f += fs) acc = gl::kmul(acc, value(f));
        }
        for (uint32_t o = 1; o < fs; o <<= 1) acc = gl::kmul(acc, shfl_xor_km(acc, o));
    } else {
        acc = gl::kzero();
        if (live) {
#pragma unroll 2
            for (uint32_t f = 1 + sub; f < c.nf; f += fs) {
                const K v = value(f);
                acc = gl::kadd(acc, gl::kmul(c.w[f - 1], gl::kmul(v, gl::ksub(v, gl::kone()))));
            }
        }
        for (uint32_t o = 1; o < fs; o <<= 1) acc = gl::kadd(acc, shfl_xor_km(acc, o));
        if (live && sub == 0) acc = gl::kmul(acc, value(0));
    }
    K total = live && sub == 0 ? acc : gl::kzero();
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) total = gl::kadd(total, shfl_xor_km(total, o));
    if (lane == 0) s_sum[warp] = total;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; w++) total = gl::kadd(total, s_sum[w]);
        if (!c.vinv) c.out[x] = total;
        else partials[c.part0 + x] = total;
    }
    if (!c.vinv) return;
    __shared__ unsigned int s_last;
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicInc(c.ticket, c.npts - 1) == c.npts - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    if (threadIdx.x < c.npts) {
        const ulonglong2 u = __ldcg(reinterpret_cast<const ulonglong2*>(partials + c.part0 + threadIdx.x));
        s_v[threadIdx.x] = gl::kmk(u.x, u.y);
    }
    __syncthreads();
    multi_coeffs(c, s_v);
}

// Larger claims: a block takes tiles of 32 hb / fs pairs, dealt out in turn so that
// the active rows (a run at the start of the time domain) spread over the blocks.
// Per chunk of factors the block folds the tile once (the folded tables go out, f0
// and f1 - f0 of every pair into shared memory), then warp (x set, pair group)
// multiplies up its points x, x + 8 / hb, .. with fs lanes per pair.  A tile whose
// gate (factor 1: has_lookup / has_read / has_write behind chi; factor 0 where no
// chi leads) is zero on both children of every pair adds nothing at any x; a
// bitness column that is zero adds nothing either.  What bounds it: the arithmetic
// of the active tiles, which is why few pairs are cut into smaller tiles (a Twist
// read check of 15 factors and 16 points with 2^14 of 2^16 rows active: first
// round 43 us, at 2^10 pairs 15; with one thread per pair walking the factors
// at up to 8 points 96 and 44, with 32 pairs a tile throughout 52 and 26).
constexpr uint32_t MF = 512;     // (factor, pair) entries per chunk
constexpr int MPTS = 4;          // points per warp: npts <= 32, 8 / hb point sets
__global__ void __launch_bounds__(256) mem_multi_eval_kernel(const __grid_constant__ MultiArgs a) {
    __shared__ K s_f[2][MF];    // f0, f1 - f0: [factor][pair]
    __shared__ K s_red[8][MPTS];
    __shared__ uint8_t s_on[256];
    __shared__ K s_v[MEM_MAX_DEG + 1];
    const int ci = multi_claim_of(a, blockIdx.x);
    const MultiClaim& c = a.c[ci];
    const uint32_t b = blockIdx.x - c.blk0;
    if (c.small) {
        multi_small(c, b, &s_red[0][0], s_v, a.partials);
        return;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t hb = c.hb, fs = c.fs, lpb = c.lpb, pb = 1u << lpb, fch = MF >> lpb, xstep = 8 / hb;
    const uint32_t sub = lane & (fs - 1), pl = (warp % hb) * (32 / fs) + lane / fs;  // factor share, pair of the tile
    const uint32_t xw = warp / hb;  // first point
    const uint64_t pairs = c.len >> 1, tiles = (pairs + pb - 1) / pb;
    const uint32_t gate = c.nf > 1 ? 1u : 0u;
    K total[MPTS];
#pragma unroll
    for (int k = 0; k < MPTS; k++) total[k] = gl::kzero();
    // with no fold to do, 256 pairs of the block's coming tiles are looked over first
    // (every column of a bitness claim, else the gate) and tiles without any are skipped
    const bool scan = !c.src;
    const uint32_t tps = 256 >> lpb;
    for (uint64_t i = 0; b + i * c.nblk < tiles; i++) {
        const uint64_t tile = b + i * c.nblk;
        if (scan && i % tps == 0) {
            __syncthreads();
            if (threadIdx.x < tps) s_on[threadIdx.x] = 0;
            __syncthreads();
            const uint64_t p = (b + (i + (threadIdx.x >> lpb)) * c.nblk) * pb + (threadIdx.x & (pb - 1));
            bool nz = false;
            if (p < pairs) {
                const uint32_t fl = c.bitness ? 1 : gate, fh = c.bitness ? c.nf : gate + 1;
#pragma unroll 4
                for (uint32_t f = fl; f < fh; f++) {
                    K f0, f1;
                    ldg_pair(c.tab + (uint64_t)f * c.len + 2 * p, f0, f1);
                    nz = nz || !gl::kiszero(f0) || !gl::kiszero(f1);
                }
            }
            if (nz) s_on[threadIdx.x >> lpb] = 1;
            __syncthreads();
        }
        if (scan && !s_on[i % tps]) continue;  // block-uniform
        K acc[MPTS], chi[MPTS];
#pragma unroll
        for (int k = 0; k < MPTS; k++) acc[k] = c.bitness ? gl::kzero() : gl::kone();
        bool on = true;
        for (uint32_t fb = 0; fb < c.nf; fb += fch) {
            const uint32_t nfc = min(fch, c.nf - fb);
            bool nz = c.bitness;
            for (uint32_t e = threadIdx.x; e < nfc * pb; e += 256) {
                const uint32_t f = e >> lpb;
                const uint64_t p = tile * pb + (e & (pb - 1));
                K f0 = gl::kzero(), f1 = gl::kzero();
                if (p < pairs) multi_factor(c, fb + f, p, true, f0, f1);
                if (!c.bitness && fb + f == gate) nz = nz || !gl::kiszero(f0) || !gl::kiszero(f1);
                s_f[0][e] = f0;
                s_f[1][e] = gl::ksub(f1, f0);
            }
            if (fb == 0 && !scan) on = __syncthreads_or(nz);
            else __syncthreads();
            if (on && xw < c.npts) {
                for (uint32_t f = sub; f < nfc; f += fs) {
                    const K f0 = s_f[0][(f << lpb) + pl], d = s_f[1][(f << lpb) + pl];
                    const bool chi_f = c.bitness && fb + f == 0;
                    if (c.bitness && !chi_f && gl::kiszero(f0) && gl::kiszero(d)) continue;
                    K v = gl::kadd(f0, gl::kscale_tiny(d, xw));
                    const K dx = gl::kscale_tiny(d, xstep);
                    const K w = c.bitness && !chi_f ? ldg_k(c.w + fb + f - 1) : gl::kzero();
#pragma unroll
                    for (int k = 0; k < MPTS; k++) {
                        if (xw + k * xstep >= c.npts) break;
                        if (!c.bitness) acc[k] = gl::kmul(acc[k], v);
                        else if (chi_f) chi[k] = v;
                        else acc[k] = gl::kadd(acc[k], gl::kmul(w, gl::kmul(v, gl::ksub(v, gl::kone()))));
                        v = gl::kadd(v, dx);
                    }
                }
            }
            __syncthreads();
        }
        if (on && xw < c.npts) {  // warp-uniform
            const bool add = sub == 0 && tile * pb + pl < pairs;
#pragma unroll
            for (int k = 0; k < MPTS; k++) {
                if (xw + k * xstep >= c.npts) break;
                for (uint32_t o = 1; o < fs; o <<= 1) {
                    const K other = shfl_xor_km(acc[k], o);
                    acc[k] = c.bitness ? gl::kadd(acc[k], other) : gl::kmul(acc[k], other);
                }
                if (add) total[k] = gl::kadd(total[k], c.bitness ? gl::kmul(chi[k], acc[k]) : acc[k]);
            }
        }
    }
#pragma unroll
    for (int k = 0; k < MPTS; k++) {
        if (xw + k * xstep >= c.npts) break;
        K v = total[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = gl::kadd(v, shfl_xor_km(v, o));
        if (lane == 0) s_red[warp][k] = v;
    }
    __syncthreads();
    if (threadIdx.x < c.npts) {
        const uint32_t x = threadIdx.x;
        K v = gl::kzero();
        for (uint32_t g = 0; g < hb; g++) v = gl::kadd(v, s_red[(x % xstep) * hb + g][x / xstep]);
        if (c.nblk > 1) {
            unsigned long long* acc = c.acc + ((b % MULTI_COPIES) * (MEM_MAX_DEG + 1) + x) * 4;
            atomicAdd(acc, (unsigned long long)(uint32_t)v.re);
            atomicAdd(acc + 1, (unsigned long long)(v.re >> 32));
            atomicAdd(acc + 2, (unsigned long long)(uint32_t)v.im);
            atomicAdd(acc + 3, (unsigned long long)(v.im >> 32));
        } else if (c.vinv) s_v[x] = v;
        else c.out[x] = v;
    }
    if (c.nblk == 1) {
        __syncthreads();
        if (c.vinv) multi_coeffs(c, s_v);
        return;
    }
    // the claim's last block to finish reduces the sums (ticket, no waits) and clears them
    __threadfence();
    __syncthreads();
    __shared__ unsigned int s_last;
    if (threadIdx.x == 0) s_last = atomicInc(c.ticket, c.nblk - 1) == c.nblk - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const bool on = threadIdx.x < 4 * c.npts;  // a thread per point and half word
    unsigned long long t[MULTI_COPIES] = {}, v = 0;
    if (on) {
        unsigned long long* acc = c.acc + threadIdx.x;
#pragma unroll
        for (uint32_t i = 0; i < MULTI_COPIES; i++) t[i] = __ldcg(acc + i * (MEM_MAX_DEG + 1) * 4);
#pragma unroll
        for (uint32_t i = 0; i < MULTI_COPIES; i++) {
            v += t[i];
            acc[i * (MEM_MAX_DEG + 1) * 4] = 0;
        }
    }
    // lo + 2^32 hi (each below 2^64: fewer than 2^32 blocks), then the component two lanes up
    uint64_t w = gl::canon(v);
    if (threadIdx.x & 1) w = gl::mul(w, 1ull << 32);
    w = gl::add(w, __shfl_down_sync(0xffffffffu, (unsigned long long)w, 1));
    const uint64_t im = __shfl_down_sync(0xffffffffu, (unsigned long long)w, 2);
    if (on && (threadIdx.x & 3) == 0) (c.vinv ? s_v : c.out)[threadIdx.x >> 2] = gl::kmk(w, im);
    if (!c.vinv) return;
    __syncthreads();
    multi_coeffs(c, s_v);
}

// Inverse Vandermonde matrices of the nodes 0..n-1 for n = 2..MEM_MAX_DEG + 1, row
// d column x: coefficient d of the x-th Lagrange basis polynomial.
constexpr uint32_t VINV_MAX = MEM_MAX_DEG + 1;
inline uint32_t vinv_off(uint32_t n) { return (n - 1) * n * (2 * n - 1) / 6; }  // sum of k^2, k < n
const std::vector<uint64_t>& vinv_host() {
    static const std::vector<uint64_t> tab = [] {
        std::vector<uint64_t> t(vinv_off(VINV_MAX + 1));
        for (uint32_t n = 1; n <= VINV_MAX; n++)
            for (uint32_t x = 0; x < n; x++) {
                std::vector<uint64_t> co(1, 1);  // prod_{j != x} (X - j)
                uint64_t den = 1;
                for (uint32_t j = 0; j < n; j++) {
                    if (j == x) continue;
                    co.push_back(0);
                    for (size_t d = co.size(); d-- > 0;)
                        co[d] = gl::sub(d ? co[d - 1] : 0, gl::mul(co[d], (uint64_t)j));
                    den = gl::mul(den, x > j ? (uint64_t)(x - j) : gl::neg((uint64_t)(j - x)));
                }
                const uint64_t s = gl::inv(den);
                for (uint32_t d = 0; d < n; d++) t[vinv_off(n) + d * n + x] = gl::mul(co[d], s);
            }
        return t;
    }();
    return tab;
}


inline K kload_h(const uint64_t* p) { return gl::kmk(p[0], p[1]); }

}  // namespace

struct neo_gpu_mem_oracle {
    neo_gpu_ctx* ctx = nullptr;
    int kind = 0;
    uint32_t ell = 0, A = 0, deg = 0, nf = 0, bit_idx = 0;
    int bitness = 0;
    uint64_t len = 0;     // current table length
    DevBuf<K> tab[2];     // ping-pong factor tables [nf][len]
    int cur = 0;
    bool pending = false; // a fold challenge not yet applied
    K pending_r{};
    DevBuf<K> w;          // bitness weights
    std::vector<K> hw;    // host copy of the weights
    DevBuf<K> partials;
    DevBuf<K> tmp, sums;  // build workspace, kept for reuse
    std::vector<K> hvals;
    bool hvals_valid = false;  // hvals holds this round's values (the claim needs round 0's)
    K claim{};
};

namespace {

uint32_t factor_count(int kind, uint32_t A, uint32_t n_cols) {
    switch (kind) {
        case NEO_MEM_SHOUT_VALUE: return 3;
        case NEO_MEM_SHOUT_ADAPTER: return 2 + A;
        case NEO_MEM_BITNESS: return 1 + n_cols;
        case NEO_MEM_TWIST_READ: return 3 + A;
        case NEO_MEM_TWIST_WRITE: return 3 + A;
        case NEO_MEM_VAL_EVAL: return 3 + A;
        case NEO_MEM_TOTAL_INC: return 2 + A;
        case NEO_MEM_PRODUCT: return n_cols;
    }
    return 0;
}

int expected_cols(int kind, uint32_t A, uint32_t n_cols) {
    switch (kind) {
        case NEO_MEM_SHOUT_VALUE: return 2;
        case NEO_MEM_SHOUT_ADAPTER: return 1 + A;
        case NEO_MEM_BITNESS: return n_cols;
        case NEO_MEM_TWIST_READ: return 4 + 2 * A;
        case NEO_MEM_TWIST_WRITE: return 3 + A;
        case NEO_MEM_VAL_EVAL: case NEO_MEM_TOTAL_INC: return 2 + A;
        case NEO_MEM_PRODUCT: return n_cols;
    }
    return -1;
}

uint32_t degree_of(int kind, uint32_t A, uint32_t n_cols) {
    switch (kind) {
        case NEO_MEM_SHOUT_VALUE: case NEO_MEM_BITNESS: return 3;
        case NEO_MEM_SHOUT_ADAPTER: case NEO_MEM_TOTAL_INC: return 2 + A;
        case NEO_MEM_TWIST_READ: case NEO_MEM_TWIST_WRITE: case NEO_MEM_VAL_EVAL: return 3 + A;
        case NEO_MEM_PRODUCT: return n_cols;
    }
    return 0;
}

// p(x) from p(0..n-1) (Lagrange on the integer nodes)
K lagrange_at(const std::vector<K>& v, K x) {
    const int n = (int)v.size();
    if (x.im == 0 && x.re < (uint64_t)n) return v[x.re];
    K acc = gl::kzero();
    for (int i = 0; i < n; i++) {
        K num = gl::kone();
        uint64_t den = 1;
        for (int j = 0; j < n; j++) {
            if (j == i) continue;
            num = gl::kmul(num, gl::ksub(x, gl::kfq((uint64_t)j)));
            den = gl::mul(den, i > j ? (uint64_t)(i - j) : gl::neg((uint64_t)(j - i)));
        }
        acc = gl::kadd(acc, gl::kmul(v[i], gl::kscale(num, gl::inv(den))));
    }
    return acc;
}

int mem_round_values(neo_gpu_mem_oracle* o);

int mem_create(neo_gpu_ctx* ctx, int kind, uint32_t ell, const uint64_t* r_point, uint32_t A, const uint64_t* r_addr,
               const uint64_t* init, uint32_t n_cols, const uint64_t* cols, bool cols_on_device,
               const uint64_t* weights, uint64_t* claim_out, neo_gpu_mem_oracle** out, bool reuse = false,
               bool lazy = false) {
    if (!ctx || !out) return NEO_ERR_ARG;
    if (!reuse) *out = nullptr;
    if (kind < NEO_MEM_SHOUT_VALUE || kind > NEO_MEM_PRODUCT) return ctx->fail(NEO_ERR_ARG, "mem_oracle: unknown kind");
    if (ell > 30) return ctx->fail(NEO_ERR_ARG, "mem_oracle: ell > 30");
    if (expected_cols(kind, A, n_cols) != (int)n_cols || (n_cols == 0 && kind != NEO_MEM_BITNESS))
        return ctx->fail(NEO_ERR_ARG, "mem_oracle: column count does not match the kind");
    const bool chi = kind <= NEO_MEM_TWIST_WRITE;
    if ((chi || kind == NEO_MEM_VAL_EVAL) && !r_point) return ctx->fail(NEO_ERR_ARG, "mem_oracle: missing r_cycle / r_time");
    if (A && !r_addr && kind != NEO_MEM_BITNESS && kind != NEO_MEM_PRODUCT && kind != NEO_MEM_SHOUT_VALUE)
        return ctx->fail(NEO_ERR_ARG, "mem_oracle: missing r_addr");
    if (kind == NEO_MEM_BITNESS && !weights && n_cols) return ctx->fail(NEO_ERR_ARG, "mem_oracle: missing weights");
    if (!cols && n_cols) return ctx->fail(NEO_ERR_ARG, "mem_oracle: null columns");
    const uint32_t deg = degree_of(kind, A, n_cols);
    if (deg > MEM_MAX_DEG) return ctx->fail(NEO_ERR_UNSUPPORTED, "mem_oracle: degree bound above 31");
    cudaSetDevice(ctx->device);
    PoolScope pool_scope(ctx);

    // reuse: rebuild into the caller's object, keeping its device buffers
    neo_gpu_mem_oracle* o = reuse ? *out : nullptr;
    const bool fresh = !o;
    if (fresh) o = new neo_gpu_mem_oracle();
    o->ctx = ctx;
    o->bit_idx = 0;
    o->cur = 0;
    o->pending = false;
    o->hvals_valid = false;
    o->hw.clear();
    o->kind = kind;
    o->ell = ell;
    o->A = A;
    o->deg = deg;
    o->nf = factor_count(kind, A, n_cols);
    o->bitness = kind == NEO_MEM_BITNESS;
    o->len = 1ULL << ell;
    const uint64_t L = o->len;
    auto fail = [&](int rc) {
        if (fresh) delete o;
        return rc;
    };
    if (o->tab[0].ensure((size_t)o->nf * L) || o->tab[1].ensure((size_t)o->nf * (L > 1 ? L / 2 : 1)))
        return fail(ctx->fail(NEO_ERR_OOM, "mem_oracle: table allocation"));
    K* T = o->tab[0].p;
    cudaStream_t S = ctx->stream;
    const cudaMemcpyKind cpk = cols_on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
    const size_t colb = L * sizeof(K);
    auto col = [&](uint32_t c) { return reinterpret_cast<const K*>(cols) + (size_t)c * L; };
    // factors f.. = columns c.. (n of them, adjacent)
    auto put = [&](uint32_t f, uint32_t c, uint32_t n = 1) {
        return n ? cudaMemcpyAsync(T + (size_t)f * L, col(c), colb * n, cpk, S) : cudaSuccess;
    };
    DevBuf<K>& tmp = o->tmp;
    // (the kinds that read r_addr have A <= 31 by the degree bound)
    const KPoint addr_pt = A && r_addr ? make_point(reinterpret_cast<const K*>(r_addr), A) : KPoint{};
    auto eqbits = [&](uint32_t f0, uint32_t c0) -> int {
        if (!A) return NEO_OK;
        if (!r_addr) return ctx->fail(NEO_ERR_ARG, "mem_oracle: address bits without r_addr");
        K* dst = T + (size_t)f0 * L;
        if (!cols_on_device && put(f0, c0, A)) return ctx->fail(NEO_ERR_CUDA, "mem_oracle: column upload");
        eqbit_kernel<<<dim3(ceil_div(L, 256), A), 256, 0, S>>>(cols_on_device ? col(c0) : dst, L, addr_pt, dst);
        NEO_LAUNCHED(ctx);
        return NEO_OK;
    };
    int rc = NEO_OK;
    if (chi) {  // factor 0 = χ_{r_cycle}
        rc = launch_chi_point(ctx, reinterpret_cast<const K*>(r_point), ell, T);
        if (rc) return fail(rc);
    }
    cudaError_t ce = cudaSuccess;
    switch (kind) {
        case NEO_MEM_SHOUT_VALUE:
            ce = put(1, 0, 2);
            break;
        case NEO_MEM_SHOUT_ADAPTER:
            ce = put(1, 0);
            if (!ce) rc = eqbits(2, 1);
            break;
        case NEO_MEM_BITNESS:
            ce = put(1, 0, n_cols);
            for (uint32_t c = 0; c < n_cols; c++) o->hw.push_back(kload_h(weights + 2 * c));
            if (!ce && n_cols && (o->w.ensure(n_cols) ||
                        cudaMemcpyAsync(o->w.p, weights, n_cols * sizeof(K), cudaMemcpyHostToDevice, S)))
                ce = cudaErrorMemoryAllocation;
            break;
        case NEO_MEM_TWIST_READ:
        case NEO_MEM_TWIST_WRITE: {
            const bool rd = kind == NEO_MEM_TWIST_READ;
            // write stream columns: has_write, inc, wa bits
            const uint32_t c_hw = rd ? 2 + A : 0, c_inc = rd ? 3 + A : 2, c_wa = rd ? 4 + A : 3;
            const uint32_t c_a = rd ? 1 : 1;  // rv (read) or wv (write)
            // columns on the device are read where they are
            if (tmp.ensure((cols_on_device ? 1 : (size_t)(4 + A)) * L)) { ce = cudaErrorMemoryAllocation; break; }
            K* terms = tmp.p;
            const K *hw = col(c_hw), *inc = col(c_inc), *aa = col(c_a), *wa = col(c_wa);
            if (!cols_on_device) {
                K* up = tmp.p + L;
                ce = cudaMemcpyAsync(up, hw, colb, cpk, S);
                if (!ce) ce = cudaMemcpyAsync(up + L, inc, colb, cpk, S);
                if (!ce) ce = cudaMemcpyAsync(up + 2 * L, aa, colb, cpk, S);
                if (!ce && A) ce = cudaMemcpyAsync(up + 3 * L, wa, colb * A, cpk, S);
                hw = up; inc = up + L; aa = up + 2 * L; wa = up + 3 * L;
            }
            if (ce) break;
            inc_terms_kernel<<<ceil_div(L, 256), 256, 0, S>>>(hw, inc, wa, A, addr_pt, L, terms);
            NEO_LAUNCHED(ctx);
            const uint32_t nblk = (uint32_t)ceil_div(L, SCAN_BLK);
            DevBuf<K>& sums = o->sums;
            if (sums.ensure(nblk)) { ce = cudaErrorMemoryAllocation; break; }
            scan_sums_kernel<<<nblk, SCAN_T, 0, S>>>(terms, L, sums.p);
            NEO_LAUNCHED(ctx);
            K init_k = init ? kload_h(init) : gl::kzero();
            scan_top_kernel<<<1, SCAN_T, 0, S>>>(sums.p, nblk, init_k);
            NEO_LAUNCHED(ctx);
            // factor 2 = Val_pre − rv  |  wv − Val_pre − inc
            scan_final_kernel<<<nblk, SCAN_T, 0, S>>>(terms, L, sums.p, rd ? 1 : 2, aa, inc, T + 2 * L);
            NEO_LAUNCHED(ctx);
            ce = put(1, 0);  // gate: has_read | has_write
            if (!ce) rc = eqbits(3, rd ? 2 : 3);
        } break;
        case NEO_MEM_VAL_EVAL:
            ce = put(0, 0, 2);
            if (ce) break;
            lt_table_kernel<<<ceil_div(std::max<uint64_t>(L >> 8, 1), LT_HIGH), 256, 0, S>>>(
                make_point(reinterpret_cast<const K*>(r_point), ell), ell, T + 2 * L);
            NEO_LAUNCHED(ctx);
            rc = eqbits(3, 2);
            break;
        case NEO_MEM_TOTAL_INC:
            ce = put(0, 0, 2);
            if (!ce) rc = eqbits(2, 2);
            break;
        case NEO_MEM_PRODUCT:
            ce = put(0, 0, n_cols);
            break;
    }
    if (ce) return fail(ctx->fail(ce == cudaErrorMemoryAllocation ? NEO_ERR_OOM : NEO_ERR_CUDA, "mem_oracle: build", ce));
    if (rc) return fail(rc);
    // claim = Σ over the hypercube = p_0(0) + p_0(1)  (the constructors' sums);
    // a lazy build (the shard: no claim asked for, or claims computed for a
    // group by mem_claims_multi) skips it
    if (!lazy) {
        rc = mem_round_values(o);
        if (rc) return fail(rc);
        o->claim = ell ? gl::kadd(o->hvals[0], o->hvals[1]) : o->hvals[0];
        if (claim_out) {
            claim_out[0] = o->claim.re;
            claim_out[1] = o->claim.im;
        }
        NEO_CK(ctx, ctx_sync(ctx));
    }
    *out = o;
    return NEO_OK;
}

}  // namespace

// True when the oracle's next round has at least one pair (its pending fold
// applied): the rounds that mem_round_launch_multi evaluates.
bool mem_round_multi_ok(const neo_gpu_mem_oracle* o) {
    const uint64_t len = o->pending ? o->len >> 1 : o->len;
    return len >= 2 && o->deg + 1 <= MEM_MAX_DEG + 1;
}

// The next round of n oracles: pending folds, then the values at x = 0..deg
// of oracle i (coeffs: the round polynomial's coefficients) into d_out[i] (device-
// visible), in one launch and without a host sync.  Every oracle must satisfy mem_round_multi_ok; n <= MULTI_MAX.
int mem_round_launch_multi(neo_gpu_ctx* ctx, neo_gpu_mem_oracle* const* os, int n, K* const* d_out,
                           DevBuf<K>& partials, bool coeffs) {
    if (n <= 0) return NEO_OK;
    if (coeffs && !ctx->vinv) {
        const std::vector<uint64_t>& t = vinv_host();
        NEO_CK(ctx, ctx_malloc(ctx, reinterpret_cast<void**>(&ctx->vinv), t.size() * 8));
        NEO_CK(ctx, cudaMemcpyAsync(ctx->vinv, t.data(), t.size() * 8, cudaMemcpyHostToDevice, ctx->stream));
    }
    if (n > MULTI_MAX) return ctx->fail(NEO_ERR_UNSUPPORTED, "mem_round_launch_multi: too many claims");
    MultiArgs a{};
    a.n = n;
    // a launch's blocks, shared out by what a claim reads of the inactive rows: every
    // column of a bitness claim, the gate of a product (which gets as much as 8 columns
    // for its products)
    auto multi_weight = [](const neo_gpu_mem_oracle* o) -> uint64_t { return o->bitness ? o->nf : 8; };
    uint64_t wsum = 0;
    for (int i = 0; i < n; i++) wsum += multi_weight(os[i]);
    MultiFold mf{};
    uint64_t fold_len = 0;
    uint32_t blocks = 0;
    uint64_t parts = 0;
    for (int i = 0; i < n; i++) {
        neo_gpu_mem_oracle* o = os[i];
        MultiClaim& c = a.c[i];
        c = MultiClaim{};
        if (o->pending) {  // a small claim's evaluation applies the fold; a large one's is a launch of its own
            c.src = o->tab[o->cur].p;
            c.r = o->pending_r;
            o->cur ^= 1;
            o->len >>= 1;
            o->pending = false;
            if (o->len >= 2 * FOLD_PAIRS) {
                mf.src[mf.n] = c.src;
                mf.dst[mf.n] = o->tab[o->cur].p;
                mf.half[mf.n] = o->len;
                mf.r[mf.n] = c.r;
                mf.f0[mf.n + 1] = mf.f0[mf.n] + o->nf;
                mf.n++;
                fold_len = std::max(fold_len, o->len);
                c.src = nullptr;
            }
        }
        o->hvals_valid = false;
        if (o->len < 2) return ctx->fail(NEO_ERR_INVARIANT, "mem_round_launch_multi: no pairs left");
        c.tab = o->tab[o->cur].p;
        c.len = o->len;
        c.nf = o->nf;
        c.npts = o->deg + 1;
        c.bitness = o->bitness;
        c.w = o->w.p;
        c.blk0 = blocks;
        c.part0 = (uint32_t)parts;
        c.out = d_out[i];
        c.vinv = coeffs ? ctx->vinv + vinv_off(c.npts) : nullptr;
        const uint64_t pairs = o->len >> 1;
        if (pairs <= SMALL_PAIRS) {
            // lanes per pair: what 256 threads leave, up to 16 and to the factors there are
            c.small = 1;
            c.fs = 1;
            while (c.fs < 16 && 2 * c.fs * pairs <= 256 && c.fs < c.nf - (c.bitness ? 1 : 0)) c.fs *= 2;
            blocks += c.npts;
            parts += c.npts;
            continue;
        }
        // eight warps cover the points; with fewer points, warps share a point's pairs
        c.hb = 1;
        while (c.hb < 8 && 8 / (2 * c.hb) >= c.npts) c.hb *= 2;
        // the blocks that are resident, two per SM, over the launch's claims (with four
        // per SM the first rounds of a fold step's 100 columns took 31 to 43 us, now 24 to
        // 28); tiles small enough (up to 16 lanes a pair)
        c.fs = 1;
        while (c.fs < 16 && 2 * c.fs <= c.nf && pairs * c.fs / (32 * c.hb) < MULTI_TILES / (uint32_t)n) c.fs *= 2;
        c.lpb = 5;
        for (uint32_t h = 1; h < c.hb; h *= 2) c.lpb++;
        for (uint32_t h = 1; h < c.fs; h *= 2) c.lpb--;
        const uint64_t tiles = (pairs + (1ull << c.lpb) - 1) >> c.lpb;
        c.nblk = (uint32_t)std::min<uint64_t>(tiles, std::max<uint64_t>(64, 2ull * 148 * multi_weight(o) / wsum));
        blocks += c.nblk;
    }
    if (parts > 0xFFFFFFFFull) return ctx->fail(NEO_ERR_UNSUPPORTED, "mem_round_launch_multi: too many partials");
    // the claims' sums and tickets (MULTI_MAX of each, in MULTI_TICKET_K entries) sit
    // behind the partials of the small claims; they return to zero after every launch,
    // so they are cleared only when the buffer is (re)allocated
    constexpr size_t ACC_WORDS = (size_t)MULTI_COPIES * (MEM_MAX_DEG + 1) * 4;
    constexpr size_t MULTI_ACC_K = MULTI_MAX * ACC_WORDS * 8 / sizeof(K);
    constexpr size_t MULTI_TICKET_K = MULTI_ACC_K + (MULTI_MAX * sizeof(unsigned int) + sizeof(K) - 1) / sizeof(K);
    const K* before = partials.p;
    const size_t cap_before = partials.cap;
    NEO_CK(ctx, partials.ensure(std::max<uint64_t>(parts, cap_before > MULTI_TICKET_K ? cap_before - MULTI_TICKET_K : 0) +
                                MULTI_TICKET_K));
    K* tail = partials.p + (partials.cap - MULTI_TICKET_K);
    if (partials.p != before || partials.cap != cap_before)
        NEO_CK(ctx, cudaMemsetAsync(tail, 0, MULTI_TICKET_K * sizeof(K), ctx->stream));
    for (int i = 0; i < n; i++) {
        a.c[i].acc = reinterpret_cast<unsigned long long*>(tail) + i * ACC_WORDS;
        a.c[i].ticket = reinterpret_cast<unsigned int*>(tail + MULTI_ACC_K) + i;
    }
    a.partials = partials.p;
    if (mf.n) {
        const uint32_t gy = std::min(mf.f0[mf.n], 65535u);
        mem_multi_fold_kernel<<<dim3(ceil_div(fold_len, 256 * FOLD_PER), gy, ceil_div(mf.f0[mf.n], gy)), 256, 0, ctx->stream>>>(mf);
        NEO_LAUNCHED(ctx);
    }
    mem_multi_eval_kernel<<<blocks, 256, 0, ctx->stream>>>(a);
    NEO_LAUNCHED(ctx);
    return NEO_OK;
}



namespace {

// round values at x = 0..deg into o->hvals (applies a pending fold first); the
// launch writes them into the context's host-mapped result buffer
int mem_round_values(neo_gpu_mem_oracle* o) {
    if (o->hvals_valid) return NEO_OK;
    neo_gpu_ctx* ctx = o->ctx;
    const uint32_t npts = o->deg + 1;
    o->hvals.assign(npts, gl::kzero());
    if (mem_round_multi_ok(o)) {
        K* out = reinterpret_cast<K*>(ctx->h_result);
        result_arm(out, 2 * (size_t)npts);
        if (int rc = mem_round_launch_multi(ctx, &o, 1, &out, o->partials, false)) return rc;
        NEO_CK(ctx, result_wait(ctx, out, 2 * (size_t)npts));
        for (uint32_t x = 0; x < npts; x++) o->hvals[x] = out[x];
        o->hvals_valid = true;
        return NEO_OK;
    }
    // one entry per factor: the final product at every x
    std::vector<K> v(o->nf);
    bool have = false;
    if (o->pending) {
        K* out = reinterpret_cast<K*>(ctx->h_result);
        have = o->len == 2 && o->nf <= 128;  // fits h_result
        if (have) result_arm(out, 2 * (size_t)o->nf);
        mem_fold_kernel<<<ceil_div((o->len >> 1) * o->nf, 256), 256, 0, ctx->stream>>>(
            o->tab[o->cur].p, o->len, o->tab[o->cur ^ 1].p, o->nf, o->pending_r, have ? out : nullptr);
        NEO_LAUNCHED(ctx);
        o->cur ^= 1;
        o->len >>= 1;
        o->pending = false;
        if (have) {
            NEO_CK(ctx, result_wait(ctx, out, 2 * (size_t)o->nf));
            std::copy(out, out + o->nf, v.begin());
        }
    }
    if (!have) {
        NEO_CK(ctx, ctx_d2h(ctx, v.data(), o->tab[o->cur].p, o->nf * sizeof(K)));
        NEO_CK(ctx, ctx_sync(ctx));
    }
    K val;
    if (o->bitness) {
        K s = gl::kzero();
        for (uint32_t f = 1; f < o->nf; f++)
            s = gl::kadd(s, gl::kmul(gl::kmul(o->hw[f - 1], v[f]), gl::ksub(v[f], gl::kone())));
        val = gl::kmul(v[0], s);
    } else {
        val = gl::kone();
        for (uint32_t f = 0; f < o->nf; f++) val = gl::kmul(val, v[f]);
    }
    for (auto& h : o->hvals) h = val;
    o->hvals_valid = true;
    return NEO_OK;
}

}  // namespace

// Claims (sums over the hypercube, p_0(0) + p_0(1)) of n lazily built oracles:
// one multi-claim evaluation of their round 0 into page-locked memory, one sync;
// oracles the multi-claim kernel cannot take are evaluated one by one.
int mem_claims_multi(neo_gpu_ctx* ctx, neo_gpu_mem_oracle* const* os, int n, K* claims, DevBuf<K>& partials,
                     HostBuf<K>& h_slots) {
    constexpr uint32_t SLOT = MEM_MAX_DEG + 1;
    bool multi = n > 0 && n <= MULTI_MAX;
    for (int i = 0; i < n && multi; i++) multi = mem_round_multi_ok(os[i]) && !os[i]->pending && os[i]->ell > 0;
    if (!multi) {
        for (int i = 0; i < n; i++) {
            neo_gpu_mem_oracle* o = os[i];
            if (int rc = mem_round_values(o)) return rc;
            o->claim = o->ell ? gl::kadd(o->hvals[0], o->hvals[1]) : o->hvals[0];
            claims[i] = o->claim;
        }
        NEO_CK(ctx, ctx_sync(ctx));
        return NEO_OK;
    }
    NEO_CK(ctx, h_slots.ensure((size_t)n * SLOT));
    std::vector<K*> dst(n);
    for (int i = 0; i < n; i++) dst[i] = h_slots.p + (size_t)i * SLOT;
    if (int rc = mem_round_launch_multi(ctx, os, n, dst.data(), partials, false)) return rc;
    NEO_CK(ctx, ctx_sync(ctx));
    for (int i = 0; i < n; i++) {
        const K* v = h_slots.p + (size_t)i * SLOT;
        os[i]->claim = gl::kadd(v[0], v[1]);
        claims[i] = os[i]->claim;
    }
    return NEO_OK;
}

static int neo_gpu_mem_oracle_create_impl_abi(neo_gpu_ctx* ctx, int kind, uint32_t ell, const uint64_t* r_point,
                                         uint32_t ell_addr, const uint64_t* r_addr, const uint64_t* init_at_r_addr,
                                         uint32_t n_cols, const uint64_t* cols, const uint64_t* weights,
                                         uint64_t* claim, neo_gpu_mem_oracle** out) {
    return mem_create(ctx, kind, ell, r_point, ell_addr, r_addr, init_at_r_addr, n_cols, cols, false, weights, claim,
                      out);
}
extern "C" int neo_gpu_mem_oracle_create(neo_gpu_ctx* ctx, int kind, uint32_t ell, const uint64_t* r_point,
                                         uint32_t ell_addr, const uint64_t* r_addr, const uint64_t* init_at_r_addr,
                                         uint32_t n_cols, const uint64_t* cols, const uint64_t* weights,
                                         uint64_t* claim, neo_gpu_mem_oracle** out) { NEO_ABI_GUARD(neo_gpu_mem_oracle_create_impl_abi(ctx, kind, ell, r_point, ell_addr, r_addr, init_at_r_addr, n_cols, cols, weights, claim, out)) }

// Rebuild into *slot when it holds an oracle (its device buffers are kept),
// create one otherwise; columns in device memory.  Fold steps call this every
// step so that no device allocation (a device-wide synchronization for
// cudaFree) happens once the buffers have grown.
int mem_oracle_build_device(neo_gpu_ctx* ctx, int kind, uint32_t ell, const uint64_t* r_point, uint32_t ell_addr,
                            const uint64_t* r_addr, const uint64_t* init_at_r_addr, uint32_t n_cols,
                            const uint64_t* d_cols, const uint64_t* weights, uint64_t* claim,
                            neo_gpu_mem_oracle** slot) {
    return mem_create(ctx, kind, ell, r_point, ell_addr, r_addr, init_at_r_addr, n_cols, d_cols, true, weights, claim,
                      slot, true, claim == nullptr);
}

static int neo_gpu_mem_oracle_create_device_impl_abi(neo_gpu_ctx* ctx, int kind, uint32_t ell, const uint64_t* r_point,
                                                uint32_t ell_addr, const uint64_t* r_addr,
                                                const uint64_t* init_at_r_addr, uint32_t n_cols,
                                                const uint64_t* d_cols, const uint64_t* weights, uint64_t* claim,
                                                neo_gpu_mem_oracle** out) {
    return mem_create(ctx, kind, ell, r_point, ell_addr, r_addr, init_at_r_addr, n_cols, d_cols, true, weights, claim,
                      out);
}
extern "C" int neo_gpu_mem_oracle_create_device(neo_gpu_ctx* ctx, int kind, uint32_t ell, const uint64_t* r_point,
                                                uint32_t ell_addr, const uint64_t* r_addr,
                                                const uint64_t* init_at_r_addr, uint32_t n_cols,
                                                const uint64_t* d_cols, const uint64_t* weights, uint64_t* claim,
                                                neo_gpu_mem_oracle** out) { NEO_ABI_GUARD(neo_gpu_mem_oracle_create_device_impl_abi(ctx, kind, ell, r_point, ell_addr, r_addr, init_at_r_addr, n_cols, d_cols, weights, claim, out)) }

static int neo_gpu_mem_oracle_evals_impl_abi(neo_gpu_mem_oracle* o, const uint64_t* xs, uint32_t nx, uint64_t* ys) {
    if (!o) return NEO_ERR_ARG;
    if ((!xs || !ys) && nx) return o->ctx->fail(NEO_ERR_ARG, "mem_oracle_evals: null buffer");
    cudaSetDevice(o->ctx->device);
    PoolScope pool_scope(o->ctx);
    int rc = mem_round_values(o);
    if (rc) return rc;
    for (uint32_t i = 0; i < nx; i++) {
        K y = lagrange_at(o->hvals, kload_h(xs + 2 * i));
        ys[2 * i] = y.re;
        ys[2 * i + 1] = y.im;
    }
    return NEO_OK;
}
extern "C" int neo_gpu_mem_oracle_evals(neo_gpu_mem_oracle* o, const uint64_t* xs, uint32_t nx, uint64_t* ys) { NEO_ABI_GUARD(neo_gpu_mem_oracle_evals_impl_abi(o, xs, nx, ys)) }

static int neo_gpu_mem_oracle_fold_impl_abi(neo_gpu_mem_oracle* o, const uint64_t* r) {
    if (!o) return NEO_ERR_ARG;
    if (!r) return o->ctx->fail(NEO_ERR_ARG, "mem_oracle_fold: null challenge");
    if (o->bit_idx >= o->ell) return NEO_OK;  // no rounds left: ignored, as in the reference
    o->hvals_valid = false;
    if (o->pending) {
        // two folds without an evaluation in between: apply the first now
        neo_gpu_ctx* ctx = o->ctx;
        cudaSetDevice(ctx->device);
        uint64_t tot = (o->len >> 1) * o->nf;
        mem_fold_kernel<<<ceil_div(tot, 256), 256, 0, ctx->stream>>>(o->tab[o->cur].p, o->len, o->tab[o->cur ^ 1].p,
                                                                     o->nf, o->pending_r, nullptr);
        NEO_LAUNCHED(ctx);
        o->cur ^= 1;
        o->len >>= 1;
    }
    o->pending = true;
    o->pending_r = kload_h(r);
    o->bit_idx++;
    return NEO_OK;
}
extern "C" int neo_gpu_mem_oracle_fold(neo_gpu_mem_oracle* o, const uint64_t* r) { NEO_ABI_GUARD(neo_gpu_mem_oracle_fold_impl_abi(o, r)) }

extern "C" uint32_t neo_gpu_mem_oracle_num_rounds(const neo_gpu_mem_oracle* o) { return o ? o->ell - o->bit_idx : 0; }
extern "C" uint32_t neo_gpu_mem_oracle_degree_bound(const neo_gpu_mem_oracle* o) { return o ? o->deg : 0; }

static int neo_gpu_mem_oracle_destroy_impl_abi(neo_gpu_mem_oracle* o) {
    if (!o) return NEO_OK;
    cudaSetDevice(o->ctx->device);
    neo_gpu_ctx* ctx = o->ctx;
    cudaStreamSynchronize(ctx->stream);
    delete o;
    pool_trim(ctx);
    return NEO_OK;
}
extern "C" int neo_gpu_mem_oracle_destroy(neo_gpu_mem_oracle* o) { NEO_ABI_GUARD(neo_gpu_mem_oracle_destroy_impl_abi(o)) }

// AddressLookupOracle weights from device columns: d_rcycle (ell K), d_has
// (2^ell K), d_bits (A columns of 2^ell K), d_table (table_len K).  Writes
// d_w (2^A K) and the claimed sum to *claim (host); synchronizes the stream.
int addr_weights_device(neo_gpu_ctx* ctx, uint32_t ell, const K* d_rcycle, uint32_t A, const K* d_has,
                        const K* d_bits, const K* d_table, uint64_t table_len, K* d_w, K* claim, AddrWs* ws) {
    cudaStream_t S = ctx->stream;
    const uint64_t L = 1ULL << ell, P = 1ULL << A;
    AddrWs local;
    AddrWs& W = ws ? *ws : local;
    DevBuf<K>& chi = W.chi;
    DevBuf<K>& part = W.part;
    DevBuf<K>& out1 = W.out1;
    DevBuf<unsigned long long>& acc = W.acc;
    NEO_CK(ctx, chi.ensure(L));
    NEO_CK(ctx, acc.ensure(4 * P));
    NEO_CK(ctx, cudaMemsetAsync(acc.p, 0, 4 * P * sizeof(unsigned long long), S));
    int rc = launch_chi_table(ctx, d_rcycle, ell, chi.p);
    if (rc) return rc;
    addr_weights_kernel<<<ceil_div(L, 256), 256, 0, S>>>(chi.p, d_has, d_bits, A, L, acc.p, acc.p + 2 * P);
    NEO_LAUNCHED(ctx);
    addr_weights_finish_kernel<<<ceil_div(P, 256), 256, 0, S>>>(acc.p, acc.p + 2 * P, P, d_w);
    NEO_LAUNCHED(ctx);
    const uint64_t n = table_len < P ? table_len : P;
    const uint32_t nb = 148;
    NEO_CK(ctx, part.ensure(nb));
    NEO_CK(ctx, out1.ensure(1));
    dot_kernel<<<nb, 256, 0, S>>>(d_table, d_w, n, part.p);
    NEO_LAUNCHED(ctx);
    mem_reduce_kernel<<<1, 256, 0, S>>>(part.p, nb, out1.p);
    NEO_LAUNCHED(ctx);
    NEO_CK(ctx, ctx_d2h(ctx, claim, out1.p, sizeof(K)));
    NEO_CK(ctx, ctx_sync(ctx));
    return NEO_OK;
}

static int neo_gpu_addr_lookup_weights_impl_abi(neo_gpu_ctx* ctx, uint32_t ell, const uint64_t* r_cycle, uint32_t ell_addr,
                                           const uint64_t* has_lookup, const uint64_t* addr_bits,
                                           const uint64_t* table, uint64_t table_len, uint64_t* weights,
                                           uint64_t* claim) {
    if (!ctx) return NEO_ERR_ARG;
    if (!r_cycle || !has_lookup || (!addr_bits && ell_addr) || !weights || !claim || (!table && table_len))
        return ctx->fail(NEO_ERR_ARG, "addr_lookup_weights: null buffer");
    if (ell > 30 || ell_addr > 30) return ctx->fail(NEO_ERR_ARG, "addr_lookup_weights: size");
    cudaSetDevice(ctx->device);
    PoolScope pool_scope(ctx);
    cudaStream_t S = ctx->stream;
    const uint64_t L = 1ULL << ell, P = 1ULL << ell_addr;
    DevBuf<K> dr, has, bits, w, tab;
    NEO_CK(ctx, dr.alloc(ell ? ell : 1));
    NEO_CK(ctx, has.alloc(L));
    NEO_CK(ctx, bits.alloc((size_t)L * (ell_addr ? ell_addr : 1)));
    NEO_CK(ctx, w.alloc(P));
    NEO_CK(ctx, tab.alloc(table_len ? table_len : 1));
    if (ell) NEO_CK(ctx, cudaMemcpyAsync(dr.p, r_cycle, ell * sizeof(K), cudaMemcpyHostToDevice, S));
    NEO_CK(ctx, cudaMemcpyAsync(has.p, has_lookup, L * sizeof(K), cudaMemcpyHostToDevice, S));
    if (ell_addr) NEO_CK(ctx, cudaMemcpyAsync(bits.p, addr_bits, (size_t)L * ell_addr * sizeof(K), cudaMemcpyHostToDevice, S));
    if (table_len) NEO_CK(ctx, cudaMemcpyAsync(tab.p, table, table_len * sizeof(K), cudaMemcpyHostToDevice, S));
    K cl;
    int rc = addr_weights_device(ctx, ell, dr.p, ell_addr, has.p, bits.p, tab.p, table_len, w.p, &cl, nullptr);
    if (rc) return rc;
    NEO_CK(ctx, ctx_d2h(ctx, weights, w.p, P * sizeof(K)));
    NEO_CK(ctx, ctx_sync(ctx));
    claim[0] = cl.re;
    claim[1] = cl.im;
    return NEO_OK;
}
extern "C" int neo_gpu_addr_lookup_weights(neo_gpu_ctx* ctx, uint32_t ell, const uint64_t* r_cycle, uint32_t ell_addr,
                                           const uint64_t* has_lookup, const uint64_t* addr_bits,
                                           const uint64_t* table, uint64_t table_len, uint64_t* weights,
                                           uint64_t* claim) { NEO_ABI_GUARD(neo_gpu_addr_lookup_weights_impl_abi(ctx, ell, r_cycle, ell_addr, has_lookup, addr_bits, table, table_len, weights, claim)) }

// ===========================================================================
// Twist address-lane oracles (TwistReadCheckAddrOracleSparseTime /
// TwistWriteCheckAddrOracleSparseTime, twist_oracle.rs:1259-1642).
//
// The reference replays a HashMap memory over the time-ordered events every
// round.  Here the reads and writes are items in time order, and the memory
// value a query item i sees at address block idx of round `bit` is
//     init_tab[idx] + Σ_{j < i, addr_j >> bit = idx} d_j,
// d_j = inc_j·hw_j·(address weight of the bound bits), init_tab the initial
// memory folded on its low address bits (the reference's init prefix weights
// are exactly that fold).  The items are kept sorted by (addr >> (bit + 1),
// time): the two blocks a query interpolates between are then one run, and the
// sums over its earlier writes are two prefix sums within the run.  A stable
// radix sort makes the order of round 0; a fold merges each pair of sibling
// runs by time.  Degree 2: values at x = 0, 1, 2, interpolated on the host.
// (One thread per query summing every earlier write of its block took 653 us a
// round at 2^14 events, each a read and a write, and 12.6 us at 2^10 beside the fold's
// launch; now 14.8 and 13.3 with the fold and the next order in it.)
// ===========================================================================
namespace {

constexpr int TA_T = 64;     // build blocks
constexpr int TE_T = 256;    // items per evaluation block

__device__ __forceinline__ uint32_t addr_bits_at(const K* bits, uint64_t L, uint32_t A, uint64_t t) {
    uint32_t a = 0;
    for (uint32_t b = 0; b < A; b++) {
        K v = bits[(uint64_t)b * L + t];
        if (v.re == 1 && v.im == 0) a |= 1u << b;
    }
    return a;
}

// An item's sort key: write flag (read kind only) : address (30 bits) : item index (time order).
__device__ __forceinline__ uint64_t ta_key(uint32_t write, uint32_t addr, uint32_t idx) {
    return ((uint64_t)write << 63) | ((uint64_t)addr << 32) | idx;
}
__device__ __forceinline__ uint32_t ta_addr(uint64_t key) { return (uint32_t)(key >> 32) & 0x7FFFFFFFu; }

// items per build block: kind 0 one for has_read != 0 and one for has_write != 0, kind 1 one for has_write != 0
__global__ void ta_count_kernel(const K* __restrict__ hr, const K* __restrict__ hw, uint64_t L, uint32_t* __restrict__ counts) {
    __shared__ uint32_t s_cnt;
    if (threadIdx.x == 0) s_cnt = 0;
    __syncthreads();
    const uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    const bool w = t < L && !gl::kiszero(hw[t]), r = t < L && hr && !gl::kiszero(hr[t]);
    const int n = __popc(__ballot_sync(0xffffffffu, w)) + __popc(__ballot_sync(0xffffffffu, r));
    if ((threadIdx.x & 31) == 0 && n) atomicAdd(&s_cnt, (uint32_t)n);
    __syncthreads();
    if (threadIdx.x == 0) counts[blockIdx.x] = s_cnt;
}

struct TaBuild {
    const K *hr, *rv, *ra, *hw, *inc, *wa, *wv;
    const K* r_cycle;
    uint32_t ell, A;
    uint64_t L;
    const uint32_t* offs;   // exclusive prefix of the per-block counts
    // outputs [N]
    uint64_t* key;
    K *wt;                  // query weight χ·has (kind 0: reads; kind 1) or write delta inc·has_write (kind 0: writes)
    K *kc;                  // a query's constant: rv, or wv − inc
    K *d;                   // kind 1: write delta
};

__global__ void ta_build_kernel(const TaBuild a) {
    __shared__ uint32_t s_warp[TA_T / 32];
    const uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    const K hw = t < a.L ? a.hw[t] : gl::kzero(), hr = t < a.L && a.hr ? a.hr[t] : gl::kzero();
    const bool w = !gl::kiszero(hw), r = !gl::kiszero(hr);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned bw = __ballot_sync(0xffffffffu, w), br = __ballot_sync(0xffffffffu, r);
    if (lane == 0) s_warp[warp] = __popc(bw) + __popc(br);
    __syncthreads();
    if (!w && !r) return;
    uint32_t n = a.offs[blockIdx.x];
    for (int i = 0; i < warp; i++) n += s_warp[i];
    const unsigned lt = (1u << lane) - 1;
    n += __popc(bw & lt) + __popc(br & lt);
    // χ_{r_cycle}(t)
    K chi = gl::kone();
    if (r || !a.hr)
        for (uint32_t i = 0; i < a.ell; i++) {
            K ri = a.r_cycle[i];
            chi = gl::kmul(chi, ((t >> i) & 1) ? ri : gl::ksub(gl::kone(), ri));
        }
    const K delta = w ? gl::kmul(a.inc[t], hw) : gl::kzero();
    if (!a.hr) {
        a.key[n] = ta_key(0, addr_bits_at(a.wa, a.L, a.A, t), n);
        a.wt[n] = gl::kmul(chi, hw);
        a.kc[n] = gl::ksub(a.wv[t], a.inc[t]);
        a.d[n] = delta;
        return;
    }
    if (r) {  // a step's read comes before its write
        a.key[n] = ta_key(0, addr_bits_at(a.ra, a.L, a.A, t), n);
        a.wt[n] = gl::kmul(chi, hr);
        a.kc[n] = a.rv[t];
        n++;
    }
    if (w) {
        a.key[n] = ta_key(1, addr_bits_at(a.wa, a.L, a.A, t), n);
        a.wt[n] = delta;
    }
}

// ---- stable radix sort of the items by 8 address bits (least significant first) ----
constexpr int RS_T = 256, RS_PER = 8, RS_TILE = RS_T * RS_PER;

__global__ void __launch_bounds__(RS_T) rs_hist_kernel(const uint64_t* __restrict__ key, uint32_t N, int shift,
                                                       uint32_t n_tiles, uint32_t* __restrict__ hist) {
    __shared__ uint32_t s_h[256];
    s_h[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t base = blockIdx.x * RS_TILE;
#pragma unroll
    for (int i = 0; i < RS_PER; i++) {
        const uint32_t p = base + i * RS_T + threadIdx.x;
        if (p < N) atomicAdd(&s_h[(ta_addr(key[p]) >> shift) & 255], 1u);
    }
    __syncthreads();
    hist[(uint64_t)threadIdx.x * n_tiles + blockIdx.x] = s_h[threadIdx.x];
}

// exclusive scan of n counters, in place, one block
__global__ void __launch_bounds__(1024) rs_scan_kernel(uint32_t* __restrict__ h, uint64_t n) {
    __shared__ uint32_t s_w[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t carry = 0;
    for (uint64_t base = 0; base < n; base += 4096) {
        const uint64_t i0 = base + 4 * (uint64_t)threadIdx.x;
        uint32_t v[4], s = 0;
#pragma unroll
        for (int e = 0; e < 4; e++) {
            v[e] = i0 + e < n ? h[i0 + e] : 0;
            s += v[e];
        }
        uint32_t inc = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += u;
        }
        if (lane == 31) s_w[warp] = inc;
        __syncthreads();
        if (warp == 0) {
            uint32_t x = s_w[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t u = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += u;
            }
            s_w[lane] = x;  // inclusive
        }
        __syncthreads();
        uint32_t run = carry + (warp ? s_w[warp - 1] : 0) + inc - s;
#pragma unroll
        for (int e = 0; e < 4; e++) {
            if (i0 + e < n) h[i0 + e] = run;
            run += v[e];
        }
        carry += s_w[31];
        __syncthreads();
    }
}

// A warp owns RS_PER * 32 consecutive items and walks them in order, so equal
// digits keep their order: rank among the warp's earlier items of the digit.
__global__ void __launch_bounds__(RS_T) rs_scatter_kernel(const uint64_t* __restrict__ key, uint32_t N, int shift,
                                                          uint32_t n_tiles, const uint32_t* __restrict__ offs,
                                                          uint64_t* __restrict__ out) {
    __shared__ uint32_t s_cnt[RS_T / 32][256];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int w = 0; w < RS_T / 32; w++) s_cnt[w][threadIdx.x] = 0;
    __syncthreads();
    const uint32_t base = blockIdx.x * RS_TILE + warp * (RS_PER * 32);
    uint64_t k[RS_PER];
    uint32_t rank[RS_PER];
#pragma unroll
    for (int i = 0; i < RS_PER; i++) {
        const uint32_t p = base + i * 32 + lane;
        k[i] = p < N ? key[p] : 0;
        const uint32_t d = p < N ? (ta_addr(k[i]) >> shift) & 255 : 256;  // past the end: a digit of its own
        const unsigned same = __match_any_sync(0xffffffffu, d);
        const uint32_t before = d < 256 ? s_cnt[warp][d] : 0;
        rank[i] = before + __popc(same & ((1u << lane) - 1));
        __syncwarp();
        if (d < 256 && lane == __ffs(same) - 1) s_cnt[warp][d] = before + __popc(same);
        __syncwarp();
    }
    __syncthreads();
    {   // first slot of (warp, digit): thread = digit
        uint32_t run = offs[(uint64_t)threadIdx.x * n_tiles + blockIdx.x];
#pragma unroll
        for (int w = 0; w < RS_T / 32; w++) {
            const uint32_t c = s_cnt[w][threadIdx.x];
            s_cnt[w][threadIdx.x] = run;
            run += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < RS_PER; i++) {
        const uint32_t p = base + i * 32 + lane;
        if (p < N) out[s_cnt[warp][(ta_addr(k[i]) >> shift) & 255] + rank[i]] = k[i];
    }
}

// ---- one round ----
struct TaEval {
    int kind;  // 0 read, 1 write
    uint32_t N, bit;
    const uint64_t* key;    // sorted by (addr >> (bit + 1), item)
    uint64_t* key_next;     // the same items for the next round: by (addr >> (bit + 2), item)
    K *wt, *d;
    const K* kc;
    const K* init_tab;      // initial memory, >= 2 entries; before the fold when pending
    int pending;            // bind the previous bit to r first
    K r;
    K* tab_out;             // pending: the folded initial memory, `half` entries
    uint64_t half;
    uint32_t nb;            // evaluation blocks; the others make the next round's order and memory
    K* recs;                // [nb][TA_REC]
    uint32_t* heads;        // [nb] 1: a run starts inside the block
    K* out;                 // the round's values at x = 0, 1, 2
    unsigned int* ticket;
};
constexpr int TA_REC = 8;   // S0..S2, U0..U2, T0, T1

// the last block: the carries into the blocks, and the round's values
__device__ __forceinline__ void ta_carries(const TaEval& a, K (*s_red)[6]) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    __threadfence();
    // carries: inclusive segmented scan of (T0, T1, head) over the blocks, TE_T at a time
    auto ldk = [](const K* q) {
        const ulonglong2 u = __ldcg(reinterpret_cast<const ulonglong2*>(q));
        return gl::kmk(u.x, u.y);
    };
    K sum[3] = {gl::kzero(), gl::kzero(), gl::kzero()};
    K in0 = gl::kzero(), in1 = gl::kzero();  // carried into this batch of blocks
    __shared__ K s_c[2][TE_T];
    __shared__ uint32_t s_f[TE_T];
    for (uint32_t base = 0; base < a.nb; base += TE_T) {
        const uint32_t blk = base + tid;
        const bool on = blk < a.nb;
        const K* r = a.recs + (uint64_t)(on ? blk : 0) * TA_REC;
        K y0 = on ? ldk(r + 6) : gl::kzero(), y1 = on ? ldk(r + 7) : gl::kzero();
        uint32_t f = on ? __ldcg(a.heads + blk) : 0;
        if (tid == 0 && !f) { y0 = gl::kadd(y0, in0); y1 = gl::kadd(y1, in1); }
        const uint32_t live_n = min((uint32_t)TE_T, a.nb - base);
        for (uint32_t o = 1; o < live_n; o <<= 1) {
            s_c[0][tid] = y0; s_c[1][tid] = y1; s_f[tid] = f;
            __syncthreads();
            if ((uint32_t)tid >= o && !f) {
                y0 = gl::kadd(y0, s_c[0][tid - o]);
                y1 = gl::kadd(y1, s_c[1][tid - o]);
                f = s_f[tid - o];
            }
            __syncthreads();
        }
        s_c[0][tid] = y0; s_c[1][tid] = y1;
        __syncthreads();
        const K c0 = tid ? s_c[0][tid - 1] : in0, c1 = tid ? s_c[1][tid - 1] : in1;
        if (on) {
            sum[0] = gl::kadd(sum[0], gl::kadd(ldk(r), gl::kmul(ldk(r + 3), c0)));
            sum[1] = gl::kadd(sum[1], gl::kadd(ldk(r + 1), gl::kmul(ldk(r + 4), c1)));
            sum[2] = gl::kadd(sum[2], gl::kadd(ldk(r + 2), gl::kmul(ldk(r + 5), gl::ksub(gl::kdbl(c1), c0))));
        }
        in0 = s_c[0][TE_T - 1];
        in1 = s_c[1][TE_T - 1];
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 3; i++) {
        K v = sum[i];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = gl::kadd(v, shfl_xor_km(v, o));
        if (lane == 0) s_red[warp][i] = v;
    }
    __syncthreads();
    if (tid < 3) {
        K v = gl::kzero();
        for (int i = 0; i < TE_T / 32; i++) v = gl::kadd(v, s_red[i][tid]);
        a.out[tid] = a.kind == 0 ? v : gl::kneg(v);
    }
}

// positions of the items in the order by (addr >> (bit + 2), item), from the one by
// (addr >> (bit + 1), item): an item moves by the sibling run's items that come before
// it in time.  Its two binary searches (the items before it in the sibling run, and the
// larger block's start, where the runs meet) go side by side, each step's loads in flight
// together: one after the other, a round's values waited for them (an oracle of 2^14 steps
// and 16 address bits: 640 us, now 628).
__device__ __forceinline__ uint32_t ta_merged(const uint64_t* key, uint32_t N, uint32_t bit, uint32_t j, uint64_t k) {
    auto order = [&](uint64_t x) { return (uint64_t)(ta_addr(x) >> (bit + 1)) << 32 | (uint32_t)x; };
    const uint32_t blk = ta_addr(k) >> (bit + 1), sib = blk ^ 1;
    const uint64_t at[2] = {(uint64_t)sib << 32 | (uint32_t)k, (uint64_t)max(blk, sib) << 32};
    uint32_t lo[2] = {0, 0}, hi[2] = {N, N};
    while (lo[0] < hi[0] || lo[1] < hi[1]) {
        uint32_t mid[2];
        uint64_t x[2];
#pragma unroll
        for (int i = 0; i < 2; i++) {
            mid[i] = lo[i] + (hi[i] - lo[i]) / 2;
            x[i] = key[min(mid[i], N - 1)];
        }
#pragma unroll
        for (int i = 0; i < 2; i++) {
            if (lo[i] == hi[i]) continue;
            if (order(x[i]) < at[i]) lo[i] = mid[i] + 1;
            else hi[i] = mid[i];
        }
    }
    return j + lo[0] - lo[1];
}

// a block's part of the round is written; the last of all blocks makes the values
__device__ __forceinline__ void ta_finish(const TaEval& a, K (*s_red)[6]) {
    __shared__ bool s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicInc(a.ticket, gridDim.x - 1) == gridDim.x - 1;
    __syncthreads();
    if (s_last) ta_carries(a, s_red);
}

// Blocks of TE_T sorted items.  A query's contribution at x = 0, 1, 2 is w times
//   child 0:  v0 − k,  0,  −(2 v1 − v0 − k);   child 1:  0,  v1 − k,  2 (2 v1 − v0 − k)
// (negated for the write check), with v0, v1 the initial values plus the prefix
// sums of its run.  For a run that began in an earlier block the block leaves the
// factors U of the two sums carried in (S0 += U0 c0, S1 += U1 c1, S2 += U2 (2 c1
// − c0)) and its own last run's sums T; the last block to finish (ticket, no
// waits) scans the carries over the blocks and adds everything up.
// A round is this one launch: a pending challenge is bound as the weights and the
// initial values are read, and what only the next round reads (the folded initial
// memory; the next order, which no challenge enters: two binary searches an item) is
// the work of further blocks beside the evaluation.  The last block of all writes the
// values, so nothing of the round is left when they are there.  The launch is one chain
// of dependent steps, and with the fold as a launch before it a round's two took 13.1
// and 6.5 us (2^15 items); in one 14.8, of which the next order 0.7.
__global__ void __launch_bounds__(TE_T) ta_eval_kernel(const TaEval a) {
    __shared__ K s_e[2][TE_T];              // exclusive prefix sums over the block (children 0, 1)
    __shared__ K s_w[2][TE_T / 32];
    __shared__ int s_h[TE_T / 32];
    __shared__ K s_red[TE_T / 32][6];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (blockIdx.x >= a.nb) {
        const uint32_t x = (blockIdx.x - a.nb) * TE_T + tid;
        if (a.key_next && x < a.N) {
            const uint64_t key = a.key[x];
            a.key_next[ta_merged(a.key, a.N, a.bit, x, key)] = key;
        }
        if (a.pending)
            for (uint64_t q = x; q < a.half; q += (uint64_t)(gridDim.x - a.nb) * TE_T)
                a.tab_out[q] = gl::klerp(a.init_tab[2 * q], a.init_tab[2 * q + 1], a.r);
        ta_finish(a, s_red);
        return;
    }
    const uint32_t p = blockIdx.x * TE_T + tid;
    const bool live = p < a.N;
    const uint64_t key = live ? a.key[p] : ~0ull;
    const uint32_t addr = ta_addr(key), idx = (uint32_t)key, seg = addr >> (a.bit + 1);
    const int child = (addr >> a.bit) & 1;
    bool head = p == 0;
    if (live && p) head = (ta_addr(a.key[p - 1]) >> (a.bit + 1)) != seg;
    const bool is_q = live && (a.kind == 1 || !(key >> 63)), is_w = live && (a.kind == 1 || (key >> 63));
    K w = live ? a.wt[idx] : gl::kzero();
    K dl = live && a.kind == 1 ? a.d[idx] : gl::kzero();
    K kc = gl::kzero(), i0 = gl::kzero(), i1 = gl::kzero();
    if (is_q) {
        kc = a.kc[idx];
        if (a.pending) {
            const K* t = a.init_tab + 4 * (uint64_t)seg;
            i0 = gl::klerp(t[0], t[1], a.r);
            if (a.half > 1) i1 = gl::klerp(t[2], t[3], a.r);  // one entry left: only x = 0 counts
        } else {
            i0 = a.init_tab[2 * (uint64_t)seg];
            i1 = a.init_tab[2 * (uint64_t)seg + 1];
        }
    }
    if (a.pending && live) {  // an item is one thread's
        const K f = ((addr >> (a.bit - 1)) & 1) ? a.r : gl::ksub(gl::kone(), a.r);
        w = gl::kmul(w, f);
        a.wt[idx] = w;
        if (a.kind == 1) {
            dl = gl::kmul(dl, f);
            a.d[idx] = dl;
        }
    }
    dl = !is_w ? gl::kzero() : a.kind == 1 ? dl : w;
    // inclusive scans of the two children's deltas and of the last head's position
    K x0 = child ? gl::kzero() : dl, x1 = child ? dl : gl::kzero();
    const K own0 = x0, own1 = x1;
    int h = live && head ? tid : -1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        K n0, n1;
        n0.re = __shfl_up_sync(0xffffffffu, x0.re, o); n0.im = __shfl_up_sync(0xffffffffu, x0.im, o);
        n1.re = __shfl_up_sync(0xffffffffu, x1.re, o); n1.im = __shfl_up_sync(0xffffffffu, x1.im, o);
        const int hh = __shfl_up_sync(0xffffffffu, h, o);
        if (lane >= o) {
            x0 = gl::kadd(x0, n0);
            x1 = gl::kadd(x1, n1);
            h = max(h, hh);
        }
    }
    if (lane == 31) { s_w[0][warp] = x0; s_w[1][warp] = x1; s_h[warp] = h; }
    __syncthreads();
    K b0 = gl::kzero(), b1 = gl::kzero(), t0 = gl::kzero(), t1 = gl::kzero();  // before this warp; the block's total
    int last_head = -1;
#pragma unroll 1
    for (int i = 0; i < TE_T / 32; i++) {
        if (i == warp) { b0 = t0; b1 = t1; h = max(h, last_head); }
        t0 = gl::kadd(t0, s_w[0][i]);
        t1 = gl::kadd(t1, s_w[1][i]);
        last_head = max(last_head, s_h[i]);
    }
    const K e0 = gl::kadd(b0, gl::ksub(x0, own0)), e1 = gl::kadd(b1, gl::ksub(x1, own1));
    s_e[0][tid] = e0;
    s_e[1][tid] = e1;
    __syncthreads();
    const bool open = h < 0;
    K c[6];
#pragma unroll
    for (int i = 0; i < 6; i++) c[i] = gl::kzero();
    if (is_q) {
        const K v0 = gl::kadd(i0, open ? e0 : gl::ksub(e0, s_e[0][h])), v1 = gl::kadd(i1, open ? e1 : gl::ksub(e1, s_e[1][h]));
        const K w2 = child ? gl::kdbl(w) : gl::kneg(w);
        const K near = gl::kmul(w, gl::ksub(child ? v1 : v0, kc));
        c[0] = child ? gl::kzero() : near;
        c[1] = child ? near : gl::kzero();
        c[2] = gl::kmul(w2, gl::ksub(gl::ksub(gl::kdbl(v1), v0), kc));
        if (open) {
            c[3] = child ? gl::kzero() : w;
            c[4] = child ? w : gl::kzero();
            c[5] = w2;
        }
    }
    const bool any_open = __syncthreads_or(is_q && open);
    const int nc = any_open ? 6 : 3;
#pragma unroll
    for (int i = 0; i < 6; i++) {
        if (i >= nc) break;
        K v = c[i];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = gl::kadd(v, shfl_xor_km(v, o));
        if (lane == 0) s_red[warp][i] = v;
    }
    __syncthreads();
    K* rec = a.recs + (uint64_t)blockIdx.x * TA_REC;
    if (tid < 6) {
        K v = gl::kzero();
        if (tid < nc)
            for (int i = 0; i < TE_T / 32; i++) v = gl::kadd(v, s_red[i][tid]);
        rec[tid] = v;
    } else if (tid < 8) {
        const int ch = tid - 6;
        const K tot = ch ? t1 : t0;
        rec[tid] = last_head < 0 ? tot : gl::ksub(tot, s_e[ch][last_head]);
    } else if (tid == 8) {
        a.heads[blockIdx.x] = last_head >= 0;
    }
    ta_finish(a, s_red);
}

// One fold of the address lane by itself (a second fold without an evaluation in
// between, or no items): item j's weights by its own bit, the initial-memory table on
// its low address bit, and the items' order.
struct TaFold {
    uint32_t N, bit;
    int kind;
    K r;
    const uint64_t* key;
    uint64_t* key_out;
    K *wt, *d;
    const K* tab;
    K* tab_out;
    uint64_t half;
};
__global__ void __launch_bounds__(256) ta_fold_kernel(const TaFold a) {
    const uint64_t j = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (j >= a.N) {
        const uint64_t q = j - a.N;
        if (q < a.half) a.tab_out[q] = gl::klerp(a.tab[2 * q], a.tab[2 * q + 1], a.r);
        return;
    }
    const uint64_t key = a.key[j];
    const uint32_t idx = (uint32_t)key;
    const K f = ((ta_addr(key) >> a.bit) & 1) ? a.r : gl::ksub(gl::kone(), a.r);
    a.wt[idx] = gl::kmul(a.wt[idx], f);
    if (a.kind == 1) a.d[idx] = gl::kmul(a.d[idx], f);
    a.key_out[ta_merged(a.key, a.N, a.bit, (uint32_t)j, key)] = key;
}

__global__ void scatter_init_kernel(const uint64_t* __restrict__ addr, const K* __restrict__ val, uint64_t n,
                                    K* __restrict__ tab) {
    uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i < n) tab[addr[i]] = val[i];
}

}  // namespace

struct neo_gpu_twist_addr {
    neo_gpu_ctx* ctx = nullptr;
    int kind = 0;
    uint32_t A = 0, bit = 0, N = 0;  // N items
    DevBuf<uint64_t> key[2];
    int kcur = 0;
    DevBuf<K> wt, kc, d, tab[2], recs;
    DevBuf<uint32_t> heads, hist;
    DevBuf<unsigned int> ticket;     // ta_eval_kernel's block counter (returns to zero after every launch)
    DevBuf<K> dcols, dr, dv;         // build workspace, kept for reuse
    DevBuf<uint32_t> counts;
    DevBuf<uint64_t> da;
    uint64_t tab_len = 0;
    int cur = 0;
    bool pending = false;
    bool next_order = false;         // key[kcur ^ 1] holds the order after the next fold
    K pending_r{};
    std::vector<K> hvals;
};

namespace {

int ta_apply_fold(neo_gpu_twist_addr* o) {
    neo_gpu_ctx* ctx = o->ctx;
    const uint64_t half = o->tab_len >> 1;
    const uint64_t n = o->N + half;
    if (n) {
        TaFold a;
        a.N = o->N; a.bit = o->bit; a.kind = o->kind; a.r = o->pending_r;
        a.key = o->key[o->kcur].p; a.key_out = o->key[o->kcur ^ 1].p;
        a.wt = o->wt.p; a.d = o->d.p;
        a.tab = o->tab[o->cur].p; a.tab_out = o->tab[o->cur ^ 1].p; a.half = half;
        ta_fold_kernel<<<ceil_div(n, 256), 256, 0, ctx->stream>>>(a);
        NEO_LAUNCHED(ctx);
    }
    o->kcur ^= 1;
    o->cur ^= 1;
    o->tab_len = half;
    o->bit++;
    o->pending = false;
    o->next_order = false;
    return NEO_OK;
}

// The round's values at x = 0, 1, 2 into dst (page-locked host memory that the caller
// polls, so every word is one store), without a host sync (the pending fold applied
// first); no items: zeros, by the host.
int ta_values_launch(neo_gpu_twist_addr* o, K* dst) {
    neo_gpu_ctx* ctx = o->ctx;
    cudaStream_t S = ctx->stream;
    // the launch binds the challenge itself once the order is there
    const bool fused = o->pending && o->next_order && o->N;
    if (o->pending && !fused) {
        int rc = ta_apply_fold(o);
        if (rc) return rc;
    }
    if (o->N == 0) {
        for (int x = 0; x < 3; x++) dst[x] = gl::kzero();
        return NEO_OK;
    }
    const uint32_t nb = ceil_div(o->N, TE_T);
    TaEval a{};
    if (fused) {
        a.pending = 1;
        a.r = o->pending_r;
        a.half = o->tab_len >> 1;
        a.tab_out = o->tab[o->cur ^ 1].p;
        o->kcur ^= 1;
        o->bit++;
    }
    a.kind = o->kind;
    a.N = o->N;
    a.bit = o->bit;
    a.key = o->key[o->kcur].p;
    a.key_next = o->bit < o->A ? o->key[o->kcur ^ 1].p : nullptr;
    a.wt = o->wt.p; a.kc = o->kc.p; a.d = o->d.p;
    a.init_tab = o->tab[o->cur].p;
    a.recs = o->recs.p;
    a.heads = o->heads.p;
    a.out = dst;
    a.ticket = o->ticket.p;
    a.nb = nb;
    // blocks of the next order (an item a thread) and of the folded memory
    uint32_t extra = a.key_next ? nb : 0;
    if (a.pending) extra = std::max(extra, (uint32_t)std::min<uint64_t>(ceil_div(a.half, TE_T), 148));
    ta_eval_kernel<<<nb + extra, TE_T, 0, S>>>(a);
    NEO_LAUNCHED(ctx);
    if (fused) {
        o->cur ^= 1;
        o->tab_len >>= 1;
        o->pending = false;
    }
    o->next_order = a.key_next != nullptr;
    return NEO_OK;
}

int ta_values(neo_gpu_twist_addr* o) {
    neo_gpu_ctx* ctx = o->ctx;
    o->hvals.assign(3, gl::kzero());
    if (o->N == 0) return o->pending ? ta_apply_fold(o) : NEO_OK;
    K* out = reinterpret_cast<K*>(ctx->h_result);
    result_arm(out, 6);
    if (int rc = ta_values_launch(o, out)) return rc;
    NEO_CK(ctx, result_wait(ctx, out, 6));
    o->hvals.assign(out, out + 3);
    return NEO_OK;
}

int ta_create(neo_gpu_ctx* ctx, int kind, uint32_t ell, const uint64_t* r_cycle, uint32_t A, uint64_t n_init,
              const uint64_t* init_addr, const uint64_t* init_val, const uint64_t* cols, bool dev,
              neo_gpu_twist_addr** out, bool reuse = false) {
    if (!ctx || !out) return NEO_ERR_ARG;
    if (!reuse) *out = nullptr;
    if (kind != 0 && kind != 1) return ctx->fail(NEO_ERR_ARG, "twist_addr: kind must be 0 (read) or 1 (write)");
    if (ell > 30 || A > 30 || A == 0) return ctx->fail(NEO_ERR_ARG, "twist_addr: ell / ell_addr out of range");
    if (!cols || (ell && !r_cycle) || (n_init && (!init_addr || !init_val)))
        return ctx->fail(NEO_ERR_ARG, "twist_addr: null buffer");
    for (uint64_t i = 0; i < n_init; i++)
        if (init_addr[i] >> A) return ctx->fail(NEO_ERR_ARG, "twist_addr: init address out of range");
    cudaSetDevice(ctx->device);
    PoolScope pool_scope(ctx);
    cudaStream_t S = ctx->stream;
    const uint64_t L = 1ULL << ell, P = 1ULL << A;
    const uint32_t n_cols = kind == 0 ? 4 + 2 * A : 3 + A;
    neo_gpu_twist_addr* o = reuse ? *out : nullptr;
    const bool fresh = !o;
    if (fresh) o = new neo_gpu_twist_addr();
    o->ctx = ctx;
    o->kind = kind;
    o->A = A;
    o->bit = 0;
    o->cur = 0;
    o->kcur = 0;
    o->pending = o->next_order = false;
    auto fail = [&](int rc) {
        if (fresh) delete o;
        return rc;
    };
    DevBuf<K>& dcols = o->dcols;
    DevBuf<K>& dr = o->dr;
    const K* C = reinterpret_cast<const K*>(cols);
    if (!dev) {
        if (dcols.ensure((size_t)n_cols * L)) return fail(ctx->fail(NEO_ERR_OOM, "twist_addr: columns"));
        if (cudaMemcpyAsync(dcols.p, cols, (size_t)n_cols * L * sizeof(K), cudaMemcpyHostToDevice, S))
            return fail(ctx->fail(NEO_ERR_CUDA, "twist_addr: column upload"));
        C = dcols.p;
    }
    if (dr.ensure(ell ? ell : 1)) return fail(ctx->fail(NEO_ERR_OOM, "twist_addr: r"));
    if (ell && cudaMemcpyAsync(dr.p, r_cycle, ell * sizeof(K), cudaMemcpyHostToDevice, S))
        return fail(ctx->fail(NEO_ERR_CUDA, "twist_addr: r upload"));
    TaBuild b{};
    if (kind == 0) {
        b.hr = C; b.rv = C + L; b.ra = C + 2 * L; b.hw = C + (2 + A) * L; b.inc = C + (3 + A) * L; b.wa = C + (4 + A) * L;
    } else {
        b.hw = C; b.wv = C + L; b.inc = C + 2 * L; b.wa = C + 3 * L;
    }
    const uint32_t nblk = ceil_div(L, TA_T);
    DevBuf<uint32_t>& counts = o->counts;
    if (counts.ensure(nblk)) return fail(ctx->fail(NEO_ERR_OOM, "twist_addr: counts"));
    ta_count_kernel<<<nblk, TA_T, 0, S>>>(b.hr, b.hw, L, counts.p);
    NEO_LAUNCHED(ctx);
    std::vector<uint32_t> hc(nblk);
    NEO_CK(ctx, ctx_d2h(ctx, hc.data(), counts.p, nblk * 4));
    NEO_CK(ctx, ctx_sync(ctx));
    uint64_t N = 0;
    for (auto& c : hc) { uint32_t v = c; c = (uint32_t)N; N += v; }
    if (N > 0x7FFFFFFFull) return fail(ctx->fail(NEO_ERR_UNSUPPORTED, "twist_addr: too many events"));
    o->N = (uint32_t)N;
    const size_t cap = N ? N : 1;
    const uint32_t n_tiles = ceil_div(cap, RS_TILE), nb = ceil_div(cap, TE_T);
    if (o->key[0].ensure(cap) || o->key[1].ensure(cap) || o->wt.ensure(cap) || o->kc.ensure(cap) ||
        (kind == 1 && o->d.ensure(cap)) || o->recs.ensure((size_t)nb * TA_REC) || o->heads.ensure(nb) ||
        o->hist.ensure((size_t)n_tiles * 256) || o->ticket.ensure(1) ||
        o->tab[0].ensure(P + 1) || o->tab[1].ensure(P / 2 + 1))
        return fail(ctx->fail(NEO_ERR_OOM, "twist_addr: event arrays"));
    NEO_CK(ctx, cudaMemsetAsync(o->ticket.p, 0, sizeof(unsigned int), S));
    NEO_CK(ctx, cudaMemcpyAsync(counts.p, hc.data(), nblk * 4, cudaMemcpyHostToDevice, S));
    b.r_cycle = dr.p; b.ell = ell; b.A = A; b.L = L; b.offs = counts.p;
    b.key = o->key[0].p; b.wt = o->wt.p; b.kc = o->kc.p; b.d = o->d.p;
    ta_build_kernel<<<nblk, TA_T, 0, S>>>(b);
    NEO_LAUNCHED(ctx);
    // round 0's order: by address bits 1..A-1, items of a run in time order
    for (uint32_t sh = 1; sh < A && N; sh += 8) {
        rs_hist_kernel<<<n_tiles, RS_T, 0, S>>>(o->key[o->kcur].p, o->N, (int)sh, n_tiles, o->hist.p);
        NEO_LAUNCHED(ctx);
        rs_scan_kernel<<<1, 1024, 0, S>>>(o->hist.p, (uint64_t)n_tiles * 256);
        NEO_LAUNCHED(ctx);
        rs_scatter_kernel<<<n_tiles, RS_T, 0, S>>>(o->key[o->kcur].p, o->N, (int)sh, n_tiles, o->hist.p, o->key[o->kcur ^ 1].p);
        NEO_LAUNCHED(ctx);
        o->kcur ^= 1;
    }
    // initial memory as a dense table over the 2^A addresses (plus one zero pad)
    NEO_CK(ctx, cudaMemsetAsync(o->tab[0].p, 0, (P + 1) * sizeof(K), S));
    NEO_CK(ctx, cudaMemsetAsync(o->tab[1].p, 0, (P / 2 + 1) * sizeof(K), S));
    if (n_init) {
        DevBuf<uint64_t>& da = o->da;
        DevBuf<K>& dv = o->dv;
        if (da.ensure(n_init) || dv.ensure(n_init)) return fail(ctx->fail(NEO_ERR_OOM, "twist_addr: init"));
        NEO_CK(ctx, cudaMemcpyAsync(da.p, init_addr, n_init * 8, cudaMemcpyHostToDevice, S));
        NEO_CK(ctx, cudaMemcpyAsync(dv.p, init_val, n_init * sizeof(K), cudaMemcpyHostToDevice, S));
        scatter_init_kernel<<<ceil_div(n_init, 256), 256, 0, S>>>(da.p, dv.p, n_init, o->tab[0].p);
        NEO_LAUNCHED(ctx);
    }
    o->tab_len = P;
    NEO_CK(ctx, ctx_sync(ctx));
    *out = o;
    return NEO_OK;
}

}  // namespace

// Rebuild into *slot when it holds an oracle (buffers kept), else create;
// columns in device memory (the fold step's per-step path).
int twist_addr_build_device(neo_gpu_ctx* ctx, int kind, uint32_t ell, const uint64_t* r_cycle, uint32_t ell_addr,
                            uint64_t n_init, const uint64_t* init_addr, const uint64_t* init_val,
                            const uint64_t* d_cols, neo_gpu_twist_addr** slot) {
    return ta_create(ctx, kind, ell, r_cycle, ell_addr, n_init, init_addr, init_val, d_cols, true, slot, true);
}

static int neo_gpu_twist_addr_create_impl_abi(neo_gpu_ctx* ctx, int kind, uint32_t ell, const uint64_t* r_cycle,
                                         uint32_t ell_addr, uint64_t n_init, const uint64_t* init_addr,
                                         const uint64_t* init_val, const uint64_t* cols, neo_gpu_twist_addr** out) {
    return ta_create(ctx, kind, ell, r_cycle, ell_addr, n_init, init_addr, init_val, cols, false, out);
}
extern "C" int neo_gpu_twist_addr_create(neo_gpu_ctx* ctx, int kind, uint32_t ell, const uint64_t* r_cycle,
                                         uint32_t ell_addr, uint64_t n_init, const uint64_t* init_addr,
                                         const uint64_t* init_val, const uint64_t* cols, neo_gpu_twist_addr** out) { NEO_ABI_GUARD(neo_gpu_twist_addr_create_impl_abi(ctx, kind, ell, r_cycle, ell_addr, n_init, init_addr, init_val, cols, out)) }

static int neo_gpu_twist_addr_create_device_impl_abi(neo_gpu_ctx* ctx, int kind, uint32_t ell, const uint64_t* r_cycle,
                                                uint32_t ell_addr, uint64_t n_init, const uint64_t* init_addr,
                                                const uint64_t* init_val, const uint64_t* d_cols,
                                                neo_gpu_twist_addr** out) {
    return ta_create(ctx, kind, ell, r_cycle, ell_addr, n_init, init_addr, init_val, d_cols, true, out);
}
extern "C" int neo_gpu_twist_addr_create_device(neo_gpu_ctx* ctx, int kind, uint32_t ell, const uint64_t* r_cycle,
                                                uint32_t ell_addr, uint64_t n_init, const uint64_t* init_addr,
                                                const uint64_t* init_val, const uint64_t* d_cols,
                                                neo_gpu_twist_addr** out) { NEO_ABI_GUARD(neo_gpu_twist_addr_create_device_impl_abi(ctx, kind, ell, r_cycle, ell_addr, n_init, init_addr, init_val, d_cols, out)) }

// The next round of a Twist address-lane oracle into dst[0..3) (page-locked),
// without a host sync; false (nothing launched) once every address bit is
// bound, when the value no longer depends on x.
int ta_round_launch(neo_gpu_twist_addr* o, K* dst, bool* launched) {
    *launched = false;
    if (o->bit + (o->pending ? 1 : 0) >= o->A) return NEO_OK;
    cudaSetDevice(o->ctx->device);
    if (int rc = ta_values_launch(o, dst)) return rc;
    *launched = true;
    return NEO_OK;
}

static int neo_gpu_twist_addr_evals_impl_abi(neo_gpu_twist_addr* o, const uint64_t* xs, uint32_t nx, uint64_t* ys) {
    if (!o) return NEO_ERR_ARG;
    if ((!xs || !ys) && nx) return o->ctx->fail(NEO_ERR_ARG, "twist_addr_evals: null buffer");
    cudaSetDevice(o->ctx->device);
    PoolScope pool_scope(o->ctx);
    int rc = ta_values(o);
    if (rc) return rc;
    for (uint32_t i = 0; i < nx; i++) {
        // after the last round the value does not depend on x (the reference's constant branch)
        K y = o->bit >= o->A ? o->hvals[0] : lagrange_at(o->hvals, kload_h(xs + 2 * i));
        ys[2 * i] = y.re;
        ys[2 * i + 1] = y.im;
    }
    return NEO_OK;
}
extern "C" int neo_gpu_twist_addr_evals(neo_gpu_twist_addr* o, const uint64_t* xs, uint32_t nx, uint64_t* ys) { NEO_ABI_GUARD(neo_gpu_twist_addr_evals_impl_abi(o, xs, nx, ys)) }

static int neo_gpu_twist_addr_fold_impl_abi(neo_gpu_twist_addr* o, const uint64_t* r) {
    if (!o) return NEO_ERR_ARG;
    if (!r) return o->ctx->fail(NEO_ERR_ARG, "twist_addr_fold: null challenge");
    const uint32_t done = o->bit + (o->pending ? 1 : 0);
    if (done >= o->A) return NEO_OK;
    cudaSetDevice(o->ctx->device);
    if (o->pending) {
        int rc = ta_apply_fold(o);
        if (rc) return rc;
    }
    o->pending = true;
    o->pending_r = kload_h(r);
    return NEO_OK;
}
extern "C" int neo_gpu_twist_addr_fold(neo_gpu_twist_addr* o, const uint64_t* r) { NEO_ABI_GUARD(neo_gpu_twist_addr_fold_impl_abi(o, r)) }

extern "C" uint32_t neo_gpu_twist_addr_num_rounds(const neo_gpu_twist_addr* o) {
    return o ? o->A - o->bit - (o->pending ? 1 : 0) : 0;
}
extern "C" uint32_t neo_gpu_twist_addr_degree_bound(const neo_gpu_twist_addr* o) { return o ? 2 : 0; }

static int neo_gpu_twist_addr_destroy_impl_abi(neo_gpu_twist_addr* o) {
    if (!o) return NEO_OK;
    cudaSetDevice(o->ctx->device);
    neo_gpu_ctx* ctx = o->ctx;
    cudaStreamSynchronize(ctx->stream);
    delete o;
    pool_trim(ctx);
    return NEO_OK;
}
extern "C" int neo_gpu_twist_addr_destroy(neo_gpu_twist_addr* o) { NEO_ABI_GUARD(neo_gpu_twist_addr_destroy_impl_abi(o)) }
