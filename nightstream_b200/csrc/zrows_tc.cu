// zrows_tc.cu -- y[row][j] = sum_c Z[row][c] v[j][c] of many int8 digit rows on the
// tensor cores (tcgen05 kind::i8), exact.
//
// The ME outputs y = Z M_j^T chi_r of compute_y_from_Z_and_r
// (crates/neo-reductions/src/common.rs:582-650): A = 128 digit rows (s8), B = the 16 t
// byte limbs of the t vectors (u8), D = s32 limb sums; the epilogue of a row is then
// sum_l 2^(8 l) D[l] mod q per component.  |D| <= 128 * 255 * ZT_MAX_COLS < 2^31.
//
// A block holds 128 rows and a range of columns.  Per chunk of 128 columns its threads
// copy the digits (16 bytes each, eight lanes a row: whole 128-byte lines) into the
// 128B-swizzled K-major tile, and one warp per vector turns the 16-byte elements of four
// columns into 16 words of limbs by byte permutes; the next chunk's loads are in flight
// meanwhile, and three blocks per SM hide the rest.  The rows' digits are read once:
// memory bounds it (13 witnesses of 2^16 columns: 46 MB).  As signed sums of tabulated
// column pairs, on the CUDA cores, it took 142 us there and 403 us at 2^18 columns and
// 12 witnesses (table builds and six 64-bit adds with carry a pair); now 23 and 45 to 54.
//
// Blocks add their range's sums into per-(row, j) 64-bit accumulators with atomics (a
// wrap past 2^64 counted apart: exact and order-free); the last block of a row group
// (ticket) reduces them.
#include <algorithm>
#include "internal.cuh"
#include "tc.cuh"

namespace {

using gl::K;

constexpr int ZT_ROWS = 128, ZT_COLS = 128, ZT_T = 256, ZT_TMAX = 4;
constexpr int ZT_A = ZT_ROWS * ZT_COLS, ZT_B = ZT_TMAX * 16 * ZT_COLS, ZT_STAGE = ZT_A + ZT_B;
constexpr uint64_t ZT_MAX_COLS = 1u << 16;
constexpr uint32_t ZT_TMEM = 64;  // columns: 16 t, a power of two
static_assert(ZT_A % 1024 == 0 && ZT_B % 1024 == 0, "swizzle atoms are 1024-byte aligned");

// Row r = (w ncols + c) 54 + rho is n bytes at Z + (w 54 + rho) m + base + c n (whole
// digit rows: ncols = 1, base = 0, n = m)
struct ZrowsArgs {
    const int8_t* Z;
    uint64_t m, base;
    uint32_t ncols;
    uint32_t R, t;
    uint64_t n;        // columns, a multiple of 16; every row begins on 16 bytes
    const K* v;        // [t][n]
    uint64_t cols;     // columns per block, a multiple of ZT_COLS
    unsigned long long* acc_lo;  // [R][t][2], zero
    unsigned int* acc_wrap;      // [R][t][2], zero
    unsigned int* tickets;       // [row groups], zero
    K* y;              // [R / 54][t][54], R a multiple of 54
    volatile uint32_t* err;  // page-locked: set when a wait gives up
};

__global__ void __launch_bounds__(ZT_T, 3) zrows_tc_kernel(const ZrowsArgs a) {
    extern __shared__ uint8_t s_raw[];
    __shared__ __align__(8) uint64_t s_done[2];  // MMAs of a stage complete
    __shared__ uint32_t s_tmem;
    __shared__ unsigned int s_last;
    uint8_t* stages = s_raw + ((1024 - (smem_u32(s_raw) & 1023)) & 1023);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t row0 = blockIdx.x * ZT_ROWS, t = a.t;
    const uint64_t c_lo = blockIdx.y * a.cols, c_hi = min(a.n, c_lo + a.cols);
    const uint32_t n = (uint32_t)((c_hi - c_lo + ZT_COLS - 1) / ZT_COLS);
    if (tid == 0) {
        mbar_init(&s_done[0], 1);
        mbar_init(&s_done[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tmem_alloc<ZT_TMEM>(&s_tmem);
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = s_tmem;

    // thread: 16 bytes at column 16 (tid & 7) of rows tid / 8 + 32 e; warp j < t: columns
    // 4 lane .. 4 lane + 3 of vector j
    uint4 za[4];
    uint4 vb[4];
    const uint32_t ak = (tid & 7) * 16, ar = tid >> 3;
    const int8_t* zr[4];  // null: no such row
#pragma unroll
    for (int e = 0; e < 4; e++) {
        const uint32_t r = row0 + ar + 32 * e, q = r / NEO_D;
        zr[e] = r < a.R ? a.Z + ((uint64_t)(q / a.ncols) * NEO_D + r % NEO_D) * a.m + a.base + (uint64_t)(q % a.ncols) * a.n : nullptr;
    }
    auto fetch = [&](uint32_t i) {
        const uint64_t c = c_lo + (uint64_t)i * ZT_COLS;
#pragma unroll
        for (int e = 0; e < 4; e++) {
            za[e] = zr[e] && c + ak < c_hi ? __ldg(reinterpret_cast<const uint4*>(zr[e] + c + ak)) : make_uint4(0, 0, 0, 0);
        }
        if (warp < (int)t) {
            const uint64_t cv = c + 4 * lane;
#pragma unroll
            for (int e = 0; e < 4; e++)
                vb[e] = cv < c_hi ? __ldg(reinterpret_cast<const uint4*>(a.v + (uint64_t)warp * a.n + cv + e)) : make_uint4(0, 0, 0, 0);
        }
    };
    if (n) fetch(0);
    uint32_t issued = 0;
    const uint32_t id = idesc_i8(16 * (int)t, true, false);
    for (uint32_t i = 0; i < n; i++) {
        uint8_t* A = stages + (i & 1) * ZT_STAGE;
        uint8_t* B = A + ZT_A;
        bool ok = true;
        if (i >= 2 && lane == 0) ok = mbar_wait(&s_done[i & 1], ((i >> 1) & 1) ^ 1);
        __syncwarp();
#pragma unroll
        for (int e = 0; e < 4; e++) *reinterpret_cast<uint4*>(A + sw128_at(ar + 32 * e, ak)) = za[e];
        if (warp < (int)t) {
            const uint32_t w[4][4] = {{vb[0].x, vb[1].x, vb[2].x, vb[3].x}, {vb[0].y, vb[1].y, vb[2].y, vb[3].y},
                                      {vb[0].z, vb[1].z, vb[2].z, vb[3].z}, {vb[0].w, vb[1].w, vb[2].w, vb[3].w}};
#pragma unroll
            for (int q = 0; q < 4; q++) {  // 4 x 4 byte transposition: limbs 4 q .. 4 q + 3
                const uint32_t lo01 = __byte_perm(w[q][0], w[q][1], 0x5140), lo23 = __byte_perm(w[q][2], w[q][3], 0x5140);
                const uint32_t hi01 = __byte_perm(w[q][0], w[q][1], 0x7362), hi23 = __byte_perm(w[q][2], w[q][3], 0x7362);
                const uint32_t o[4] = {__byte_perm(lo01, lo23, 0x5410), __byte_perm(lo01, lo23, 0x7632),
                                       __byte_perm(hi01, hi23, 0x5410), __byte_perm(hi01, hi23, 0x7632)};
#pragma unroll
                for (int b = 0; b < 4; b++) *reinterpret_cast<uint32_t*>(B + sw128_at(warp * 16 + 4 * q + b, 4 * lane)) = o[b];
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        if (i + 1 < n) fetch(i + 1);
        if (__syncthreads_or(!ok)) break;  // block-uniform
        issued++;
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;");
            const uint32_t a0 = smem_u32(A), b0 = smem_u32(B);
#pragma unroll
            for (int k = 0; k < 4; k++) mma_i8(tmem, sw128_desc(a0 + 32 * k), sw128_desc(b0 + 32 * k), id, (i > 0 || k > 0) ? 1u : 0u);
            mma_commit(&s_done[i & 1]);
        }
    }
    // the last commit covers every MMA of the block (waited for after a failed wait too,
    // before the TMEM goes back)
    uint32_t okw = 1;
    if (lane == 0 && issued) {
        okw = mbar_wait(&s_done[(issued - 1) & 1], ((issued - 1) >> 1) & 1) && issued == n ? 1u : 0u;
        if (!okw) *a.err = 0x40u;
    }
    okw = __shfl_sync(0xffffffffu, okw, 0);
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t row = row0 + (warp & 3) * 32 + lane;
    for (uint32_t j = warp >> 2; j < (okw && n ? t : 0); j += 2) {
        int x[16];
        const uint32_t taddr = tmem + ((uint32_t)((warp & 3) * 32) << 16) + 16 * j;
        tmem_ld(taddr, x);
        if (row >= a.R) continue;
#pragma unroll
        for (int e = 0; e < 2; e++) {
            // sum_l 2^(8 l) x_l as lo + 2^32 hi, |lo|, |hi| < 2^56
            int64_t lo = 0, hi = 0;
#pragma unroll
            for (int l = 3; l >= 0; l--) {
                lo = lo * 256 + x[8 * e + l];
                hi = hi * 256 + x[8 * e + 4 + l];
            }
            const uint64_t c = gl::add(gl::from_i64(lo), gl::mul(gl::from_i64(hi), 1ull << 32));
            const uint64_t at = ((uint64_t)row * t + j) * 2 + e;
            if (c == 0) continue;
            const unsigned long long old = atomicAdd(a.acc_lo + at, (unsigned long long)c);
            if (old + c < old) atomicAdd(a.acc_wrap + at, 1u);
        }
    }
    __threadfence();
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;");
        tmem_dealloc<ZT_TMEM>(tmem);
    }
    if (tid == 0) s_last = atomicInc(a.tickets + blockIdx.x, gridDim.y - 1) == gridDim.y - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (uint32_t i = tid; i < ZT_ROWS * t; i += ZT_T) {
        const uint32_t r = row0 + i / t, j = i % t;
        if (r >= a.R) break;
        uint64_t c[2];
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const uint64_t at = ((uint64_t)r * t + j) * 2 + e;
            // lo + 2^64 wraps (mod q), 2^64 = 2^32 - 1; wraps < 2^32, so the product is below 2^64
            c[e] = gl::add(gl::canon(__ldcg(a.acc_lo + at)), gl::canon((uint64_t)__ldcg(a.acc_wrap + at) * 0xFFFFFFFFull));
        }
        a.y[((uint64_t)(r / NEO_D) * t + j) * NEO_D + r % NEO_D] = gl::kmk(c[0], c[1]);
    }
}

static int zrows_launch(neo_gpu_ctx* ctx, ZrowsArgs a) {
    const uint32_t groups = (a.R + ZT_ROWS - 1) / ZT_ROWS;
    const uint64_t chunks = (a.n + ZT_COLS - 1) / ZT_COLS;
    // three blocks per SM, as many as are resident
    uint64_t splits = std::min<uint64_t>(chunks, std::max<uint64_t>(1, 3 * 148 / groups));
    a.cols = std::min<uint64_t>((chunks + splits - 1) / splits * ZT_COLS, ZT_MAX_COLS);
    splits = (a.n + a.cols - 1) / a.cols;
    // accumulators and tickets, cleared together
    const size_t n_acc = (size_t)a.R * a.t * 2, lo_bytes = n_acc * 8, wrap_bytes = n_acc * 4;
    void* scratch = nullptr;
    NEO_CK(ctx, ctx_scratch(ctx, lo_bytes + wrap_bytes + groups * sizeof(unsigned int), &scratch));
    uint8_t* sb = reinterpret_cast<uint8_t*>(scratch);
    NEO_CK(ctx, cudaMemsetAsync(sb, 0, lo_bytes + wrap_bytes + groups * sizeof(unsigned int), ctx->stream));
    a.acc_lo = reinterpret_cast<unsigned long long*>(sb);
    a.acc_wrap = reinterpret_cast<unsigned int*>(sb + lo_bytes);
    a.tickets = reinterpret_cast<unsigned int*>(sb + lo_bytes + wrap_bytes);
    a.err = ctx_host_err(ctx);
    constexpr size_t smem = 2 * ZT_STAGE + 1024;
    static SmemLimit limit;
    NEO_CK(ctx, limit.at_least(zrows_tc_kernel, smem));
    zrows_tc_kernel<<<dim3(groups, (uint32_t)splits), ZT_T, smem, ctx->stream>>>(a);
    NEO_LAUNCHED(ctx);
    return NEO_OK;
}

}  // namespace

// y of R digit rows (layout [w][t][54], row = w * 54 + rho); *done = false when the
// shape does not suit the kernel (the caller keeps its own): rows that are not 64-byte
// aligned, or more than four vectors
int launch_zrows(neo_gpu_ctx* ctx, const int8_t* d_Z, uint32_t R, uint64_t m, uint32_t t, const K* d_v, K* d_y,
                 bool* done) {
    *done = false;
    if (t == 0 || t > ZT_TMAX || m % 64 || m == 0 || R == 0) return NEO_OK;
    if ((reinterpret_cast<uintptr_t>(d_Z) & 15) || (reinterpret_cast<uintptr_t>(d_v) & 15)) return NEO_OK;
    ZrowsArgs a{};
    a.Z = d_Z;
    a.m = a.n = m;
    a.ncols = 1;
    a.R = R;
    a.t = t;
    a.v = d_v;
    a.y = d_y;
    *done = true;
    return zrows_launch(ctx, a);
}

// Bus openings y[w][c][rho] = sum_j Z[w 54 + rho][base + c steps + j] v[j] of n_w
// witnesses and ncols chunks of `steps` digits; *done = false when a chunk does not
// begin on 16 bytes in every row
int launch_bus_rows(neo_gpu_ctx* ctx, const int8_t* d_Z, uint32_t n_w, uint64_t m, uint64_t base, uint64_t steps,
                    uint32_t ncols, const K* d_v, K* d_y, bool* done) {
    *done = false;
    if (steps == 0 || ncols == 0 || m % 16 || base % 16 || steps % 16) return NEO_OK;
    if ((reinterpret_cast<uintptr_t>(d_Z) & 15) || (reinterpret_cast<uintptr_t>(d_v) & 15)) return NEO_OK;
    if ((uint64_t)n_w * ncols * NEO_D > 0x7FFFFFFFull) return NEO_OK;
    ZrowsArgs a{};
    a.Z = d_Z;
    a.m = m;
    a.base = base;
    a.ncols = ncols;
    a.n = steps;
    a.R = n_w * ncols * NEO_D;
    a.t = 1;
    a.v = d_v;
    a.y = d_y;
    *done = true;
    return zrows_launch(ctx, a);
}
