// core.cu -- context, CCS upload, decomposition, Pi_RLC mix, Pi_DEC split and
// ME evaluations y = Z (M^T chi_r).
#include "internal.cuh"
#include <algorithm>

using gl::K;

static int neo_gpu_ctx_create_impl_abi(int device, neo_gpu_ctx** out) {
    if (!out) return NEO_ERR_ARG;
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return NEO_ERR_CUDA;
    if (device < 0 || device >= ndev) return NEO_ERR_ARG;
    if (cudaSetDevice(device) != cudaSuccess) return NEO_ERR_CUDA;
    neo_gpu_ctx* c = new neo_gpu_ctx();
    c->device = device;
    if (cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking) != cudaSuccess) {
        delete c;
        return NEO_ERR_CUDA;
    }
    if (cudaMalloc(&c->d_err, sizeof(uint32_t)) != cudaSuccess || cudaMemset(c->d_err, 0, sizeof(uint32_t)) != cudaSuccess) {
        cudaStreamDestroy(c->stream);
        delete c;
        return NEO_ERR_CUDA;
    }
    if (cudaHostAlloc(&c->h_result, CTX_RESULT_BYTES, cudaHostAllocMapped) != cudaSuccess) {
        cudaFree(c->d_err);
        cudaStreamDestroy(c->stream);
        delete c;
        return NEO_ERR_OOM;
    }
    memset(c->h_result, 0, CTX_RESULT_BYTES);
    // without a pool (an old driver) the buffers come from cudaMalloc
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    if (cudaMemPoolCreate(&c->pool, &props) == cudaSuccess) {
        uint64_t keep = ~0ull;  // what it keeps is bounded by pool_trim
        cudaMemPoolSetAttribute(c->pool, cudaMemPoolAttrReleaseThreshold, &keep);
    } else {
        c->pool = nullptr;
        cudaGetLastError();
    }
    *out = c;
    return NEO_OK;
}
extern "C" int neo_gpu_ctx_create(int device, neo_gpu_ctx** out) { NEO_ABI_GUARD(neo_gpu_ctx_create_impl_abi(device, out)) }

// Stream on which DevBuf allocations of this thread are made (stream-ordered,
// from the device's memory pool) and later freed; null: cudaMalloc / cudaFree.
thread_local cudaStream_t g_alloc_stream = nullptr;
thread_local PoolRef g_pool;
thread_local uint64_t g_pool_frees = 0;

// Unused memory above CTX_POOL_KEEP bytes goes back to the device.  A free counts once
// the stream has been seen to pass it, so the stream is waited for, but only where there
// is something to give back or to show (waiting whenever more than the bound was held
// added 10 us to a small oracle's 270 beside 2 GB).
void pool_trim(neo_gpu_ctx* ctx) {
    uint64_t held = 0, used = 0;
    if (!ctx->pool || cudaMemPoolGetAttribute(ctx->pool, cudaMemPoolAttrReservedMemCurrent, &held)) return;
    if (held <= ctx->pool_live + CTX_POOL_KEEP && ctx->pool_unseen <= POOL_UNSEEN) return;
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(ctx->stream, &st) || st != cudaStreamCaptureStatusNone) return;
    if (cudaStreamSynchronize(ctx->stream)) return;
    ctx->pool_unseen = 0;
    if (!cudaMemPoolGetAttribute(ctx->pool, cudaMemPoolAttrUsedMemCurrent, &used) && held > used + CTX_POOL_KEEP)
        cudaMemPoolTrimTo(ctx->pool, used + CTX_POOL_KEEP);
}

static int neo_gpu_ctx_destroy_impl_abi(neo_gpu_ctx* ctx) {
    if (!ctx) return NEO_ERR_ARG;
    cudaSetDevice(ctx->device);
    cudaStreamSynchronize(ctx->stream);
    if (ctx->scratch) cudaFree(ctx->scratch);
    if (ctx->commit_buf) cudaFree(ctx->commit_buf);
    if (ctx->vinv) cudaFree(ctx->vinv);
    if (ctx->d_err) cudaFree(ctx->d_err);
    if (ctx->h_result) cudaFreeHost(ctx->h_result);
    if (ctx->pool) cudaMemPoolDestroy(ctx->pool);
    cudaStreamDestroy(ctx->stream);
    delete ctx;
    return NEO_OK;
}
extern "C" int neo_gpu_ctx_destroy(neo_gpu_ctx* ctx) { NEO_ABI_GUARD(neo_gpu_ctx_destroy_impl_abi(ctx)) }

extern "C" const char* neo_gpu_last_error(const neo_gpu_ctx* ctx) { return ctx ? ctx->err.c_str() : "null context"; }
extern "C" uint64_t neo_gpu_kernel_launches(const neo_gpu_ctx* ctx) { return ctx ? ctx->launches : 0; }
int check_device_error(neo_gpu_ctx* ctx) {
    uint32_t e = 0;
    NEO_CK(ctx, ctx_d2h(ctx, &e, ctx->d_err, 4));
    NEO_CK(ctx, ctx_sync(ctx));
    if (e) {
        NEO_CK(ctx, cudaMemsetAsync(ctx->d_err, 0, 4, ctx->stream));
        *ctx_host_err(ctx) = 0;  // the same call's error, not the next one's
        char buf[128];
        if (e == (1u << 16)) {  // set by the small-digit commitment form only
            snprintf(buf, sizeof buf, "commitment digits outside [-63, 63] on the small-digit path");
            return ctx->fail(NEO_ERR_INVARIANT, buf);
        }
        snprintf(buf, sizeof buf, "device wait timed out (error bits 0x%x)", e);
        return ctx->fail(NEO_ERR_CUDA, buf);
    }
    return check_host_error(ctx);
}

// Bounded device wait: one thread polls *flag up to `limit` times (about
// 1 us apart); a wait that runs out sets bit 0x10 of the context's error word
// (err, as the commitment kernel's bounded mbarrier waits do; or the page-locked
// one, host_err, as those of the ME outputs and the RLC mix) and returns.
__global__ void wait_flag_kernel(const volatile uint32_t* flag, uint32_t limit, uint32_t* err, volatile uint32_t* host_err) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    for (uint32_t it = 0; it < limit; it++) {
        if (*flag) return;
        __nanosleep(1000);
    }
    if (err) atomicOr(err, 0x10u);
    if (host_err) *host_err = 0x10u;
}

static int neo_gpu_wait_probe_impl_abi(neo_gpu_ctx* ctx, uint32_t set_flag, uint32_t spin_limit) {
    if (!ctx) return NEO_ERR_ARG;
    if (spin_limit == 0 || spin_limit > (1u << 20)) return ctx->fail(NEO_ERR_ARG, "wait_probe: spin_limit in [1, 2^20]");
    cudaSetDevice(ctx->device);
    PoolScope pool_scope(ctx);
    DevBuf<uint32_t> flag;
    NEO_CK(ctx, flag.alloc(1));
    NEO_CK(ctx, cudaMemsetAsync(flag.p, 0, 4, ctx->stream));
    if (set_flag) NEO_CK(ctx, cudaMemsetAsync(flag.p, 0xFF, 4, ctx->stream));
    wait_flag_kernel<<<1, 32, 0, ctx->stream>>>(flag.p, spin_limit, ctx->d_err, nullptr);
    NEO_LAUNCHED(ctx);
    return check_device_error(ctx);  // synchronizes; a timeout is reported and cleared
}
extern "C" int neo_gpu_wait_probe(neo_gpu_ctx* ctx, uint32_t set_flag, uint32_t spin_limit) { NEO_ABI_GUARD(neo_gpu_wait_probe_impl_abi(ctx, set_flag, spin_limit)) }

static int neo_gpu_wait_probe_async_impl_abi(neo_gpu_ctx* ctx, uint32_t spin_limit) {
    if (!ctx) return NEO_ERR_ARG;
    if (spin_limit == 0 || spin_limit > (1u << 20)) return ctx->fail(NEO_ERR_ARG, "wait_probe: spin_limit in [1, 2^20]");
    cudaSetDevice(ctx->device);
    PoolScope pool_scope(ctx);
    DevBuf<uint32_t> flag;
    NEO_CK(ctx, flag.alloc(1));
    NEO_CK(ctx, cudaMemsetAsync(flag.p, 0, 4, ctx->stream));
    wait_flag_kernel<<<1, 32, 0, ctx->stream>>>(flag.p, spin_limit, nullptr, ctx_host_err(ctx));
    NEO_LAUNCHED(ctx);
    return NEO_OK;
}
extern "C" int neo_gpu_wait_probe_async(neo_gpu_ctx* ctx, uint32_t spin_limit) { NEO_ABI_GUARD(neo_gpu_wait_probe_async_impl_abi(ctx, spin_limit)) }

static int neo_gpu_ctx_stream_impl_abi(const neo_gpu_ctx* ctx, void** stream) {
    if (!ctx || !stream) return NEO_ERR_ARG;
    *stream = (void*)ctx->stream;
    return NEO_OK;
}
extern "C" int neo_gpu_ctx_stream(const neo_gpu_ctx* ctx, void** stream) { NEO_ABI_GUARD(neo_gpu_ctx_stream_impl_abi(ctx, stream)) }
static int neo_gpu_synchronize_impl_abi(neo_gpu_ctx* ctx) {
    if (!ctx) return NEO_ERR_ARG;
    cudaSetDevice(ctx->device);
    return check_device_error(ctx);  // waits for the stream, then reports (and clears) device-side errors
}
extern "C" int neo_gpu_synchronize(neo_gpu_ctx* ctx) { NEO_ABI_GUARD(neo_gpu_synchronize_impl_abi(ctx)) }

// ---------------------------------------------------------------------------
// CCS upload: CSC as given, plus a CSR copy made on the device (a row's entries in
// any order: every use sums them in F_q exactly).  On the host the transposition
// of 590 k nonzeros and its copies took 7 ms of a 2^16-row Pi_CCS oracle's life;
// these kernels, bound by their scattered 8- and 4-byte accesses, take 28 us.
// ---------------------------------------------------------------------------
struct CcsRanges {  // the nonzeros of each matrix (none for an identity)
    uint64_t lo[16], hi[16];
    uint64_t first[16];  // the first that belongs to a column
};
// blockIdx.y = matrix: values made canonical in place, entries per row at ptr[row + 1] (ptr may be null)
__global__ void csr_count_kernel(const __grid_constant__ CcsRanges g, const uint32_t* __restrict__ row,
                                 uint64_t* __restrict__ val, uint32_t n, unsigned long long* __restrict__ ptr) {
    const uint32_t j = blockIdx.y;
    const uint64_t k = g.lo[j] + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (k >= g.hi[j]) return;
    val[k] = gl::canon(val[k]);
    if (ptr && k >= g.first[j]) atomicAdd(ptr + (uint64_t)j * (n + 1) + row[k] + 1, 1ull);
}

// Inclusive scan of each matrix's n + 1 counters (blockIdx.y), two launches: blocks
// of SCAN_N counters in place with their totals, then the totals before a block
// added to it (the result again as the fill's cursors).
constexpr uint32_t CSR_SCAN_N = 1024;
__device__ __forceinline__ uint64_t warp_sum_u64(uint64_t x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, (unsigned long long)x, o);
    return x;
}
__global__ void __launch_bounds__(256) csr_scan_kernel(uint64_t* __restrict__ ptr, uint32_t n, uint64_t* __restrict__ sums) {
    __shared__ uint64_t s_w[8];
    uint64_t* p = ptr + (uint64_t)blockIdx.y * (n + 1);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t i0 = blockIdx.x * (uint64_t)CSR_SCAN_N + 4 * threadIdx.x;
    uint64_t v[4], run = 0;
#pragma unroll
    for (int e = 0; e < 4; e++) v[e] = i0 + e <= n ? p[i0 + e] : 0;
#pragma unroll
    for (int e = 0; e < 4; e++) v[e] = run += v[e];
    uint64_t inc = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint64_t u = __shfl_up_sync(0xffffffffu, (unsigned long long)inc, o);
        if (lane >= o) inc += u;
    }
    if (lane == 31) s_w[warp] = inc;
    __syncthreads();
    uint64_t before = inc - run;
    for (int w = 0; w < warp; w++) before += s_w[w];
#pragma unroll
    for (int e = 0; e < 4; e++)
        if (i0 + e <= n) p[i0 + e] = before + v[e];
    if (threadIdx.x == 255) sums[(uint64_t)blockIdx.y * gridDim.x + blockIdx.x] = before + run;
}
__global__ void __launch_bounds__(256) csr_scan_add_kernel(uint64_t* __restrict__ ptr, uint32_t n,
                                                           const uint64_t* __restrict__ sums,
                                                           unsigned long long* __restrict__ cursor) {
    __shared__ uint64_t s_w[8];
    uint64_t b = 0;
    for (uint32_t i = threadIdx.x; i < blockIdx.x; i += 256) b += sums[(uint64_t)blockIdx.y * gridDim.x + i];
    b = warp_sum_u64(b);
    if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = b;
    __syncthreads();
    b = 0;
#pragma unroll
    for (int w = 0; w < 8; w++) b += s_w[w];
    const uint64_t base = (uint64_t)blockIdx.y * (n + 1), i0 = blockIdx.x * (uint64_t)CSR_SCAN_N;
#pragma unroll
    for (int e = 0; e < 4; e++) {
        const uint64_t i = i0 + threadIdx.x + 256 * e;
        if (i > n) break;
        const uint64_t x = ptr[base + i] + b;
        ptr[base + i] = x;
        cursor[base + i] = x;
    }
}

// blockIdx.y = matrix, a thread per column: its entries to the next free slots of their rows
__global__ void csr_fill_kernel(const __grid_constant__ CcsRanges g, const uint64_t* __restrict__ csc_ptr,
                                const uint32_t* __restrict__ row, const uint64_t* __restrict__ val, uint32_t n, uint32_t m,
                                unsigned long long* __restrict__ cursor, uint32_t* __restrict__ csr_col,
                                uint64_t* __restrict__ csr_val) {
    const uint32_t j = blockIdx.y;
    const uint64_t c = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (c >= m) return;
    if (g.hi[j] == g.lo[j]) return;  // an identity's column pointers are not there
    const uint64_t base = g.lo[j];
    const uint64_t* cp = csc_ptr + (uint64_t)j * (m + 1);
    for (uint64_t k = cp[c]; k < cp[c + 1]; k++) {
        const uint64_t pos = base + atomicAdd(cursor + (uint64_t)j * (n + 1) + row[base + k], 1ull);
        csr_col[pos] = (uint32_t)c;
        csr_val[pos] = val[base + k];
    }
}

int dev_ccs_upload(neo_gpu_ctx* ctx, const neo_ccs_desc* d, DevCcs& o, bool want_csr) {
    if (!d || d->t == 0 || d->m == 0 || d->n == 0 || d->t > 16 || d->n_terms == 0 || d->n_terms > 16)
        return ctx->fail(NEO_ERR_ARG, "ccs: bad dimensions");
    o.n = d->n; o.m = d->m; o.t = d->t; o.n_terms = d->n_terms;
    o.is_identity.assign(d->is_identity, d->is_identity + d->t);
    o.f_coeff.assign(d->f_coeff, d->f_coeff + d->n_terms);
    o.f_exps.assign(d->f_exps, d->f_exps + (size_t)d->n_terms * d->t);
    o.nnz_off.assign(d->nnz_off, d->nnz_off + d->t + 1);
    const uint64_t nnz = o.nnz_off[d->t];
    uint64_t max_cnt = 0;
    CcsRanges g{};
    for (uint32_t j = 0; j < d->t; j++) {
        if (o.is_identity[j]) continue;
        // what the kernels index with: a matrix's range inside the nonzeros, columns one after the
        // other inside the range (entries before the first column belong to none), rows below n
        const uint64_t base = o.nnz_off[j], end = o.nnz_off[j + 1], cnt = end - base;
        if (base > end || end > nnz) return ctx->fail(NEO_ERR_ARG, "ccs: nnz_off decreases");
        const uint64_t* cp = d->col_ptr + (size_t)j * (d->m + 1);
        if (cp[d->m] != cnt) return ctx->fail(NEO_ERR_ARG, "ccs: col_ptr inconsistent with nnz_off");
        uint64_t down = 0;
        for (uint32_t c = 0; c < d->m; c++) down |= (uint64_t)(cp[c] > cp[c + 1]);
        if (down) return ctx->fail(NEO_ERR_ARG, "ccs: col_ptr decreases");
        g.lo[j] = base;
        g.hi[j] = end;
        g.first[j] = base + cp[0];
        uint32_t top = 0;
        for (uint64_t k = 0; k < cnt; k++) top = std::max(top, d->row_idx[base + k]);
        if (cnt && top >= d->n) return ctx->fail(NEO_ERR_ARG, "ccs: row index out of range");
        max_cnt = std::max(max_cnt, cnt);
    }
    const size_t nn = std::max<uint64_t>(nnz, 1), n_cp = (size_t)d->t * (d->m + 1), n_rp = (size_t)d->t * (d->n + 1);
    cudaStream_t S = ctx->stream;
    NEO_CK(ctx, o.csc_ptr.alloc(n_cp));
    NEO_CK(ctx, o.csc_row.alloc(nn));
    NEO_CK(ctx, o.csc_val.alloc(nn));
    for (uint32_t j = 0, e; j < d->t; j = e) {  // one copy per run of matrices (an identity's ranges are not read)
        e = j + 1;
        if (o.is_identity[j]) continue;
        while (e < d->t && !o.is_identity[e]) e++;
        NEO_CK(ctx, cudaMemcpyAsync(o.csc_ptr.p + (size_t)j * (d->m + 1), d->col_ptr + (size_t)j * (d->m + 1),
                                    (e - j) * (d->m + 1) * 8ull, cudaMemcpyHostToDevice, S));
    }
    if (nnz) {
        NEO_CK(ctx, cudaMemcpyAsync(o.csc_row.p, d->row_idx, nnz * 4, cudaMemcpyHostToDevice, S));
        NEO_CK(ctx, cudaMemcpyAsync(o.csc_val.p, d->vals, nnz * 8, cudaMemcpyHostToDevice, S));
    }
    const dim3 nz_grid(ceil_div(std::max<uint64_t>(max_cnt, 1), 256), d->t);
    if (!want_csr) {
        csr_count_kernel<<<nz_grid, 256, 0, S>>>(g, o.csc_row.p, o.csc_val.p, d->n, nullptr);
        NEO_LAUNCHED(ctx);
        return NEO_OK;
    }
    DevBuf<unsigned long long> cursor;
    NEO_CK(ctx, cursor.alloc(n_rp));
    NEO_CK(ctx, o.csr_ptr.alloc(n_rp));
    NEO_CK(ctx, o.csr_col.alloc(nn));
    NEO_CK(ctx, o.csr_val.alloc(nn));
    NEO_CK(ctx, cudaMemsetAsync(o.csr_ptr.p, 0, n_rp * 8, S));
    csr_count_kernel<<<nz_grid, 256, 0, S>>>(g, o.csc_row.p, o.csc_val.p, d->n,
                                             reinterpret_cast<unsigned long long*>(o.csr_ptr.p));
    NEO_LAUNCHED(ctx);
    const dim3 sg(ceil_div((uint64_t)d->n + 1, CSR_SCAN_N), d->t);
    DevBuf<uint64_t> sums;
    NEO_CK(ctx, sums.alloc((size_t)sg.x * sg.y));
    csr_scan_kernel<<<sg, 256, 0, S>>>(o.csr_ptr.p, d->n, sums.p);
    NEO_LAUNCHED(ctx);
    csr_scan_add_kernel<<<sg, 256, 0, S>>>(o.csr_ptr.p, d->n, sums.p, cursor.p);
    NEO_LAUNCHED(ctx);
    csr_fill_kernel<<<dim3(ceil_div(d->m, 256), d->t), 256, 0, S>>>(g, o.csc_ptr.p, o.csc_row.p, o.csc_val.p, d->n, d->m,
                                                                   cursor.p, o.csr_col.p, o.csr_val.p);
    NEO_LAUNCHED(ctx);
    if (!cursor.s) NEO_CK(ctx, ctx_sync(ctx));  // a plain allocation is freed at once
    return NEO_OK;
}

// ---------------------------------------------------------------------------
// chi table: w[mask] = prod_i (bit_i(mask) ? b_i : 1 - b_i)
// (crates/neo-reductions/src/engines/optimized_engine/oracle.rs:1525-1540)
// ---------------------------------------------------------------------------
// A thread has one low index of CHI_LOW bits and the block CHI_HIGH high ones, each
// formed by a warp (a factor per lane): about two products an entry instead of one per
// bit (2^18 entries: 28 us, now 7.5, for a 4 MB table).
constexpr uint32_t CHI_LOW = 8, CHI_HIGH = 8;
__device__ __forceinline__ K chi_factor(const K* pts, uint32_t i, uint64_t idx) {
    const K b = pts[i];
    return ((idx >> i) & 1) ? b : gl::ksub(gl::kone(), b);
}
__device__ __forceinline__ void chi_entries(const K* pts, uint32_t nbits, K* __restrict__ out) {
    __shared__ K s_hi[CHI_HIGH];
    const uint32_t low = min(nbits, CHI_LOW), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t n_hi = 1ull << (nbits - low), h0 = blockIdx.x * (uint64_t)CHI_HIGH;
    K h = gl::kone();
    if (low + lane < nbits) h = chi_factor(pts, low + lane, (h0 + warp) << low);
#pragma unroll 1
    for (int o = 16; o > 0; o >>= 1) {
        K x;
        x.re = __shfl_xor_sync(0xffffffffu, (unsigned long long)h.re, o);
        x.im = __shfl_xor_sync(0xffffffffu, (unsigned long long)h.im, o);
        h = gl::kmul(h, x);
    }
    if (lane == 0) s_hi[warp] = h;
    K w = gl::kone();
#pragma unroll 1
    for (uint32_t i = 0; i < low; i++) w = gl::kmul(w, chi_factor(pts, i, threadIdx.x));
    __syncthreads();
    if (threadIdx.x >> low) return;
#pragma unroll
    for (uint32_t v = 0; v < CHI_HIGH; v++)
        if (h0 + v < n_hi) out[((h0 + v) << low) + threadIdx.x] = gl::kmul(w, s_hi[v]);
}
__global__ void __launch_bounds__(256) chi_table_kernel(const K* __restrict__ bits, uint32_t nbits, K* __restrict__ out) {
    chi_entries(bits, nbits, out);
}
__global__ void __launch_bounds__(256) chi_point_kernel(const __grid_constant__ KPoint p, uint32_t nbits, K* __restrict__ out) {
    chi_entries(p.x, nbits, out);
}
static unsigned chi_blocks(uint32_t nbits) { return nbits <= CHI_LOW ? 1u : (unsigned)ceil_div(1ull << (nbits - CHI_LOW), CHI_HIGH); }

int launch_chi_table(neo_gpu_ctx* ctx, const K* d_bits, uint32_t nbits, K* d_out) {
    chi_table_kernel<<<chi_blocks(nbits), 256, 0, ctx->stream>>>(d_bits, nbits, d_out);
    NEO_LAUNCHED(ctx);
    return NEO_OK;
}
int launch_chi_point(neo_gpu_ctx* ctx, const K* h_point, uint32_t nbits, K* d_out) {
    chi_point_kernel<<<chi_blocks(nbits), 256, 0, ctx->stream>>>(make_point(h_point, nbits), nbits, d_out);
    NEO_LAUNCHED(ctx);
    return NEO_OK;
}

// The tables chi(bits[j+1..nbits)) of every j < nbits in one launch: table j
// (2^(nbits-j-1) entries) sits at n - n/2^j, n = 2^nbits, so an index's
// leading one bits give its j.
__global__ void suffix_chi_kernel(const __grid_constant__ KPoint p, uint32_t nbits, K* __restrict__ out) {
    const uint64_t n = 1ULL << nbits;
    const uint64_t idx = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (idx + 1 >= n) return;
    const uint32_t j = __clzll(~(idx << (64 - nbits)));  // leading ones of the nbits-bit index
    const uint64_t local = idx - (n - (n >> j));
    K w = gl::kone();
    for (uint32_t i = 0; i + j + 1 < nbits; i++) {
        const K b = p.x[j + 1 + i];
        w = gl::kmul(w, ((local >> i) & 1) ? b : gl::ksub(gl::kone(), b));
    }
    out[idx] = w;
}

int launch_suffix_chi_tables(neo_gpu_ctx* ctx, const K* h_point, uint32_t nbits, K* d_out) {
    if (nbits == 0) return NEO_OK;
    const uint64_t n = 1ULL << nbits;
    suffix_chi_kernel<<<ceil_div(n - 1, 256), 256, 0, ctx->stream>>>(make_point(h_point, nbits), nbits, d_out);
    NEO_LAUNCHED(ctx);
    return NEO_OK;
}

// ---------------------------------------------------------------------------
// decomp_b (b = 2, balanced) (crates/neo-ajtai/src/decomp.rs:118-158)
// ---------------------------------------------------------------------------
__global__ void decomp_b2_kernel(const uint64_t* __restrict__ z, uint64_t m, int8_t* __restrict__ Z) {
    uint64_t c = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (c >= m) return;
    uint64_t u = gl::canon(z[c]);
    const uint64_t half = (GL_Q - 1) / 2;
    int64_t a = u <= half ? (int64_t)u : -(int64_t)(GL_Q - u);
#pragma unroll
    for (int row = 0; row < NEO_D; row++) {
        int64_t digit = (a & 1) == 0 ? 0 : (a >= 0 ? 1 : -1);
        Z[(uint64_t)row * m + c] = (int8_t)digit;
        a = (a - digit) >> 1;
    }
}

static int neo_gpu_decomp_b2_impl_abi(neo_gpu_ctx* ctx, const uint64_t* z, uint64_t m, int8_t* Z) {
    if (!ctx || !z || !Z || m == 0) return ctx ? ctx->fail(NEO_ERR_ARG, "decomp: bad args") : NEO_ERR_ARG;
    cudaSetDevice(ctx->device);
    PoolScope pool_scope(ctx);
    DevBuf<uint64_t> dz;
    DevBuf<int8_t> dZ;
    NEO_CK(ctx, dz.alloc(m));
    NEO_CK(ctx, dZ.alloc((size_t)NEO_D * m));
    NEO_CK(ctx, cudaMemcpyAsync(dz.p, z, m * 8, cudaMemcpyHostToDevice, ctx->stream));
    decomp_b2_kernel<<<ceil_div(m, 256), 256, 0, ctx->stream>>>(dz.p, m, dZ.p);
    NEO_LAUNCHED(ctx);
    NEO_CK(ctx, ctx_d2h(ctx, Z, dZ.p, (size_t)NEO_D * m));
    NEO_CK(ctx, ctx_sync(ctx));
    return NEO_OK;
}
extern "C" int neo_gpu_decomp_b2(neo_gpu_ctx* ctx, const uint64_t* z, uint64_t m, int8_t* Z) { NEO_ABI_GUARD(neo_gpu_decomp_b2_impl_abi(ctx, z, m, Z)) }

// ---------------------------------------------------------------------------
// Pi_RLC mix: Z_mix[:, c] = sum_i a_i(X) z_{i,c}(X) mod Phi_81 over the
// integers (all entries are small, so this equals the F_q computation of
// optimized_engine/common.rs:1221-1379 with rot_from_coeffs common.rs:398-430).
// Zmix = [rot_1 .. rot_k] (54 x 54k) times the stacked digit planes
// (54k x m), exact in int32, on the tensor cores (rlc_tc.cu).
// ---------------------------------------------------------------------------
// integer rot(a): column t = a X^t mod Phi_81 (commit.rs:46-54 recurrence)
static void rot_int8(const int8_t* a, int8_t* out) {
    int32_t col[NEO_D], nxt[NEO_D];
    for (int r = 0; r < NEO_D; r++) col[r] = a[r];
    for (int t = 0; t < NEO_D; t++) {
        for (int r = 0; r < NEO_D; r++) out[r * NEO_D + t] = (int8_t)col[r];
        int32_t last = col[NEO_D - 1];
        nxt[0] = -last;
        for (int q = 1; q < NEO_D; q++) nxt[q] = col[q - 1];
        nxt[27] -= last;
        memcpy(col, nxt, sizeof col);
    }
}

int rlc_mix_device(neo_gpu_ctx* ctx, const int8_t* rho_coeffs_host, const int8_t* d_Zs, uint32_t count, uint64_t m,
                   int32_t* d_Zmix, int8_t* d_rot_scratch) {
    std::vector<int8_t> rot((size_t)count * NEO_D * NEO_D);
    for (uint32_t i = 0; i < count; i++) {
        for (int r = 0; r < NEO_D; r++)
            if (rho_coeffs_host[i * NEO_D + r] < -2 || rho_coeffs_host[i * NEO_D + r] > 2)
                return ctx->fail(NEO_ERR_ARG, "rlc: rho coefficient outside {-2..2}");
        if (count == 1) {
            memset(rot.data(), 0, NEO_D * NEO_D);
            for (int r = 0; r < NEO_D; r++) rot[r * NEO_D + r] = 1;  // identity (common.rs:560-564)
        } else {
            rot_int8(rho_coeffs_host + i * NEO_D, rot.data() + (size_t)i * NEO_D * NEO_D);
        }
    }
    // rows padded to RLC_ROT_ROW bytes for the kernel's 16-byte shared loads
    std::vector<int8_t> rot_pad((size_t)count * NEO_D * RLC_ROT_ROW, 0);
    for (size_t row = 0; row < (size_t)count * NEO_D; row++)
        memcpy(&rot_pad[row * RLC_ROT_ROW], &rot[row * NEO_D], NEO_D);
    NEO_CK(ctx, cudaMemcpyAsync(d_rot_scratch, rot_pad.data(), rot_pad.size(), cudaMemcpyHostToDevice, ctx->stream));
    NEO_CK(ctx, ctx_sync(ctx));  // rot_pad is pageable host memory that goes away on return
    return launch_rlc_mix(ctx, d_rot_scratch, d_Zs, count, m, d_Zmix);
}

static int neo_gpu_rlc_mix_impl_abi(neo_gpu_ctx* ctx, const int8_t* rho_coeffs, const int8_t* Zs, uint32_t count,
                               uint64_t m, int32_t* Zmix) {
    if (!ctx) return NEO_ERR_ARG;
    if (!rho_coeffs || !Zs || !Zmix || count == 0 || count > 64 || m == 0) return ctx->fail(NEO_ERR_ARG, "rlc: bad args");
    cudaSetDevice(ctx->device);
    PoolScope pool_scope(ctx);
    DevBuf<int8_t> dZs, drot;
    DevBuf<int32_t> dmix;
    NEO_CK(ctx, dZs.alloc((size_t)count * NEO_D * m, MIX_PAD));
    NEO_CK(ctx, drot.alloc((size_t)count * NEO_D * RLC_ROT_ROW));
    NEO_CK(ctx, dmix.alloc((size_t)NEO_D * m));
    NEO_CK(ctx, cudaMemcpyAsync(dZs.p, Zs, dZs.bytes(), cudaMemcpyHostToDevice, ctx->stream));
    int rc = rlc_mix_device(ctx, rho_coeffs, dZs.p, count, m, dmix.p, drot.p);
    if (rc) return rc;
    NEO_CK(ctx, ctx_d2h(ctx, Zmix, dmix.p, dmix.bytes()));
    NEO_CK(ctx, ctx_sync(ctx));
    return check_host_error(ctx);
}
extern "C" int neo_gpu_rlc_mix(neo_gpu_ctx* ctx, const int8_t* rho_coeffs, const int8_t* Zs, uint32_t count,
                               uint64_t m, int32_t* Zmix) { NEO_ABI_GUARD(neo_gpu_rlc_mix_impl_abi(ctx, rho_coeffs, Zs, count, m, Zmix)) }

// ---------------------------------------------------------------------------
// Pi_DEC split (common.rs:75-268; balanced_divrem common.rs:44-58)
// flags[0] = out-of-range error, flags[1 + i] = plane i nonzero
// ---------------------------------------------------------------------------
// Z_mix entries are int32, so the digits come from 32-bit arithmetic; b = 2
// (the fold step's base) takes the balanced remainder and an exact shift
// instead of a division.
// block-aggregate the nonzero plane mask; one atomic per block, and none
// once every plane it saw is already flagged (a single address that every
// warp hit serialised the kernel)
__device__ __forceinline__ void split_flags(uint32_t nz_mask, uint32_t* flags) {
    for (int o = 16; o > 0; o >>= 1) nz_mask |= __shfl_xor_sync(0xffffffffu, nz_mask, o);
    __shared__ uint32_t s_mask;
    if (threadIdx.x == 0) s_mask = 0;
    __syncthreads();
    if ((threadIdx.x & 31) == 0 && nz_mask) atomicOr(&s_mask, nz_mask);
    __syncthreads();
    if (threadIdx.x == 0 && s_mask && (s_mask & ~__ldcg(flags + 1))) atomicOr(&flags[1], s_mask);
}
template <bool B2>
__global__ void split_b_kernel(const int32_t* __restrict__ Zmix, uint64_t len, uint32_t k, int32_t b,
                               int8_t* __restrict__ planes, uint32_t* __restrict__ flags) {
    uint64_t idx = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    uint32_t nz_mask = 0;
    if (idx < len) {
        int32_t v = Zmix[idx];
        // b^k, saturated once it exceeds every int32 (the check is then moot)
        int64_t B = 1;
        for (uint32_t i = 0; i < k && B <= INT32_MAX; i++) B *= b;
        if ((int64_t)v >= B || (int64_t)v <= -B) atomicOr(&flags[0], 1u);
        const int32_t half = b / 2;
        for (uint32_t i = 0; i < k; i++) {
            int32_t r, q;
            if (B2) {  // v % 2 in {-1, 0, 1} (sign of v), v - r even
                r = (v & 1) ? (v < 0 ? -1 : 1) : 0;
                q = (v - r) >> 1;
            } else {
                r = v % b;
                q = (v - r) / b;
                if (r > half) { r -= b; q += 1; }
                else if (r < -half) { r += b; q -= 1; }
            }
            planes[(uint64_t)i * len + idx] = (int8_t)r;
            if (r) nz_mask |= 1u << i;
            v = q;
        }
        if (v != 0) atomicOr(&flags[0], 1u);
    }
    split_flags(nz_mask, flags);
}

// b = 2, eight entries a thread: a digit is the sign times a bit of the magnitude, so a
// plane's eight bytes are built packed and leave in one store.  Bound by its stores, k
// bytes an entry; byte by byte it was 186 us for 2^18 columns into 12 planes (220 MB)
// and 13.6 for 2^14, now 38 and 4.2.
__global__ void __launch_bounds__(256) split_b2_kernel(const int4* __restrict__ Zmix, uint64_t n8, uint32_t k,
                                                       uint2* __restrict__ planes, uint32_t* __restrict__ flags) {
    const uint64_t idx = blockIdx.x * 256ull + threadIdx.x;
    uint32_t nz_mask = 0;
    if (idx < n8) {
        const int4 x = Zmix[2 * idx], y = Zmix[2 * idx + 1];
        const int v[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
        uint32_t mag[8], neg[2] = {0, 0}, all = 0;
#pragma unroll
        for (int e = 0; e < 8; e++) {
            mag[e] = v[e] < 0 ? 0u - (uint32_t)v[e] : (uint32_t)v[e];
            neg[e >> 2] |= v[e] < 0 ? 0xFFu << (8 * (e & 3)) : 0u;
            all |= mag[e];
        }
        if (all >> k) atomicOr(&flags[0], 1u);
        nz_mask = all & ((1u << k) - 1);
        for (uint32_t i = 0; i < k; i++) {
            uint32_t d[2];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const uint32_t* g = mag + 4 * h;
                const uint32_t bits = ((g[0] >> i) & 1) | (((g[1] >> i) & 1) << 8) | (((g[2] >> i) & 1) << 16) | (((g[3] >> i) & 1) << 24);
                d[h] = bits | (neg[h] & (bits * 255));
            }
            planes[(uint64_t)i * n8 + idx] = make_uint2(d[0], d[1]);
        }
    }
    split_flags(nz_mask, flags);
}

int split_b_device(neo_gpu_ctx* ctx, const int32_t* d_Zmix, uint64_t len, uint32_t k, uint32_t b, int8_t* d_planes,
                   uint32_t* d_flags) {
    if (k == 0 || k > 31 || b < 2 || b > 64) return ctx->fail(NEO_ERR_UNSUPPORTED, "split_b: k/b out of range");
    NEO_CK(ctx, cudaMemsetAsync(d_flags, 0, 2 * sizeof(uint32_t), ctx->stream));
    // whole eights, and planes that begin on 8 bytes (54 m entries: m a multiple of 4)
    if (b == 2 && len % 8 == 0 && !(reinterpret_cast<uintptr_t>(d_Zmix) & 15) && !(reinterpret_cast<uintptr_t>(d_planes) & 7))
        split_b2_kernel<<<ceil_div(len / 8, 256), 256, 0, ctx->stream>>>(reinterpret_cast<const int4*>(d_Zmix), len / 8, k,
                                                                        reinterpret_cast<uint2*>(d_planes), d_flags);
    else if (b == 2)
        split_b_kernel<true><<<ceil_div(len, 256), 256, 0, ctx->stream>>>(d_Zmix, len, k, 2, d_planes, d_flags);
    else
        split_b_kernel<false><<<ceil_div(len, 256), 256, 0, ctx->stream>>>(d_Zmix, len, k, (int32_t)b, d_planes, d_flags);
    NEO_LAUNCHED(ctx);
    return NEO_OK;
}

static int neo_gpu_split_b_impl_abi(neo_gpu_ctx* ctx, const int32_t* Zmix, uint64_t len, uint32_t k, uint32_t b,
                               int8_t* planes, uint8_t* nonzero) {
    if (!ctx) return NEO_ERR_ARG;
    if (!Zmix || !planes || !nonzero || len == 0) return ctx->fail(NEO_ERR_ARG, "split_b: bad args");
    cudaSetDevice(ctx->device);
    PoolScope pool_scope(ctx);
    DevBuf<int32_t> dmix;
    DevBuf<int8_t> dpl;
    DevBuf<uint32_t> dfl;
    NEO_CK(ctx, dmix.alloc(len));
    NEO_CK(ctx, dpl.alloc((size_t)k * len));
    NEO_CK(ctx, dfl.alloc(2));
    NEO_CK(ctx, cudaMemcpyAsync(dmix.p, Zmix, len * 4, cudaMemcpyHostToDevice, ctx->stream));
    int rc = split_b_device(ctx, dmix.p, len, k, b, dpl.p, dfl.p);
    if (rc) return rc;
    uint32_t flags[2];
    NEO_CK(ctx, ctx_d2h(ctx, flags, dfl.p, 8));
    NEO_CK(ctx, ctx_d2h(ctx, planes, dpl.p, (size_t)k * len));
    NEO_CK(ctx, ctx_sync(ctx));
    if (flags[0]) return ctx->fail(NEO_ERR_INVARIANT, "DEC split: entry out of range for k_rho digits");
    for (uint32_t i = 0; i < k; i++) nonzero[i] = (flags[1] >> i) & 1;
    return NEO_OK;
}
extern "C" int neo_gpu_split_b(neo_gpu_ctx* ctx, const int32_t* Zmix, uint64_t len, uint32_t k, uint32_t b,
                               int8_t* planes, uint8_t* nonzero) { NEO_ABI_GUARD(neo_gpu_split_b_impl_abi(ctx, Zmix, len, k, b, planes, nonzero)) }

// ---------------------------------------------------------------------------
// ME evaluations: v_j = M_j^T chi_r (CSC), y[w][j][rho] = sum_c Z_w[rho][c] v_j[c]
// (crates/neo-reductions/src/common.rs:582-650; oracle.rs:1694-1768)
// ---------------------------------------------------------------------------
// blockIdx.y: the matrix.  Bound by the latency of the dependent loads pointer -> row ->
// chi, so all matrices go in one launch (four at 2^10 columns: 18 us one by one, 6 together; at 2^18 69 and 54).
__global__ void matT_chi_kernel(const uint64_t* __restrict__ csc_ptr, const uint32_t* __restrict__ csc_row,
                                const uint64_t* __restrict__ csc_val, const __grid_constant__ MatSel sel, uint32_t n,
                                uint32_t m, uint64_t n_sz, const K* __restrict__ chi, K* __restrict__ v) {
    uint64_t c = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (c >= m) return;
    const uint32_t q = blockIdx.y;
    csc_ptr += (uint64_t)sel.j[q] * ((uint64_t)m + 1);
    csc_row += sel.off[q];
    csc_val += sel.off[q];
    v += (uint64_t)q * m;
    uint64_t n_eff = n < n_sz ? n : n_sz;
    if (sel.id[q]) {
        v[c] = c < n_eff ? chi[c] : gl::kzero();
        return;
    }
    K acc = gl::kzero();
    for (uint64_t k = csc_ptr[c]; k < csc_ptr[c + 1]; k++) {
        uint32_t r = csc_row[k];
        if (r < n_eff) acc = gl::kadd(acc, gl::kscale(chi[r], csc_val[k]));
    }
    v[c] = acc;
}

// one block per (w, rho); threads stride over columns; t accumulators.
template <int TMAX>
__global__ void __launch_bounds__(256) zv_dot_kernel(const int8_t* __restrict__ Z, uint64_t m, uint32_t t,
                                                     const K* __restrict__ v, K* __restrict__ y) {
    const uint32_t row = blockIdx.x;  // w*54 + rho
    const int8_t* zr = Z + (uint64_t)row * m;
    K acc[TMAX];
#pragma unroll
    for (int j = 0; j < TMAX; j++) acc[j] = gl::kzero();
    for (uint64_t c = threadIdx.x; c < m; c += blockDim.x) {
        int z = zr[c];
        if (z == 0) continue;
#pragma unroll
        for (int j = 0; j < TMAX; j++) {
            if (j < (int)t) {
                K x = v[(uint64_t)j * m + c];
                acc[j] = z == 1 ? gl::kadd(acc[j], x) : (z == -1 ? gl::ksub(acc[j], x) : gl::kadd(acc[j], gl::kscale_small(x, z)));
            }
        }
    }
    __shared__ K red[TMAX][8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int j = 0; j < TMAX; j++) {
        K a = acc[j];
        for (int o = 16; o > 0; o >>= 1) {
            K b;
            b.re = __shfl_xor_sync(0xffffffffu, a.re, o);
            b.im = __shfl_xor_sync(0xffffffffu, a.im, o);
            a = gl::kadd(a, b);
        }
        if (lane == 0) red[j][warp] = a;
    }
    __syncthreads();
    if (threadIdx.x < t) {
        K a = gl::kzero();
        for (int wv = 0; wv < (int)(blockDim.x >> 5); wv++) a = gl::kadd(a, red[threadIdx.x][wv]);
        // y layout [w][t][54]
        uint32_t w = row / NEO_D, rho = row % NEO_D;
        y[((uint64_t)w * t + threadIdx.x) * NEO_D + rho] = a;
    }
}

// ysc[q] = sum_rho b^rho y[q][rho], one warp per vector (as one thread's chain of 108
// products it took 16 us, now 3)
__global__ void __launch_bounds__(128) y_scalars_kernel(const K* __restrict__ y, uint32_t count, uint32_t b, K* __restrict__ ysc) {
    const uint32_t q = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;  // (w, j)
    if (q >= count) return;
    const uint64_t pw = gl::pow(b, lane);  // b^lane, and b^(lane + 32) for the second entry
    const K* v = y + (uint64_t)q * NEO_D;
    K acc = gl::kscale(v[lane], pw);
    if (lane + 32 < NEO_D) acc = gl::kadd(acc, gl::kscale(v[lane + 32], gl::mul(pw, gl::pow(b, 32))));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        K x;
        x.re = __shfl_xor_sync(0xffffffffu, (unsigned long long)acc.re, o);
        x.im = __shfl_xor_sync(0xffffffffu, (unsigned long long)acc.im, o);
        acc = gl::kadd(acc, x);
    }
    if (lane == 0) ysc[q] = acc;
}

int launch_me_y(neo_gpu_ctx* ctx, const DevCcs& ccs, const int8_t* d_Z, uint32_t n_w, uint64_t m, const K* d_chi,
                uint32_t ell_n, uint32_t b, K* d_vj, K* d_y, K* d_ysc) {
    uint64_t n_sz = 1ULL << ell_n;
    matT_chi_kernel<<<dim3(ceil_div(m, 256), ccs.t), 256, 0, ctx->stream>>>(
        ccs.csc_ptr.p, ccs.csc_row.p, ccs.csc_val.p, mat_sel(ccs, nullptr, ccs.t), ccs.n, (uint32_t)m, n_sz, d_chi, d_vj);
    NEO_LAUNCHED(ctx);
    bool done = false;
    if (int rc = launch_zrows(ctx, d_Z, n_w * NEO_D, m, ccs.t, d_vj, d_y, &done)) return rc;
    if (!done) {
        if (ccs.t <= 4)
            zv_dot_kernel<4><<<n_w * NEO_D, 256, 0, ctx->stream>>>(d_Z, m, ccs.t, d_vj, d_y);
        else
            zv_dot_kernel<16><<<n_w * NEO_D, 256, 0, ctx->stream>>>(d_Z, m, ccs.t, d_vj, d_y);
        NEO_LAUNCHED(ctx);
    }
    if (d_ysc) {
        y_scalars_kernel<<<ceil_div(n_w * ccs.t, 4), 128, 0, ctx->stream>>>(d_y, n_w * ccs.t, b, d_ysc);
        NEO_LAUNCHED(ctx);
    }
    return NEO_OK;
}

static int neo_gpu_me_y_impl_abi(neo_gpu_ctx* ctx, const neo_ccs_desc* desc, const int8_t* Z, uint32_t n_w, uint32_t ell_n,
                            const uint64_t* r, uint32_t b, uint64_t* y, uint64_t* y_scalars) {
    if (!ctx) return NEO_ERR_ARG;
    if (!desc || !Z || !r || !y || !y_scalars || n_w == 0 || ell_n == 0 || ell_n > 30)
        return ctx->fail(NEO_ERR_ARG, "me_y: bad args");
    cudaSetDevice(ctx->device);
    PoolScope pool_scope(ctx);
    DevCcs ccs;
    int rc = dev_ccs_upload(ctx, desc, ccs, false);  // the transposed products read the columns only
    if (rc) return rc;
    uint64_t m = desc->m;
    DevBuf<int8_t> dZ;
    DevBuf<K> dchi, dvj, dy, dysc;
    NEO_CK(ctx, dZ.alloc((size_t)n_w * NEO_D * m));
    NEO_CK(ctx, dchi.alloc(1ULL << ell_n));
    NEO_CK(ctx, dvj.alloc((size_t)ccs.t * m));
    NEO_CK(ctx, dy.alloc((size_t)n_w * ccs.t * NEO_D));
    NEO_CK(ctx, dysc.alloc((size_t)n_w * ccs.t));
    NEO_CK(ctx, cudaMemcpyAsync(dZ.p, Z, dZ.bytes(), cudaMemcpyHostToDevice, ctx->stream));
    if ((rc = launch_chi_point(ctx, reinterpret_cast<const K*>(r), ell_n, dchi.p))) return rc;
    if ((rc = launch_me_y(ctx, ccs, dZ.p, n_w, m, dchi.p, ell_n, b, dvj.p, dy.p, dysc.p))) return rc;
    NEO_CK(ctx, ctx_d2h(ctx, y, dy.p, dy.bytes()));
    NEO_CK(ctx, ctx_d2h(ctx, y_scalars, dysc.p, dysc.bytes()));
    NEO_CK(ctx, ctx_sync(ctx));
    return check_host_error(ctx);
}
extern "C" int neo_gpu_me_y(neo_gpu_ctx* ctx, const neo_ccs_desc* desc, const int8_t* Z, uint32_t n_w, uint32_t ell_n,
                            const uint64_t* r, uint32_t b, uint64_t* y, uint64_t* y_scalars) { NEO_ABI_GUARD(neo_gpu_me_y_impl_abi(ctx, desc, Z, n_w, ell_n, r, b, y, y_scalars)) }
