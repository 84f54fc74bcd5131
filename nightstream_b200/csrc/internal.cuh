// internal.cuh -- context, status handling and device buffers shared by the
// CUDA translation units of libneo_gpu.so.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <string>
#include <utility>
#include <vector>
#include "../../include/neo_gpu.h"
#include "abi_guard.h"
#include "gl.cuh"
#include "mix_words.h"

#define NEO_D 54
// bytes per rot(a) row in the RLC mix scratch: 54 int8 entries, zero padded
constexpr int RLC_ROT_ROW = 64;

struct neo_gpu_ctx {
    int device = 0;
    cudaStream_t stream = nullptr;
    cudaMemPool_t pool = nullptr;    // this context's device buffers (PoolScope)
    uint64_t pool_live = 0;          // their bytes
    uint64_t pool_unseen = 0;        // bytes freed since pool_trim last waited for the stream
    std::string err;
    uint64_t launches = 0;
    // page-locked, device-mapped: kernels write a round's few values here, so that a
    // round ends with its launch instead of a copy (a call reads it before it returns)
    void* h_result = nullptr;
    uint32_t* d_err = nullptr;       // device error word (bounded-wait timeouts); 0 = ok
    void* scratch = nullptr;         // growable per-context scratch (stream-ordered use)
    size_t scratch_bytes = 0;
    // tensor-core commitment workspace (commit_tc.cu): accumulators and tickets, zero between calls
    void* commit_buf = nullptr;
    uint32_t commit_groups = 0;
    size_t commit_words = 0;
    uint64_t* vinv = nullptr;        // inverse Vandermonde tables (mem_oracle.cu), once a batched round needs them
    int fail(int code, const char* what, cudaError_t e = cudaSuccess) {
        char buf[512];
        if (e != cudaSuccess)
            snprintf(buf, sizeof buf, "%s: %s", what, cudaGetErrorString(e));
        else
            snprintf(buf, sizeof buf, "%s", what);
        err = buf;
        return code;
    }
};

constexpr size_t CTX_RESULT_BYTES = 4096;
// the last word of h_result: nonzero once a kernel's bounded wait gave up
inline volatile uint32_t* ctx_host_err(neo_gpu_ctx* c) {
    return reinterpret_cast<volatile uint32_t*>(static_cast<char*>(c->h_result) + CTX_RESULT_BYTES - 8);
}
// for a call that has waited for the launches it asks about
inline int check_host_error(neo_gpu_ctx* c) {
    const uint32_t e = *ctx_host_err(c);
    if (!e) return NEO_OK;
    *ctx_host_err(c) = 0;
    char buf[64];
    snprintf(buf, sizeof buf, "device wait timed out (error bits 0x%x)", e);
    return c->fail(NEO_ERR_CUDA, buf);
}

// wait for the context's stream (a spinning stream synchronization: batch
// workers that slept in blocking waits were measured no faster)
inline cudaError_t ctx_sync(neo_gpu_ctx* c) { return cudaStreamSynchronize(c->stream); }

// A launch's few field elements in page-locked memory (h_result and the like) are
// awaited word by word: `result_arm` fills the words with a value that no field
// element has, and `result_wait` looks until the launch has overwritten every one.
// The words are a launch's last stores: they leave by its last block (a ticket), which
// has seen all others finish; or by every block or thread for its own words, behind what
// else it stores (multi_small's points, mem_fold_kernel's factors), and are waited for
// all.  So nothing of the launch is left to do when they are there, and what it stored
// is read by later launches of the stream only.  A stream synchronization learns of the
// end when the launch has retired, about 4.5 us later: a Twist read oracle of 2^16 rows
// takes 518 us with it and 450 without, a bitness oracle of 2^12 321 and 274, Pi_CCS of
// 2^10 rows 675 and 621.  Polling is bounded (about a millisecond), then the stream is
// synchronized, which also is how an error of the launch is found; a launch under
// capture ends there too.
inline void result_arm(void* p, size_t words) { memset(p, 0xFF, words * 8); }
inline bool result_ready(const void* p, size_t words) {
    const uint64_t* w = static_cast<const uint64_t*>(p);
    for (size_t i = words; i-- > 0;)
        if (__atomic_load_n(w + i, __ATOMIC_ACQUIRE) == ~0ull) return false;
    return true;
}
inline cudaError_t result_wait(neo_gpu_ctx* c, const void* p, size_t words) {
    for (int spin = 0; spin < (1 << 15); spin++) {
        if (result_ready(p, words)) return cudaSuccess;
#if defined(__x86_64__)
        __builtin_ia32_pause();
#endif
    }
    // words still missing behind a good synchronization: a launch that did not write them
    const cudaError_t e = ctx_sync(c);
    return e != cudaSuccess || result_ready(p, words) ? e : cudaErrorNotReady;
}

// device -> host copy on the context's stream
inline cudaError_t ctx_d2h(neo_gpu_ctx* c, void* dst, const void* src, size_t bytes) {
    return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, c->stream);
}

#define NEO_CK(ctx, call)                                                         \
    do {                                                                          \
        cudaError_t _e = (call);                                                  \
        if (_e != cudaSuccess) {                                                  \
            return (ctx)->fail(_e == cudaErrorMemoryAllocation ? NEO_ERR_OOM      \
                                                               : NEO_ERR_CUDA,    \
                               #call, _e);                                        \
        }                                                                         \
    } while (0)

#define NEO_LAUNCHED(ctx)                                                         \
    do {                                                                          \
        (ctx)->launches++;                                                        \
        cudaError_t _e = cudaGetLastError();                                      \
        if (_e != cudaSuccess) return (ctx)->fail(NEO_ERR_CUDA, "kernel launch", _e); \
    } while (0)

// Ajtai public parameters of one m on one device, shared by every context on
// that device (the reference keeps one PP per (d, m) in a global registry,
// crates/neo-ajtai/src/s_module.rs:23-222).
struct PPEntry {
    int device = 0;
    uint64_t m = 0;
    uint32_t kappa = 0;
    uint64_t* d_pp = nullptr;       // [kappa][m][54] canonical u64
    uint8_t* d_pp_limbs = nullptr;  // tensor-core tiles: [ceil(m/2)][128 rows][128 B], pre-swizzled
    bool tc = false;                // d_pp_limbs holds the tiles of the current d_pp
};
PPEntry* pp_lookup(int device, uint64_t m);
// PP registry writes (commit.cu): pp_slot / pp_finish are called with pp_mutex() held
#include <mutex>
std::mutex& pp_mutex();
int pp_slot(neo_gpu_ctx* ctx, uint32_t kappa, uint64_t m, PPEntry** out);
int pp_finish(neo_gpu_ctx* ctx, PPEntry* pp, uint32_t kappa);

// Owning device buffer (freed on scope exit).
// Stream of this thread's stream-ordered allocations (set by batch workers,
// whose thread uses a single context); null: plain cudaMalloc / cudaFree.
extern thread_local cudaStream_t g_alloc_stream;

// The buffers of calls on a context come from the context's own memory pool,
// ordered on its stream: cudaMalloc and cudaFree cost 10 to 200 us each here and
// wait for the whole device, and an oracle's life has 15 to 36 of them (a Twist read
// oracle of 2^16 rows takes 1.8 ms with them and 0.45 from the pool, Pi_CCS of 2^16 rows
// and 13 witnesses 20 to 50 ms and 6.9, the mix and split of 13 witnesses of 2^14
// columns 5.5 ms and 2.1).
// A PoolScope is open for the duration of an entry point, on its thread only.
//
// What is freed stays with the pool, up to CTX_POOL_KEEP bytes beside those in use:
// the calls that free buffers (the destructions, and entry points with temporaries)
// give the rest back before they return (pool_trim).  The pool's own release
// threshold is no such bound: it counts the bytes in use too, so a context with more
// than that alive would keep nothing and map every buffer anew, and it acts at the
// next synchronization, which may be a later call's.
//
// An allocation anywhere else in the process that would fail takes unused memory from
// the pools (the driver does that), but only what a wait on the stream has seen freed:
// such a wait follows once POOL_UNSEEN bytes were.
constexpr uint64_t CTX_POOL_KEEP = 1ull << 30, POOL_UNSEEN = 64ull << 20;
struct PoolRef {
    cudaMemPool_t pool = nullptr;
    cudaStream_t stream = nullptr;
    neo_gpu_ctx* ctx = nullptr;  // whose bytes the allocations count to
};
extern thread_local PoolRef g_pool;
extern thread_local uint64_t g_pool_frees;  // buffers this thread gave to a pool
void pool_trim(neo_gpu_ctx* ctx);
struct PoolScope {
    PoolRef prev;
    neo_gpu_ctx* ctx;
    uint64_t frees;
    explicit PoolScope(neo_gpu_ctx* c) : prev(g_pool), ctx(c), frees(g_pool_frees) {
        if (!g_alloc_stream && ctx->pool) g_pool = {c->pool, c->stream, c};
    }
    ~PoolScope() {  // behind the frees of the entry point's own buffers
        g_pool = prev;
        if (!prev.pool && frees != g_pool_frees) pool_trim(ctx);
    }
    PoolScope(const PoolScope&) = delete;
    PoolScope& operator=(const PoolScope&) = delete;
};
inline cudaError_t pool_alloc(void** p, size_t bytes) {
    // a capture would turn the allocation into a node of the graph: refused, as cudaMalloc is
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    if (cudaError_t e = cudaStreamIsCapturing(g_pool.stream, &st)) return e;
    if (st != cudaStreamCaptureStatusNone) return cudaErrorStreamCaptureUnsupported;
    cudaError_t e = cudaMallocFromPoolAsync(p, bytes, g_pool.pool, g_pool.stream);
    if (e == cudaErrorMemoryAllocation) {  // give back what the pool holds and try once more
        cudaGetLastError();
        cudaStreamSynchronize(g_pool.stream);
        cudaMemPoolTrimTo(g_pool.pool, 0);
        e = cudaMallocFromPoolAsync(p, bytes, g_pool.pool, g_pool.stream);
    }
    return e;
}
// cudaMalloc for what outlives calls (PP, context workspaces): on failure the
// context's pool gives back what it holds first
inline cudaError_t ctx_malloc(neo_gpu_ctx* ctx, void** p, size_t bytes) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e == cudaErrorMemoryAllocation && ctx->pool) {
        cudaGetLastError();
        cudaStreamSynchronize(ctx->stream);
        cudaMemPoolTrimTo(ctx->pool, 0);
        e = cudaMalloc(p, bytes);
    }
    return e;
}

template <typename T>
struct DevBuf {
    T* p = nullptr;
    size_t n = 0;
    cudaStream_t s = nullptr;  // stream the allocation was ordered on (null: cudaMalloc); outlives the buffer
    neo_gpu_ctx* owner = nullptr;  // the context of whose pool the allocation is, or null
    size_t owned = 0;
    DevBuf() = default;
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    ~DevBuf() { release(); }
    size_t cap = 0;
    // pad: entries behind the buffer that may be read too
    cudaError_t alloc(size_t count, size_t pad = 0) {
        release();
        n = count;
        cap = count;
        if (count == 0) return cudaSuccess;
        s = g_alloc_stream;
        cudaError_t e;
        if (s) {
            e = cudaMallocAsync(reinterpret_cast<void**>(&p), (count + pad) * sizeof(T), s);
        } else if (g_pool.pool) {
            s = g_pool.stream;
            e = pool_alloc(reinterpret_cast<void**>(&p), (count + pad) * sizeof(T));
            if (e == cudaSuccess) {
                owner = g_pool.ctx;
                owner->pool_live += owned = (count + pad) * sizeof(T);
            }
        } else {
            e = cudaMalloc(&p, (count + pad) * sizeof(T));
        }
        if (e != cudaSuccess) {
            p = nullptr;
            s = nullptr;
            n = cap = 0;
        }
        return e;
    }
    // keep the allocation when it is large enough (reused workspaces)
    cudaError_t ensure(size_t count) {
        if (p && count <= cap) {
            n = count;
            return cudaSuccess;
        }
        return alloc(count);
    }
    void release() {
        if (p) {
            if (s) {
                cudaFreeAsync(p, s);
                g_pool_frees++;
                if (owner) {
                    owner->pool_live -= owned;
                    owner->pool_unseen += owned;
                }
            } else {
                cudaFree(p);
            }
        }
        p = nullptr;
        s = nullptr;
        owner = nullptr;
        n = 0;
        cap = 0;
    }
    void swap(DevBuf& o) {
        std::swap(p, o.p);
        std::swap(n, o.n);
        std::swap(s, o.s);
        std::swap(owner, o.owner);
        std::swap(owned, o.owned);
        std::swap(cap, o.cap);
    }
    size_t bytes() const { return n * sizeof(T); }
};

// Page-locked host buffer: a cudaMemcpyAsync from or to it is queued on the
// stream and does not wait for the stream's earlier work (a pageable source
// makes the copy synchronous).  Reused across rounds; freed on scope exit.
template <typename T>
struct HostBuf {
    T* p = nullptr;
    size_t cap = 0;
    HostBuf() = default;
    HostBuf(const HostBuf&) = delete;
    HostBuf& operator=(const HostBuf&) = delete;
    ~HostBuf() {
        if (p) cudaFreeHost(p);
    }
    cudaError_t ensure(size_t count) {
        if (p && count <= cap) return cudaSuccess;
        if (p) cudaFreeHost(p);
        p = nullptr;
        cap = 0;
        cudaError_t e = cudaHostAlloc(reinterpret_cast<void**>(&p), (count ? count : 1) * sizeof(T), cudaHostAllocDefault);
        if (e == cudaSuccess) cap = count;
        return e;
    }
};

// Device-side CCS copy in both CSR (row SpMV) and CSC (transposed SpMV) form.
struct DevCcs {
    uint32_t n = 0, m = 0, t = 0;
    std::vector<uint8_t> is_identity;
    std::vector<uint64_t> f_coeff;
    std::vector<uint32_t> f_exps;
    uint32_t n_terms = 0;
    // per matrix offsets into the packed arrays
    std::vector<uint64_t> nnz_off;
    DevBuf<uint64_t> csr_ptr;   // [t][n+1] (relative to nnz_off[j])
    DevBuf<uint32_t> csr_col;   // [nnz]
    DevBuf<uint64_t> csr_val;   // [nnz]
    DevBuf<uint64_t> csc_ptr;   // [t][m+1]
    DevBuf<uint32_t> csc_row;   // [nnz]
    DevBuf<uint64_t> csc_val;   // [nnz]
};
// Grow-only scratch owned by the context; valid until the next call that grows it.
inline cudaError_t ctx_scratch(neo_gpu_ctx* ctx, size_t bytes, void** p) {
    if (bytes > ctx->scratch_bytes) {
        const bool pooled = g_alloc_stream == ctx->stream;  // stream-ordered: no device-wide wait
        if (ctx->scratch) {
            if (pooled) {
                cudaFreeAsync(ctx->scratch, ctx->stream);
            } else {
                cudaStreamSynchronize(ctx->stream);
                cudaFree(ctx->scratch);
            }
            ctx->scratch = nullptr;
            ctx->scratch_bytes = 0;
        }
        cudaError_t e = pooled ? cudaMallocAsync(&ctx->scratch, bytes, ctx->stream) : ctx_malloc(ctx, &ctx->scratch, bytes);
        if (e != cudaSuccess) return e;
        ctx->scratch_bytes = bytes;
    }
    *p = ctx->scratch;
    return cudaSuccess;
}
int dev_ccs_upload(neo_gpu_ctx* ctx, const neo_ccs_desc* desc, DevCcs& out, bool want_csr = true);
// matrices of one launch (blockIdx.y): index, first nonzero, identity
struct MatSel {
    uint64_t off[16];
    uint8_t j[16], id[16];
};
inline MatSel mat_sel(const DevCcs& c, const int* js, uint32_t n) {  // js null: matrices 0..n-1
    MatSel s{};
    for (uint32_t q = 0; q < n && q < 16; q++) {
        const uint32_t j = js ? (uint32_t)js[q] : q;
        s.j[q] = (uint8_t)j;
        s.off[q] = c.nnz_off[j];
        s.id[q] = c.is_identity[j];
    }
    return s;
}

// A point of up to 32 coordinates as a kernel argument: it rides in the launch, where a
// small copy from pageable memory cost the host 6 to 8 us and the stream 1.5.
struct KPoint {
    gl::K x[32];
};
inline KPoint make_point(const gl::K* h, uint32_t n) {
    KPoint p{};
    for (uint32_t i = 0; i < n && i < 32; i++) p.x[i] = h[i];
    return p;
}

// Kernels callable from several translation units.  chi(point) over 2^nbits entries, the
// point on the host or on the device
int launch_chi_point(neo_gpu_ctx* ctx, const gl::K* h_point, uint32_t nbits, gl::K* d_out);
int launch_chi_table(neo_gpu_ctx* ctx, const gl::K* d_bits, uint32_t nbits, gl::K* d_out);
// chi(bits[j+1..nbits)) for every j < nbits, table j at 2^nbits - 2^(nbits-j), in one launch
int launch_suffix_chi_tables(neo_gpu_ctx* ctx, const gl::K* h_point, uint32_t nbits, gl::K* d_out);
int launch_me_y(neo_gpu_ctx* ctx, const DevCcs& ccs, const int8_t* d_Z, uint32_t n_w, uint64_t m,
                const gl::K* d_chi, uint32_t ell_n, uint32_t b, gl::K* d_vj_scratch, gl::K* d_y,
                gl::K* d_ysc);
// y[row][j] = sum_c Z[row][c] v[j][c] of R int8 digit rows (y layout [w][t][54]); *done = false
// (nothing launched) when m % 64 != 0 or t > 4
int launch_zrows(neo_gpu_ctx* ctx, const int8_t* d_Z, uint32_t R, uint64_t m, uint32_t t, const gl::K* d_v,
                 gl::K* d_y, bool* done);
// the RLC mix on the tensor cores (d_rot: [count][54][RLC_ROT_ROW], 16-byte aligned; d_Zs on
// four bytes, with MIX_PAD readable bytes behind the digits)
int launch_rlc_mix(neo_gpu_ctx* ctx, const int8_t* d_rot, const int8_t* d_Zs, uint32_t count, uint64_t m, int32_t* d_Zmix);
// bus openings y[w][c][rho] = sum_j Z[w 54 + rho][base + c steps + j] v[j]; *done = false
// (nothing launched) unless m, base and steps are multiples of 16
int launch_bus_rows(neo_gpu_ctx* ctx, const int8_t* d_Z, uint32_t n_w, uint64_t m, uint64_t base, uint64_t steps,
                    uint32_t ncols, const gl::K* d_v, gl::K* d_y, bool* done);
// What the caller knows about the digits of a commitment: any int8
// (TC_DIGITS_ANY: the cyclic tensor-core form), |digit| <= 63 by construction
// (TC_DIGITS_SMALL: the small-digit form, a violation is reported through the
// device error word), or nothing (TC_DIGITS_CHECK: the small-digit form, redone in
// the cyclic form on the device when a digit turned out too large).
enum { TC_DIGITS_ANY = 0, TC_DIGITS_SMALL = 1, TC_DIGITS_CHECK = 2 };
int launch_commit(neo_gpu_ctx* ctx, const int8_t* d_digits, uint32_t n_vec, uint64_t m, uint64_t* d_out,
                  int digits = TC_DIGITS_CHECK);
int tc_pp_prepare(neo_gpu_ctx* ctx, PPEntry* pp);
int launch_commit_tc(neo_gpu_ctx* ctx, const PPEntry* pp, const int8_t* d_digits, uint32_t n_vec, uint64_t* d_out,
                     int digits);
// reads and clears the device error word (synchronizes the stream)
int check_device_error(neo_gpu_ctx* ctx);

// AddressLookupOracle weight table and claimed sum from device columns (mem_oracle.cu);
// ws (may be null) keeps the temporaries across calls
struct AddrWs {
    DevBuf<gl::K> chi, part, out1;
    DevBuf<unsigned long long> acc;
};
int addr_weights_device(neo_gpu_ctx* ctx, uint32_t ell, const gl::K* d_rcycle, uint32_t A, const gl::K* d_has,
                        const gl::K* d_bits, const gl::K* d_table, uint64_t table_len, gl::K* d_w, gl::K* claim,
                        AddrWs* ws);
// Memory-oracle builds that reuse the object in *slot (mem_oracle.cu)
int mem_oracle_build_device(neo_gpu_ctx* ctx, int kind, uint32_t ell, const uint64_t* r_point, uint32_t ell_addr,
                            const uint64_t* r_addr, const uint64_t* init_at_r_addr, uint32_t n_cols,
                            const uint64_t* d_cols, const uint64_t* weights, uint64_t* claim,
                            neo_gpu_mem_oracle** slot);
int twist_addr_build_device(neo_gpu_ctx* ctx, int kind, uint32_t ell, const uint64_t* r_cycle, uint32_t ell_addr,
                            uint64_t n_init, const uint64_t* init_addr, const uint64_t* init_val,
                            const uint64_t* d_cols, neo_gpu_twist_addr** slot);

inline unsigned ceil_div(uint64_t a, uint64_t b) { return (unsigned)((a + b - 1) / b); }

// A kernel's dynamic shared-memory limit (cudaFuncAttributeMaxDynamicSharedMemorySize)
// is a process-wide attribute of the function.  Host threads that set it to
// their own launch's size would undo each other: a thread launching with 56 KB
// fails ("too many resources requested for launch") when another thread set
// 4 KB in between.  SmemLimit only ever raises the attribute, under a lock, so
// every launch that follows its own at_least() call stays within the limit.
struct SmemLimit {
    std::mutex mu;
    size_t cur = 48 * 1024;
    template <typename Kernel>
    cudaError_t at_least(Kernel* kernel, size_t bytes) {
        std::lock_guard<std::mutex> lk(mu);
        if (bytes > cur) cur = bytes;
        return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cur);
    }
};
