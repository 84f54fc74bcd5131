// rlc_tc.cu -- the Pi_RLC mix on the tensor cores (tcgen05 kind::i8), exact.
//
// Zmix[r][c] = sum_i sum_k rot_i[r][k] Z_i[k][c] over the integers
// (optimized_engine/common.rs:1221-1379): A = 128 columns of Z (rows of the tile are
// columns c, K runs over a witness's 54 digit rows, padded to 64), B = the 54 rows of
// rot_i, D = s32.  Two witnesses make a 128-byte K step.
//
// The digits lie column-contiguous and the tile wants K-contiguous: a lane loads four
// columns of four digit rows, transposes the 4 x 4 bytes by byte permutes and stores a
// word per column.  Every digit is read once, and three blocks per SM hide the loads.
// By dp4a, which issues slowly here, 13 witnesses of 2^10 columns took 29 us, of 2^14 40
// (three threads a column, each reading it all) and of 2^16 69; now 9.5, 10 and 26.
#include "internal.cuh"
#include "tc.cuh"

namespace {

constexpr int MT_COLS = 128, MT_N = 64, MT_T = 256;
constexpr int MT_A = MT_COLS * 128, MT_B = MT_N * 128, MT_STAGE = MT_A + MT_B;
constexpr uint32_t MT_TMEM = 64;
static_assert(RLC_ROT_ROW == 64, "a witness is 64 bytes of K");

struct MixArgs {
    const int8_t* rot;  // [count][54][RLC_ROT_ROW]
    const int8_t* Z;    // [count][54][m], and MIX_PAD bytes more
    uint32_t count;
    uint64_t m;
    int32_t* out;       // [54][m]
    volatile uint32_t* err;
};

// WORDS: every digit row begins on four bytes (m a multiple of 4); else four columns come
// from two words (13 witnesses of 2^14 - 1 columns: 15 us; byte by byte 49, by dp4a 39).
template <bool WORDS>
__global__ void __launch_bounds__(MT_T, 3) rlc_mix_tc_kernel(const MixArgs a) {
    extern __shared__ uint8_t s_raw[];
    __shared__ __align__(8) uint64_t s_done[2];
    __shared__ uint32_t s_tmem;
    uint8_t* stages = s_raw + ((1024 - (smem_u32(s_raw) & 1023)) & 1023);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint64_t c0 = blockIdx.x * (uint64_t)MT_COLS;
    const uint32_t n = (a.count + 1) / 2;
    if (tid == 0) {
        mbar_init(&s_done[0], 1);
        mbar_init(&s_done[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tmem_alloc<MT_TMEM>(&s_tmem);
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = s_tmem;

    // a warp has 8 of the column quads (warp & 3) and one witness of the step (warp >> 2);
    // a lane one quad and the K quads kq = lane / 8 + 4 e (rows 4 kq .. 4 kq + 3 of 54)
    const uint32_t h = warp >> 2, cq = (warp & 3) * 8 + (lane & 7), kl = lane >> 3;
    const uint64_t c = c0 + 4 * cq;
    const MixRows rows = {a.Z, a.m, a.count};
    uint32_t z[4][4], zn[4][4];  // zn: the words after (rows on any byte)
    uint4 rb[2];
    auto fetch = [&](uint32_t i) {
        const uint32_t w = 2 * i + h;
        const int8_t* zw = a.Z + (uint64_t)w * NEO_D * a.m + c;
        const bool on = w < a.count && c < a.m;
#pragma unroll
        for (int e = 0; e < 4; e++)
#pragma unroll
            for (int b = 0; b < 4; b++) {
                const uint32_t k = 4 * (kl + 4 * e) + b;
                const bool in = on && k < NEO_D;
                if constexpr (WORDS) {
                    z[e][b] = in ? __ldg(reinterpret_cast<const uint32_t*>(zw + (uint64_t)k * a.m)) : 0u;
                } else {
                    mix_fetch(rows, w, k, c, z[e][b], zn[e][b]);  // shifted when they are used
                }
            }
#pragma unroll
        for (int e = 0; e < 2; e++) {  // 16-byte piece q & 7 of row q / 8
            const uint32_t q = tid + MT_T * e, r = q >> 3, wr = 2 * i + ((q & 7) >> 2);
            rb[e] = r < NEO_D && wr < a.count
                        ? __ldg(reinterpret_cast<const uint4*>(a.rot + ((uint64_t)wr * NEO_D + r) * RLC_ROT_ROW + (q & 3) * 16))
                        : make_uint4(0, 0, 0, 0);
        }
    };
    fetch(0);
    uint32_t issued = 0;
    const uint32_t id = idesc_i8(MT_N, true, true);
    for (uint32_t i = 0; i < n; i++) {
        uint8_t* A = stages + (i & 1) * MT_STAGE;
        uint8_t* B = A + MT_A;
        bool ok = true;
        if (i >= 2 && lane == 0) ok = mbar_wait(&s_done[i & 1], ((i >> 1) & 1) ^ 1);
        __syncwarp();
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const uint32_t k = 64 * h + 4 * (kl + 4 * e);
            if constexpr (!WORDS) {
#pragma unroll
                for (int b = 0; b < 4; b++) z[e][b] = mix_quad(rows, 2 * i + h, 4 * (kl + 4 * e) + b, c, z[e][b], zn[e][b]);
            }
            const uint32_t l01 = __byte_perm(z[e][0], z[e][1], 0x5140), l23 = __byte_perm(z[e][2], z[e][3], 0x5140);
            const uint32_t h01 = __byte_perm(z[e][0], z[e][1], 0x7362), h23 = __byte_perm(z[e][2], z[e][3], 0x7362);
            *reinterpret_cast<uint32_t*>(A + sw128_at(4 * cq, k)) = __byte_perm(l01, l23, 0x5410);
            *reinterpret_cast<uint32_t*>(A + sw128_at(4 * cq + 1, k)) = __byte_perm(l01, l23, 0x7632);
            *reinterpret_cast<uint32_t*>(A + sw128_at(4 * cq + 2, k)) = __byte_perm(h01, h23, 0x5410);
            *reinterpret_cast<uint32_t*>(A + sw128_at(4 * cq + 3, k)) = __byte_perm(h01, h23, 0x7632);
        }
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const uint32_t q = tid + MT_T * e;
            *reinterpret_cast<uint4*>(B + sw128_at(q >> 3, (q & 7) * 16)) = rb[e];
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
        if (!okw) *a.err = 0x80u;
    }
    okw = __shfl_sync(0xffffffffu, okw, 0);
    asm volatile("tcgen05.fence::after_thread_sync;");
    // lane: column c0 + 32 (warp & 3) + lane; warps 0..3 output rows 0..31, 4..7 rows 32..53
    const uint64_t cc = c0 + (warp & 3) * 32 + lane;
    for (uint32_t r0 = (warp >> 2) * 32; r0 < (okw ? (warp >> 2) * 32 + 32 : 0); r0 += 16) {
        int x[16];
        const uint32_t taddr = tmem + ((uint32_t)((warp & 3) * 32) << 16) + r0;
        tmem_ld(taddr, x);
#pragma unroll
        for (int e = 0; e < 16; e++)
            if (cc < a.m && r0 + e < NEO_D) a.out[(uint64_t)(r0 + e) * a.m + cc] = x[e];
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;");
        tmem_dealloc<MT_TMEM>(tmem);
    }
}

}  // namespace

int launch_rlc_mix(neo_gpu_ctx* ctx, const int8_t* d_rot, const int8_t* d_Zs, uint32_t count, uint64_t m, int32_t* d_Zmix) {
    if (reinterpret_cast<uintptr_t>(d_Zs) & 3) return ctx->fail(NEO_ERR_ARG, "rlc: digits must begin on four bytes");
    MixArgs a{};
    a.rot = d_rot;
    a.Z = d_Zs;
    a.count = count;
    a.m = m;
    a.out = d_Zmix;
    a.err = ctx_host_err(ctx);
    constexpr size_t smem = 2 * MT_STAGE + 1024;
    auto launch = [&](auto kernel, SmemLimit& limit) -> int {
        NEO_CK(ctx, limit.at_least(kernel, smem));
        kernel<<<ceil_div(m, MT_COLS), MT_T, smem, ctx->stream>>>(a);
        NEO_LAUNCHED(ctx);
        return NEO_OK;
    };
    static SmemLimit words, bytes;
    if (m % 4 == 0) return launch(rlc_mix_tc_kernel<true>, words);
    return launch(rlc_mix_tc_kernel<false>, bytes);
}
