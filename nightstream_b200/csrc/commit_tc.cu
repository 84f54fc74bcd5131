// commit_tc.cu -- Ajtai commitment as an exact int8 tensor-core GEMM (tcgen05).
//
// c_i(X) = sum_j M[i][j](X) z_j(X) mod Phi_81 (crates/neo-ajtai/src/commit.rs:679-744),
// as a GEMM of PP byte limbs and windows of one short sequence per column:
//
//   D[(i,l)][(v,o)] = sum_{j, s<64} A[(i,l)][(j,s)] G_{v,j}[o + s]
//   A[(i,l)][(j,s)] = byte l of M[i][j][s]  (u8; 0 for s >= 54 and j = m, the pad of an odd m)
//
// M = 128 = kappa * 8 rows, K = 64 per column (one 128-byte K block holds
// exactly two columns).  Two forms of the sequence G (s8):
//
//  * Small digits (|z| <= 63): [X^r] X^s z mod Phi_81 is h(r - s) for r >= 27 and
//    -h(r - 27 - s) for r < 27, where h has period 81 and
//      h(x) = -z[x + 27] (-27 <= x < 0),  z[x] - z[x + 27] (0 <= x < 27),  z[x] (27 <= x < 54)
//    (X^54 = -X^27 - 1, X^81 = 1 mod Phi_81).  So the 54 output rows are the
//    windows o = 0..53 of G[w] = h(80 - w): row r = 80 - o for o >= 27, and
//    r = 26 - o with the finished sum negated for o < 27.  56 rows and
//    128 sequence bytes per vector, 7 chunks of 16 bytes per phase.
//  * Any int8 digit (cyclic): the product mod X^81 - 1, G[w] = z[(80 - w) mod 81]
//    (z[x] = 0 for x >= 54), rows o = 0..80, output row 80 - o, folded 81 -> 54
//    with X^54 = -X^27 - 1 when the sum is finished.  88 rows and 160 bytes per
//    vector, 9 chunks.
//
// Accumulation is int32 in TMEM; a CTA covers at most 512 K blocks, so
// |D| <= 255*128*65536 < 2^31: no overflow.  CTAs split K and groups of NV
// vectors.
//
// B is never materialised row by row.  Writing o = 16a + 8h + b, the window of
// row o is the 16-byte-aligned chunks a + k (k < 4) of the phase sequence
// G_p[x] = G[x + p], p = 8h + b.  So the builders write, per column, the 16
// phases as chunks laid out [chunk][h][v][b][16 B], and a no-swizzle K-major
// descriptor with 8-row-group stride 128 B and K-chunk stride LBO = NV*256 B
// walks all rows (a, h, v, b): row group g = (2a + h) NV + v sits at g*128 and
// its K chunk k at (a + k) LBO.
//
// One launch per call.  Warp roles of a CTA: a bulk-copy producer (A tiles,
// stored in HBM in the 128B-swizzled K-major layout, 16 KB per K block), the
// MMA issuer, four builder warps, and two transposer warps that read the digit
// rows (16 to 64 columns at a time) and write G straight into shared memory.  All
// eight warps are the epilogue then: it recombines the 8 limbs of every
// (i, column) mod q in registers and adds the value's 32-bit halves into 64-bit
// accumulators in L2 (exact and order-free); the last CTA of a vector group
// (ticket) reduces them, writes the commitments and leaves the accumulators zero.
//
// What bounds it, and what it measured, stands at commit_win_kernel.
#include "internal.cuh"
#include "tc.cuh"
#include <algorithm>

namespace {

constexpr int TC_A_BYTES = 128 * 128;       // 16 KB
constexpr int TC_BUILDERS = 128;            // warps 2..5: B builders
constexpr int TC_TRANSPOSERS = 64;          // warps 6, 7
constexpr int TC_MAX_KB = 512;              // K blocks per CTA (int32 overflow bound)
constexpr uint32_t TC_MIN_KB = 4;           // K blocks per CTA worth a CTA of its own (1 vector, m = 2^10: 12.3 us with 2, 11.8 with 4, 12.3 with 8)
// ---------------------------------------------------------------------------
// prep: PP -> pre-swizzled u8 limb tiles  PPL[kb][row][128 B]
// ---------------------------------------------------------------------------
// One CTA per K block kb (columns 2kb, 2kb+1): thread (i, jj, g) loads the 8
// coefficients s = 8g..8g+7 of M[i][2kb+jj] (one coalesced 64-byte run),
// splits them into 8 byte planes l and stores each 8-byte piece at row
// (i, l), K offset 64 jj + 8g of the swizzled tile in shared memory; the
// 16 KB tile then goes out as 1024 contiguous 16-byte stores.  The last K
// block of an odd m has zeros in place of its second column.
__global__ void __launch_bounds__(256) pp_limbs_kernel(const uint64_t* __restrict__ pp, uint32_t kappa, uint64_t m,
                                                       uint8_t* __restrict__ ppl) {
    __shared__ __align__(16) uint8_t tile[TC_A_BYTES];
    const uint64_t kb = blockIdx.x;
    const uint32_t t = threadIdx.x;
    const uint32_t i = t >> 4, jj = (t >> 3) & 1, g = t & 7;
    uint64_t w[8];
#pragma unroll
    for (int e = 0; e < 8; e++) {
        const uint32_t s_ = g * 8 + e;
        w[e] = (i < kappa && s_ < NEO_D && kb * 2 + jj < m) ? pp[((uint64_t)i * m + kb * 2 + jj) * NEO_D + s_] : 0;
    }
    const uint32_t k = jj * 64 + g * 8;  // K byte offset of this 8-byte piece
#pragma unroll
    for (int l = 0; l < 8; l++) {
        uint64_t v = 0;
#pragma unroll
        for (int e = 0; e < 8; e++) v |= ((w[e] >> (8 * l)) & 0xFFull) << (8 * e);
        const uint32_t row = i * 8 + l;
        *reinterpret_cast<uint64_t*>(tile + row * 128 + ((((k >> 4) ^ (row & 7)) << 4) | (k & 15))) = v;
    }
    __syncthreads();
    uint4* dst = reinterpret_cast<uint4*>(ppl + kb * TC_A_BYTES);
    const uint4* src = reinterpret_cast<const uint4*>(tile);
#pragma unroll
    for (int q = 0; q < TC_A_BYTES / 16 / 256; q++) dst[t + 256 * q] = src[t + 256 * q];
}


// ---------------------------------------------------------------------------
// main kernel
// ---------------------------------------------------------------------------
struct TcArgs {
    const uint8_t* ppl;        // pre-swizzled limb tiles
    const int8_t* digits;      // [n_vec][54][m]
    const uint8_t* G;          // not fused: [n_groups][n_kb] records
    unsigned long long* acc;   // [n_groups][2][16][NPAD] sums acc0, acc1 (zero between calls)
    uint32_t* tickets;         // [n_groups] (zero between calls)
    uint64_t* out;             // [n_vec][kappa][54]
    uint32_t* err;             // error word (timeouts)
    uint32_t* bad;             // small form: bit 16 set when a sequence entry leaves int8
    const uint32_t* only_if;   // null, or the whole launch does nothing while *only_if is zero
    uint64_t m;
    uint32_t n_vec, kappa, n_groups, n_ksplit, kb_per_cta, n_kb;
};

// Shapes of one form (CYC: any int8 digit) at NV vectors per CTA.  FUSED: the
// CTA's transposer warps make G from the digits; else win_seq_kernel made it.
template <int NV, bool CYC, bool FUSED>
struct Win {
    static constexpr int OUT = CYC ? 81 : NEO_D;        // windows that make outputs
    static constexpr int BLOCKS = CYC ? 6 : 4;          // 16-row blocks per vector
    static constexpr int NCH = BLOCKS + 3;              // 16-byte chunks of a phase
    static constexpr int SEQ = CYC ? 160 : 128;         // bytes of G
    // MMA N: whole 8-row groups up to the last output (56 or 88 rows a vector), in 16s
    static constexpr int NPAD = ((OUT + 7) / 8 * 8 * NV + 15) / 16 * 16;
    static constexpr uint32_t LBO = 2 * NV * 128;       // K-direction core-matrix stride
    static constexpr int BCOL = NCH * LBO;              // B bytes per column
    static constexpr int B_BYTES = 2 * BCOL;            // two columns per K block
    // two CTAs per SM: while one waits on its rings the other issues MMAs (one
    // CTA with 6 vectors, N = 2 x 192 and rings of 6 / 4 took 320 us where 4
    // vectors and two CTAs took 298: 12 vectors at m = 2^16)
    static constexpr int CTAS = 2;
    static constexpr int THREADS = 256;                 // 8 warps: two per TMEM lane group in the epilogue
    static constexpr int TILE = TC_TRANSPOSERS / NV;    // fused: columns per G tile, one (column, vector) per transposer thread
    static constexpr int KPT = FUSED ? TILE / 2 : 1;    // K blocks per G buffer
    // strides of a vector and of a column in a G buffer.  Odd counts of 16 bytes
    // between vectors: the builders' word loads (lanes = vectors, phases) fall
    // on distinct banks; fused also between columns, for the transposers'
    // 16-byte stores (lanes = columns).  Else a K block's record is one copy.
    static constexpr int VP = FUSED ? SEQ + 16 : 2 * SEQ + 16;
    static constexpr int CP = FUSED ? NV * VP + (NV == 1 ? 0 : 16) : SEQ;
    static constexpr int G_BYTES = FUSED ? TILE * CP : NV * VP;
    // WPK builder warps make one K block: lanes (warp, sub, v, b) share its four
    // (column, half of the chunks) tasks
    static constexpr int WPK = NV == 4 ? (FUSED ? 4 : 2) : 1;
    static constexpr int SUB = 4 / NV;
    static constexpr int TASKS = 4 / (SUB * WPK);       // per lane
    static constexpr int CPP = (NCH + 1) / 2;           // chunks per task
    static constexpr int BSTAGES = NV == 4 ? (FUSED ? 2 : 3) : 4;
    static constexpr int ASTAGES = NV == 2 && CYC ? 3 : 4;
    // groups of warps that build: at most BSTAGES, so that a warp waiting for a B
    // buffer has seen that buffer's use before the last one end (phase parities
    // stay unambiguous)
    static constexpr int NB = TC_BUILDERS / 32 / WPK;
    static constexpr int GSTAGES = FUSED ? 2 : 4;
    static constexpr int SMEM = ASTAGES * TC_A_BYTES + BSTAGES * B_BYTES + GSTAGES * G_BYTES;
    static constexpr int DYN = SMEM + 1024 /*alignment*/ + 256 /*barriers*/;
    static constexpr uint32_t TMEM_COLS = NPAD <= 64 ? 64 : (NPAD <= 128 ? 128 : 256);
    static_assert(NPAD <= 256 && NPAD % 16 == 0, "one MMA per K step (M = 128: N <= 256, N % 16 == 0)");
    static_assert(B_BYTES % 128 == 0 && G_BYTES % 16 == 0 && (VP / 16) % 2 == 1 && (!FUSED || (CP / 16) % 2 == 1), "alignment");
    static_assert((OUT + 7) / 8 % 2 == 1, "an odd count of 8-row groups: the last chunk is read at h = 0 only");
    static_assert(NB <= BSTAGES && TASKS >= 1, "builder warps");
    static_assert(FUSED ? KPT >= BSTAGES : GSTAGES > BSTAGES, "a G buffer's last use is over when a B buffer is free");
    static_assert((2 * (ASTAGES + BSTAGES + GSTAGES) + 1) * 8 + 4 <= 256, "barrier space");
    static_assert(DYN + 64 + 1024 <= 233472 / CTAS, "shared memory of the resident CTAs");
    static_assert(TMEM_COLS * CTAS <= 512, "TMEM columns of the resident CTAs");
};

// One digit; volatile keeps a batch of loads together in program order.  Rows
// are m bytes apart, and lines of L1 would be claimed for 16 bytes each: .cg.
__device__ __forceinline__ int ld_digit(const int8_t* p) {
    int v;
    asm volatile("ld.global.cg.s8 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

// acc0 + 2^32 acc1 mod q of one (i, column): sums of signed terms below 2^35
__device__ __forceinline__ uint64_t acc_value(unsigned long long acc0, unsigned long long acc1) {
    const uint64_t h = gl::from_i64((long long)acc1);
    return gl::add(gl::from_i64((long long)acc0), gl::reduce128(h << 32, h >> 32));
}

template <bool CYC>
__device__ __forceinline__ void build_sequence(const int (&z)[NEO_D], uint4* dst, bool& bad) {
    constexpr int SEQ = CYC ? 160 : 128;
#pragma unroll
    for (int q = 0; q < SEQ / 16; q++) {
        uint32_t w4[4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
            uint32_t word = 0;
#pragma unroll
            for (int b = 0; b < 4; b++) {
                const int w = q * 16 + e * 4 + b;
                int g = 0;  // entries no output reads (A is zero for s >= 54) stay zero
                if constexpr (CYC) {
                    const int x = w <= 80 ? 80 - w : 161 - w;
                    g = x >= 0 && x < NEO_D ? z[x] : 0;
                } else {
                    g = w < 27 ? -z[26 - w]
                      : w < 54 ? z[80 - w]
                      : w < 81 ? z[80 - w] - z[107 - w]
                      : w < 108 ? -z[107 - w] : 0;
                    if (w >= 54 && w < 81) bad |= g > 127 || g < -127;   // g and -g fit int8
                    if (w < 54) bad |= z[w] == -128;                      // and so does -z
                }
                word |= (uint32_t)(uint8_t)(int8_t)g << (8 * b);
            }
            w4[e] = word;
        }
        dst[q] = make_uint4(w4[0], w4[1], w4[2], w4[3]);
    }
}

// Entry w of G of four columns as one word (byte c = column c), from four-column
// words of the digit rows.
__device__ __forceinline__ uint32_t seq_word(const uint32_t (&z)[NEO_D], int w) {
    return w < 27 ? __vneg4(z[26 - w])
         : w < 54 ? z[80 - w]
         : w < 81 ? __vsub4(z[80 - w], z[107 - w])
         : w < 108 ? __vneg4(z[107 - w]) : 0;
}

// G of every (vector, column), one record of NV * VP bytes per (vector group, K
// block) so that the GEMM fetches it with one copy: vector v, column jj at
// v VP + jj SEQ.  A block makes 128 columns of one vector, four per thread
// (V4: digit rows in aligned 4-byte words; else byte loads): a warp reads whole
// 128-byte lines, the sequences are staged in shared memory and written in runs
// of 2 SEQ bytes.
constexpr int SEQ_COLS = 128, SEQ_T = SEQ_COLS / 4;
template <bool V4>
__global__ void __launch_bounds__(SEQ_T) win_seq_kernel(const int8_t* __restrict__ digits, uint64_t m, uint32_t n_kb,
                                                        uint8_t* __restrict__ G, uint32_t* __restrict__ bad_flag) {
    using S = Win<4, false, false>;
    constexpr int NV = 4;
    constexpr int PITCH = S::SEQ + 16;  // per column; a thread's four columns are SEQ_T apart in the stage
    __shared__ __align__(16) uint8_t s_out[SEQ_COLS * PITCH];
    // (vector, columns): a grid of one dimension, as the vectors may be more than 65535
    const uint32_t per = (n_kb + SEQ_COLS / 2 - 1) / (SEQ_COLS / 2), v = blockIdx.x / per, tid = threadIdx.x;
    const uint64_t j0 = (uint64_t)(blockIdx.x % per) * SEQ_COLS, j = j0 + 4 * tid;
    const int8_t* zv = digits + (uint64_t)v * NEO_D * m;
    uint32_t z[NEO_D];
    if constexpr (V4) {  // m % 4 == 0: a word is inside the row or past it
        const int8_t* zp = zv + (j < m ? j : 0);
#pragma unroll
        for (int x = 0; x < NEO_D; x++) z[x] = __ldg(reinterpret_cast<const uint32_t*>(zp + (uint64_t)x * m));
#pragma unroll
        for (int x = 0; x < NEO_D; x++) z[x] = j < m ? z[x] : 0;
    } else {
#pragma unroll
        for (int x = 0; x < NEO_D; x++) {
            uint32_t w = 0;
#pragma unroll
            for (int c = 0; c < 4; c++) {  // past the row (and the pad of an odd m's last K block): zero
                const uint32_t d = j + c < m ? (uint8_t)__ldg(zv + (uint64_t)x * m + j + c) : 0u;
                w |= d << (8 * c);
            }
            z[x] = w;
        }
    }
    // a digit of -128, or a difference that leaves int8 or whose negative does
    uint32_t bad = 0;
#pragma unroll
    for (int x = 0; x < NEO_D; x++) bad |= __vcmpeq4(z[x], 0x80808080u);
#pragma unroll
    for (int x = 0; x < 27; x++) {
        const uint32_t d = __vsub4(z[x], z[x + 27]);
        bad |= ((z[x] ^ z[x + 27]) & (z[x] ^ d)) & 0x80808080u;  // signed overflow
        bad |= __vcmpeq4(d, 0x80808080u);
    }
    if (bad) atomicOr(bad_flag, 1u << 16);
#pragma unroll
    for (int q = 0; q < S::SEQ / 16; q++) {
        uint32_t o[4][4];  // [column][word]
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int w = 16 * q + 4 * e;
            const uint32_t a = seq_word(z, w), b = seq_word(z, w + 1), c = seq_word(z, w + 2), d = seq_word(z, w + 3);
            const uint32_t ab0 = __byte_perm(a, b, 0x5140), ab1 = __byte_perm(a, b, 0x7362);
            const uint32_t cd0 = __byte_perm(c, d, 0x5140), cd1 = __byte_perm(c, d, 0x7362);
            o[0][e] = __byte_perm(ab0, cd0, 0x5410);
            o[1][e] = __byte_perm(ab0, cd0, 0x7632);
            o[2][e] = __byte_perm(ab1, cd1, 0x5410);
            o[3][e] = __byte_perm(ab1, cd1, 0x7632);
        }
#pragma unroll
        for (int c = 0; c < 4; c++)  // column 4 tid + c at stage row c SEQ_T + tid: a store's lanes on distinct banks
            *reinterpret_cast<uint4*>(s_out + (c * SEQ_T + tid) * PITCH + q * 16) = make_uint4(o[c][0], o[c][1], o[c][2], o[c][3]);
    }
    __syncwarp();
    constexpr uint32_t CH = S::SEQ / 16;
    const uint64_t kb0 = j0 / 2;
    const uint32_t cols = 2 * (uint32_t)min((uint64_t)SEQ_COLS / 2, n_kb - kb0);
    uint8_t* out = G + ((uint64_t)(v / NV) * n_kb + kb0) * (NV * S::VP) + (v % NV) * S::VP;
#pragma unroll 4
    for (uint32_t e = tid; e < cols * CH; e += SEQ_T) {
        const uint32_t c = e / CH, q = e % CH;
        *reinterpret_cast<uint4*>(out + (uint64_t)(c / 2) * (NV * S::VP) + (c & 1) * S::SEQ + q * 16) =
            *reinterpret_cast<const uint4*>(s_out + ((c & 3) * SEQ_T + (c >> 2)) * PITCH + q * 16);
    }
}
static_assert(SEQ_T == 32, "win_seq_kernel: one warp, synchronised as one");

// A producer's last copies have landed before its CTA ends, also after another role gave up
// (bounded waits; when nobody did, the MMAs have waited for them already).
__device__ __noinline__ void drain(uint64_t* full, uint32_t stages, uint32_t issued) {
    for (uint32_t it = issued > stages ? issued - stages : 0; it < issued; it++)
        if (!mbar_wait(&full[it % stages], (it / stages) & 1)) break;
}

// What bounds it (calls back to back, us).  One vector: HBM (537 MB of tiles at m = 2^16:
// 87 = 6.2 TB/s; before, with separate sequence and reduce launches and 112-byte sequences
// per half of the rows, 127).  Groups of four: shared memory.  Per K block the MMAs
// read 352 wavefronts of 128 bytes, the builders store 91 and load 68, the A tile
// and G arrive with 136, against 478 cycles of MMA (N = 224; MMAs alone reach 4.5
// POPS): 12 ternary vectors at m = 2^16 take 290 (361 before), of which the
// sequence launch 34; m = 2^14 87 (119), m = 2^10 23 (43).  Windows of one
// 81-periodic sequence need 7 chunks a phase where one sequence per half of the
// rows needed 10.  One launch instead of four: 1 vector at m = 2^10 11.4 (26), of which
// 9.7 the kernel.  Any digit: 5 vectors at m = 10006 50 (94); an odd m, which ran on CUDA
// cores, 1 vector at m = 5001 17 (806).
template <int NV, bool CYC, bool FUSED>
__global__ void __launch_bounds__(Win<NV, CYC, FUSED>::THREADS, Win<NV, CYC, FUSED>::CTAS)
commit_win_kernel(const __grid_constant__ TcArgs a) {
    using S = Win<NV, CYC, FUSED>;
    if (a.only_if && __ldcg(a.only_if) == 0) return;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    // 1024-align the tile buffers (dynamic smem base alignment is not guaranteed)
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sA = smem;                                        // [ASTAGES][16 KB]
    uint8_t* sB = sA + S::ASTAGES * TC_A_BYTES;                // [BSTAGES][B_BYTES]
    uint8_t* sG = sB + S::BSTAGES * S::B_BYTES;                // [GSTAGES][G_BYTES]
    uint64_t* bars = reinterpret_cast<uint64_t*>(sG + S::GSTAGES * S::G_BYTES);
    uint64_t* full_a = bars;                                   // A tile landed
    uint64_t* empty_a = full_a + S::ASTAGES;                   // MMAs done reading the A tile
    uint64_t* full_b = empty_a + S::ASTAGES;                   // B phases built
    uint64_t* empty_b = full_b + S::BSTAGES;                   // MMAs done reading the B phases
    uint64_t* full_g = empty_b + S::BSTAGES;                   // G buffer written
    uint64_t* empty_g = full_g + S::GSTAGES;                   // builders done reading the G buffer
    uint64_t* done = empty_g + S::GSTAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
    __shared__ int s_abort;
    __shared__ bool s_last;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t group = blockIdx.x % a.n_groups, ks = blockIdx.x / a.n_groups;
    const uint32_t kb0 = ks * a.kb_per_cta;
    const uint32_t kb1 = min(a.n_kb, kb0 + a.kb_per_cta);
    const uint32_t nkb = kb1 > kb0 ? kb1 - kb0 : 0;
    const uint32_t nvalid = min((uint32_t)NV, a.n_vec - group * NV);  // vectors of this group

    if (threadIdx.x == 0) {
        s_abort = 0;
        for (int s = 0; s < S::ASTAGES; s++) {
            mbar_init(&full_a[s], 1);
            mbar_init(&empty_a[s], 1);
        }
        for (int s = 0; s < S::BSTAGES; s++) {
            mbar_init(&full_b[s], S::WPK);
            mbar_init(&empty_b[s], 1);
        }
        for (int s = 0; s < S::GSTAGES; s++) {
            mbar_init(&full_g[s], FUSED ? TC_TRANSPOSERS / 32 : 1);
            mbar_init(&empty_g[s], S::KPT * S::WPK);
        }
        mbar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc<S::TMEM_COLS>(tmem_slot);
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = *tmem_slot;
    // a role's wait, by lane 0 for its warp so that every exit is warp-uniform:
    // 0 go, 1 timed out, 2 another role aborted
    auto warp_wait = [&](bool go) -> uint32_t {
        uint32_t st = go ? (s_abort ? 2u : 0u) : 1u;
        return __shfl_sync(0xffffffffu, st, 0);
    };

    if (warp == 0) {
        // ---- producer: A tiles ----
        if (lane == 0) {
            uint32_t it = 0;
            for (; it < nkb; it++) {
                const int s = it % S::ASTAGES;
                const uint32_t ph = (it / S::ASTAGES) & 1;
                if (it >= S::ASTAGES && !mbar_wait(&empty_a[s], ph ^ 1)) { atomicOr(a.err, 1u); s_abort = 1; break; }
                if (s_abort) break;
                mbar_expect_tx(&full_a[s], TC_A_BYTES);
                bulk_g2s(sA + s * TC_A_BYTES, a.ppl + (uint64_t)(kb0 + it) * TC_A_BYTES, TC_A_BYTES, &full_a[s]);
            }
            drain(full_a, S::ASTAGES, it);
        }
    } else if (warp == 1) {
        // ---- MMA issuer: one M = 128, N = NPAD MMA per 32-byte K step ----
        if (lane == 0) {
            const uint32_t id = idesc_i8(S::NPAD, false, true);
            for (uint32_t it = 0; it < nkb; it++) {
                const int sa = it % S::ASTAGES, sb = it % S::BSTAGES;
                if (!mbar_wait(&full_a[sa], (it / S::ASTAGES) & 1) || !mbar_wait(&full_b[sb], (it / S::BSTAGES) & 1)) {
                    atomicOr(a.err, 2u);
                    s_abort = 1;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;");
                const uint32_t a0 = smem_u32(sA + sa * TC_A_BYTES), b0 = smem_u32(sB + sb * S::B_BYTES);
#pragma unroll
                for (int k = 0; k < 4; k++) {  // column k/2, s in [32(k%2), 32(k%2)+32): chunks 2(k%2), 2(k%2)+1
                    const uint32_t bcol = b0 + (k >> 1) * S::BCOL + (k & 1) * 2 * S::LBO;
                    mma_i8(tmem, sw128_desc(a0 + 32 * k), ns_desc(bcol, S::LBO), id, (it > 0 || k > 0) ? 1u : 0u);
                }
                mma_commit(&empty_a[sa]);  // tiles free once these MMAs complete
                mma_commit(&empty_b[sb]);
            }
            mma_commit(done);
        }
    } else if (!FUSED && warp >= 2 + TC_BUILDERS / 32) {
        // ---- second producer: the records of G (one thread of the last two warps) ----
        if (lane == 0 && warp == 2 + TC_BUILDERS / 32) {
            uint32_t it = 0;
            for (; it < nkb; it++) {
                const int s = it % S::GSTAGES;
                if (it >= S::GSTAGES && !mbar_wait(&empty_g[s], ((it / S::GSTAGES) & 1) ^ 1)) { atomicOr(a.err, 0x20u); s_abort = 1; break; }
                if (s_abort) break;
                mbar_expect_tx(&full_g[s], S::G_BYTES);
                bulk_g2s(sG + s * S::G_BYTES, a.G + ((uint64_t)group * a.n_kb + kb0 + it) * S::G_BYTES, S::G_BYTES, &full_g[s]);
            }
            drain(full_g, S::GSTAGES, it);
        }
    } else if (FUSED && warp >= 2 + TC_BUILDERS / 32) {
        // ---- transposers: thread (column, vector) of a G tile ----
        const int tt = threadIdx.x - 64 - TC_BUILDERS;
        const int col = tt % S::TILE, v = tt / S::TILE;
        const int8_t* zv = a.digits + (uint64_t)(group * NV + v) * NEO_D * a.m;
        const uint32_t nt = (nkb + S::KPT - 1) / S::KPT;
        bool bad = false;
        for (uint32_t t = 0; t < nt; t++) {
            const int sg = t & 1;
            const uint64_t j = 2ull * (kb0 + t * S::KPT) + col;
            const bool live = (uint32_t)v < nvalid && j < a.m && j < 2ull * kb1;
            // all 54 loads are issued here, in flight together and across the wait
            // (a thread without a column reads column 0 and drops it)
            const int8_t* zp = live ? zv + j : a.digits;
            int z[NEO_D];
#pragma unroll
            for (int x = 0; x < NEO_D; x++) z[x] = ld_digit(zp + (uint64_t)x * a.m);
            bool go = true;
            if (lane == 0 && t >= 2) go = mbar_wait(&empty_g[sg], ((t >> 1) & 1) ^ 1);
            const uint32_t st = warp_wait(go);
            if (st == 1 && lane == 0) {
                atomicOr(a.err, 0x20u);
                s_abort = 1;
            }
            if (st) break;
#pragma unroll
            for (int x = 0; x < NEO_D; x++) z[x] = live ? z[x] : 0;
            build_sequence<CYC>(z, reinterpret_cast<uint4*>(sG + sg * S::G_BYTES + col * S::CP + v * S::VP), bad);
            __syncwarp();
            if (lane == 0) mbar_arrive(&full_g[sg]);
        }
        if (!CYC && bad) atomicOr(a.bad, 1u << 16);
    } else {
        // ---- B builders: WPK warps make every NB-th K block, so that NB are in
        // the making.  Lane (sub, v, b < 8), task (column jj, half of
        // the chunks): CPP chunks of both phases p = b + 8h, G_p = G[16c + p,
        // 16c + p + 16), at [jj][c][h][v][b]; the phases share the words read
        // once.  A warp's stores fill whole 128-byte rows ----
        const int b = lane & 7, v = (lane >> 3) % NV, sub = lane / (8 * NV);
        const uint32_t sh = 8 * (b & 3);
        for (uint32_t it = (warp - 2) / S::WPK; it < nkb; it += S::NB) {
            const int sb = it % S::BSTAGES;
            const uint32_t t = it / S::KPT, kt = it % S::KPT;  // G buffer and the K block in it
            const int sg = t % S::GSTAGES;
            bool go = true;
            if (lane == 0) {
                // empty_b first: once the MMAs of K block it - BSTAGES are done, every
                // earlier use of G buffer sg is over (GSTAGES > BSTAGES), so its phase
                // parity cannot be mistaken for the one before the last
                if (it >= S::BSTAGES) go = mbar_wait(&empty_b[sb], ((it / S::BSTAGES) & 1) ^ 1);
                if (go) go = mbar_wait(&full_g[sg], (t / S::GSTAGES) & 1);
            }
            const uint32_t st = warp_wait(go);
            if (st == 1 && lane == 0) {
                atomicOr(a.err, 4u);
                s_abort = 1;
            }
            if (st) break;
#pragma unroll
            for (int task = 0; task < S::TASKS; task++) {
                const int tk = (task * S::WPK + (warp - 2) % S::WPK) * S::SUB + sub, jj = tk & 1, c0 = (tk >> 1) * S::CPP;
                const uint32_t* src = reinterpret_cast<const uint32_t*>(sG + sg * S::G_BYTES + (2 * kt + jj) * S::CP +
                                                                        v * S::VP + 16 * c0) + (b >> 2);
                uint32_t w[4 * S::CPP + 3];
#pragma unroll
                for (int q = 0; q < 4 * S::CPP + 3; q++) w[q] = src[q];
                uint8_t* dst = sB + sb * S::B_BYTES + jj * S::BCOL + c0 * S::LBO + v * 128 + b * 16;
#pragma unroll
                for (int c = 0; c < S::CPP; c++) {
                    if (c0 + c >= S::NCH) break;
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        if (h && c0 + c >= S::NCH - 1) break;  // the last 16-row block has its first 8 rows only
                        const int o = 4 * c + 2 * h;
                        *reinterpret_cast<uint4*>(dst + h * (NV * 128) + c * S::LBO) =
                            make_uint4(__funnelshift_r(w[o], w[o + 1], sh), __funnelshift_r(w[o + 1], w[o + 2], sh),
                                       __funnelshift_r(w[o + 2], w[o + 3], sh), __funnelshift_r(w[o + 3], w[o + 4], sh));
                    }
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&full_b[sb]);
                mbar_arrive(&empty_g[sg]);
            }
        }
    }
    // ---- epilogue, every warp: lane group warp & 3, every other 32 columns.  Lane
    // (i, l) holds limb row l of output row i; three exchange steps turn 8 columns
    // of 8 limbs into one column per lane, as L + 2^32 H with L and H the sums of
    // its low and high four limbs (|.| < 2^56) ----
    uint32_t okw = 0;  // lane 0 waits for the warp
    // the issuer's last commit covers every MMA of the CTA: waited for after an abort too,
    // before the TMEM and the shared memory go back
    if (lane == 0) okw = (nkb > 0 && mbar_wait(done, 0) && !s_abort) ? 1u : 0u;
    const bool ok = __shfl_sync(0xffffffffu, okw, 0) != 0;
    if (nkb > 0 && !ok && lane == 0) atomicOr(a.err, 8u);
    asm volatile("tcgen05.fence::after_thread_sync;");
    {
        const int lg = warp & 3;  // TMEM lane group this warp may access
        const uint32_t i = (uint32_t)(lg * 4 + (lane >> 3));
        const bool u4 = lane & 4, u2 = lane & 2, u1 = lane & 1;
        const int col8 = (u2 ? 4 : 0) + (u1 ? 2 : 0) + (u4 ? 1 : 0);  // the lane's column of each eight
        unsigned long long* acc0 = a.acc + ((uint64_t)group * 32 + i) * S::NPAD + col8;
        unsigned long long* acc1 = acc0 + 16 * S::NPAD;
        constexpr uint32_t STEPS = (S::NPAD + 31) / 32;  // TMEM is allocated past the last whole 32 columns
        for (uint32_t step = warp >> 2; step < (ok ? STEPS : 0); step += 2) {
            // CTAs start at different columns, so that they do not all add to the same lines at once
            const int cb = (int)((step + ks) % STEPS * 32);
            uint32_t x[32];
            const uint32_t taddr = tmem + ((uint32_t)(lg * 32) << 16) + (uint32_t)cb;
            tmem_ld(taddr, x);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const uint32_t* y = x + 8 * q;
                long long s4[4], s2[2];
#pragma unroll
                for (int c = 0; c < 4; c++) {  // limbs l, l + 2
                    const int keep = (int)(u2 ? y[c + 4] : y[c]);
                    const int got = __shfl_xor_sync(0xffffffffu, (int)(u2 ? y[c] : y[c + 4]), 2);
                    s4[c] = (long long)(u2 ? got : keep) + (long long)(u2 ? keep : got) * 65536;
                }
#pragma unroll
                for (int c = 0; c < 2; c++) {  // limbs l, l + 1 (and l + 2, l + 3)
                    const long long keep = u1 ? s4[c + 2] : s4[c];
                    const long long got = __shfl_xor_sync(0xffffffffu, u1 ? s4[c] : s4[c + 2], 1);
                    s2[c] = (u1 ? got : keep) + (u1 ? keep : got) * 256;
                }
                const long long keep = u4 ? s2[1] : s2[0];
                const long long got = __shfl_xor_sync(0xffffffffu, u4 ? s2[0] : s2[1], 4);
                const long long L = u4 ? got : keep, H = u4 ? keep : got;
                const int g = cb / 8 + q, vv = g % NV, ah = g / NV;  // row group (a, h), vector
                // L + 2^32 H with 2^64 = 2^32 - 1: (L_lo - H_hi) + 2^32 (L_hi + H_lo + H_hi)
                if ((uint32_t)vv < nvalid && 8 * ah + col8 < S::OUT && i < a.kappa) {
                    const long long hh = H >> 32;
                    atomicAdd(acc0 + 8 * g, (unsigned long long)((L & 0xFFFFFFFFll) - hh));
                    atomicAdd(acc1 + 8 * g, (unsigned long long)((L >> 32) + (H & 0xFFFFFFFFll) + hh));
                }
            }
        }
        __threadfence();
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;");
        tmem_dealloc<S::TMEM_COLS>(tmem);
    }
    if (threadIdx.x == 0) s_last = atomicInc(a.tickets + group, a.n_ksplit - 1) == a.n_ksplit - 1;
    __syncthreads();
    if (!s_last) return;
    // ---- the group's last CTA: outputs, then zero accumulators for the next call.
    // 64 threads per (vector, row i), one output row each; the loads of 4 pairs
    // are in flight together ----
    __threadfence();
    unsigned long long* ga = a.acc + (uint64_t)group * 32 * S::NPAD;
    const int r = threadIdx.x & 63;
    if (r < NEO_D) {
        // windows of output r: the small form's one, the cyclic form's two (folded)
        const int o1 = CYC || r >= 27 ? 80 - r : 26 - r, o2 = r >= 27 ? 53 - r : 26 - r;
        const unsigned long long* p1 = ga + 8 * ((o1 >> 3) * NV) + (o1 & 7);
        const unsigned long long* p2 = ga + 8 * ((o2 >> 3) * NV) + (o2 & 7);
        const uint32_t pairs = nvalid * 16;
        for (uint32_t e0 = threadIdx.x >> 6; e0 < pairs; e0 += 16) {
            unsigned long long w[4][CYC ? 4 : 2];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const uint32_t e = min(e0 + 4 * u, pairs - 1), off = (e & 15) * S::NPAD + (e >> 4) * 8;
                w[u][0] = __ldcg(p1 + off);
                w[u][1] = __ldcg(p1 + off + 16 * S::NPAD);
                if constexpr (CYC) {
                    w[u][2] = __ldcg(p2 + off);
                    w[u][3] = __ldcg(p2 + off + 16 * S::NPAD);
                }
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const uint32_t e = e0 + 4 * u, i = e & 15, v = e >> 4;
                uint64_t c = acc_value(w[u][0], w[u][1]);
                if constexpr (CYC) c = gl::sub(c, acc_value(w[u][2], w[u][3]));
                else if (r < 27) c = gl::neg(c);
                if (e < pairs && i < a.kappa) a.out[((uint64_t)(group * NV + v) * a.kappa + i) * NEO_D + r] = c;
            }
        }
    }
    __syncthreads();
    for (uint32_t e = threadIdx.x; e < 16 * S::NPAD; e += S::THREADS) reinterpret_cast<ulonglong2*>(ga)[e] = make_ulonglong2(0, 0);
}

// The context's commitment workspace: accumulators and tickets that every
// launch finds and leaves zero, and the digit-check flag.
int commit_ws(neo_gpu_ctx* ctx, uint32_t n_groups, size_t acc_words, TcArgs* a, uint32_t** flag) {
    if (n_groups > ctx->commit_groups || acc_words > ctx->commit_words) {
        const uint32_t groups = std::max<uint32_t>({n_groups, ctx->commit_groups, 16});
        const size_t words = std::max(acc_words, ctx->commit_words);
        const size_t bytes = 256 + ((size_t)groups * 4 + 255) / 256 * 256 + words * 8;
        const bool pooled = g_alloc_stream == ctx->stream;
        if (ctx->commit_buf) {
            if (pooled) {
                cudaFreeAsync(ctx->commit_buf, ctx->stream);
            } else {
                cudaStreamSynchronize(ctx->stream);
                cudaFree(ctx->commit_buf);
            }
            ctx->commit_buf = nullptr;
            ctx->commit_groups = 0;
            ctx->commit_words = 0;
        }
        void* p = nullptr;
        NEO_CK(ctx, pooled ? cudaMallocAsync(&p, bytes, ctx->stream) : ctx_malloc(ctx, &p, bytes));
        ctx->commit_buf = p;
        NEO_CK(ctx, cudaMemsetAsync(p, 0, bytes, ctx->stream));
        ctx->commit_groups = groups;
        ctx->commit_words = words;
    }
    uint8_t* p = reinterpret_cast<uint8_t*>(ctx->commit_buf);
    *flag = reinterpret_cast<uint32_t*>(p);
    a->tickets = reinterpret_cast<uint32_t*>(p + 256);
    a->acc = reinterpret_cast<unsigned long long*>(p + 256 + ((size_t)ctx->commit_groups * 4 + 255) / 256 * 256);
    return NEO_OK;
}

// K blocks per CTA up to which a group of four small-digit vectors is fused: one
// launch less, but the transposers read the digit rows 16 bytes at a time, which
// costs more than win_seq_kernel once that hides behind enough K blocks (12
// vectors, L2 flushed before a call: m = 2^14 100.4 us fused, 96.9 apart; 2^15 168 and
// 169, 2^16 308 and 309; on new digits without the flush 2^16 345 and 341).  One and two
// vectors, and any digits, are fused at every size (1 vector at m = 2^16, when it was
// built apart too: 91 us fused, 104 apart).
constexpr uint32_t FUSED_KB = 64;

template <int NV, bool CYC, bool FUSED>
int launch_gemm(neo_gpu_ctx* ctx, const TcArgs& a) {
    using S = Win<NV, CYC, FUSED>;
    static SmemLimit limit;
    NEO_CK(ctx, limit.at_least(commit_win_kernel<NV, CYC, FUSED>, S::DYN));
    commit_win_kernel<NV, CYC, FUSED><<<a.n_groups * a.n_ksplit, S::THREADS, S::DYN, ctx->stream>>>(a);
    NEO_LAUNCHED(ctx);
    return NEO_OK;
}

template <int NV, bool CYC>
int launch_win(neo_gpu_ctx* ctx, TcArgs a) {
    a.n_groups = (a.n_vec + NV - 1) / NV;
    // whole waves of 148 SMs x the CTAs one SM holds, at most TC_MAX_KB K
    // blocks per CTA and not fewer than TC_MIN_KB: a CTA with less does not pay
    // for its launch, its sums and its ticket
    uint32_t n_ksplit;
    for (uint32_t waves = 1;; waves++) {
        n_ksplit = std::max(1u, (148 * Win<NV, CYC, true>::CTAS * waves) / a.n_groups);
        n_ksplit = std::min(n_ksplit, (a.n_kb + TC_MIN_KB - 1) / TC_MIN_KB);
        if ((a.n_kb + n_ksplit - 1) / n_ksplit <= TC_MAX_KB) break;
    }
    a.kb_per_cta = (a.n_kb + n_ksplit - 1) / n_ksplit;
    a.n_ksplit = (a.n_kb + a.kb_per_cta - 1) / a.kb_per_cta;
    if constexpr (NV == 4 && !CYC) {
        if (a.kb_per_cta > FUSED_KB) {
            void* G = nullptr;
            NEO_CK(ctx, ctx_scratch(ctx, (size_t)a.n_groups * a.n_kb * Win<4, false, false>::G_BYTES, &G));
            uint8_t* g = reinterpret_cast<uint8_t*>(G);
            a.G = g;
            const uint64_t grid64 = (uint64_t)((a.n_kb + SEQ_COLS / 2 - 1) / (SEQ_COLS / 2)) * a.n_vec;
            if (grid64 > 0x7FFFFFFFull) return ctx->fail(NEO_ERR_UNSUPPORTED, "commit: too many vectors for one launch");
            const unsigned grid = (unsigned)grid64;
            if (a.m % 4 == 0 && reinterpret_cast<uintptr_t>(a.digits) % 4 == 0)
                win_seq_kernel<true><<<grid, SEQ_T, 0, ctx->stream>>>(a.digits, a.m, a.n_kb, g, a.bad);
            else
                win_seq_kernel<false><<<grid, SEQ_T, 0, ctx->stream>>>(a.digits, a.m, a.n_kb, g, a.bad);
            NEO_LAUNCHED(ctx);
            return launch_gemm<4, false, false>(ctx, a);
        }
    }
    return launch_gemm<NV, CYC, true>(ctx, a);
}

// Vectors per CTA.  Small digits: 4 (N = 224) reads each A tile from shared
// memory once per four vectors; one or two vectors alone take their own size
// instead of padding.  Any digit: 2 (N = 176), the most that leaves TMEM and
// shared memory for two CTAs per SM.
int launch_small(neo_gpu_ctx* ctx, const TcArgs& a) {
    if (a.n_vec == 1) return launch_win<1, false>(ctx, a);
    if (a.n_vec == 2) return launch_win<2, false>(ctx, a);
    return launch_win<4, false>(ctx, a);
}
int launch_any(neo_gpu_ctx* ctx, const TcArgs& a) {
    return a.n_vec == 1 ? launch_win<1, true>(ctx, a) : launch_win<2, true>(ctx, a);
}
size_t acc_words(uint32_t n_vec) { return ((size_t)n_vec + 3) / 4 * 4 * 32 * 96; }  // both forms: at most 88 rows, with room a vector

}  // namespace

// ---------------------------------------------------------------------------
int tc_pp_prepare(neo_gpu_ctx* ctx, PPEntry* pp) {
    if (pp->kappa * 8 > 128) return ctx->fail(NEO_ERR_UNSUPPORTED, "tensor-core commit: kappa <= 16");
    pp->tc = false;
    const uint64_t n_kb = (pp->m + 1) / 2;
    if (!pp->d_pp_limbs) {  // size depends on m only
        const cudaError_t e = ctx_malloc(ctx, reinterpret_cast<void**>(&pp->d_pp_limbs), n_kb * TC_A_BYTES);
        if (e == cudaErrorMemoryAllocation && pp->m % 2) {
            // 8 KB of tiles a column beside 8 kappa 54 bytes of PP: an odd column count, which the
            // CUDA-core kernels serve too, does without them
            cudaGetLastError();
            pp->d_pp_limbs = nullptr;
            return NEO_OK;
        }
        NEO_CK(ctx, e);
    }
    pp_limbs_kernel<<<(unsigned)n_kb, 256, 0, ctx->stream>>>(pp->d_pp, pp->kappa, pp->m, pp->d_pp_limbs);
    NEO_LAUNCHED(ctx);
    NEO_CK(ctx, ctx_sync(ctx));
    pp->tc = true;
    return NEO_OK;
}

int launch_commit_tc(neo_gpu_ctx* ctx, const PPEntry* pp, const int8_t* d_digits, uint32_t n_vec, uint64_t* d_out,
                     int digits) {
    TcArgs a{};
    a.ppl = pp->d_pp_limbs;
    a.digits = d_digits;
    a.out = d_out;
    a.err = ctx->d_err;
    a.m = pp->m;
    a.n_vec = n_vec;
    a.kappa = pp->kappa;
    a.n_kb = (uint32_t)((pp->m + 1) / 2);
    uint32_t* flag = nullptr;
    if (int rc = commit_ws(ctx, (n_vec + (n_vec > 1)) / (n_vec > 1 ? 2 : 1), acc_words(n_vec), &a, &flag)) return rc;
    if (digits == TC_DIGITS_ANY) return launch_any(ctx, a);
    // the caller's promise covers an even m, and a broken one is reported; else
    // a digit that leaves the small form's range has the second launch redo the
    // commitment in the general form (it ends at once when there was none)
    const bool promised = digits == TC_DIGITS_SMALL && pp->m % 2 == 0;
    a.bad = promised ? ctx->d_err : flag;
    if (!promised) NEO_CK(ctx, cudaMemsetAsync(flag, 0, 4, ctx->stream));
    if (int rc = launch_small(ctx, a)) return rc;
    if (promised) return NEO_OK;
    a.only_if = flag;
    return launch_any(ctx, a);
}
