// gemm_pair.cu -- kernel (c): prompt-sized dequant-GEMM on the 5th-generation tensor cores, two SMs per tile.
//
// y[M][N] (+)= x[M][K] . dequant(W[N][K])^T for M > 64 activation rows: what LowBitLinear.forward asks of xe_linear.forward_new
// during prefill (reference low_bit_linear.py:700-708).  The same kernel serves an MLP's first half (act(gate) * up in the
// epilogue) and the routed feed-forwards of a mixture of experts (one launch over every expert's rows).
//
// A cluster of two CTAs computes a tile of 256 features x N tokens (N = 16 .. 256) with tcgen05.mma.cta_group::2: the EXPANDED
// WEIGHTS are the A operand (128 features per CTA), the tokens are B, and each CTA stages HALF of the tokens.  What bounds the
// one-CTA tile of 256 tokens x 128 features it replaced was the L2: 32 KB of activations + 4.4 KB of packed weights per CTA and
// k-block of 0.46 us are 12 TB/s over the chip, and four 53 KB stages left no depth to hide it; a pair moves 16 + 4.4 KB per CTA
// for the same arithmetic.  At 128-token tiles the bound was the chain load -> expand -> MMA through one ring (0.33 us per
// k-block, the MMAs 0.14): here activations, packed weights and expanded tiles have rings of their own, so the expansion runs
// ahead of the activations and four groups of warps have four k-blocks in flight.  Measured per k-block: 0.19 us up to 170 tokens
// (fp16; see pair_plan for the other paces), 0.282 at 256, where the tensor pipe is busy 512 of 525 clocks; 14336 x 4096 at 4000
// tokens 1357 -> 1494 TFLOP/s, 4096 x 11008 at 512 tokens in fp16 59.7 -> 42.6 us.  All of a cool GPU in short recorded chains; in a
// long stream of calls, under the power cap, the latter takes 51.  At 128 tokens the MMAs need 256 of 360 clocks: A and B both come from
// shared memory, beside the expansion's stores.
//   warp 0       TMA: this CTA's half of the tokens, boxes of 32 rows x 64 elements (128-byte swizzle), ring of kX slots;
//   warp 1       CTA 0: issues the MMAs (M = 256, N, K = 16; four per k-block) in warp-uniform control flow, one commit per ring
//                (multicast to both CTAs); CTA 1: relays "my half has landed" to CTA 0's barrier;
//   warp 2       bulk copies of the PACKED weights of two 64-row groups (codes, scales, minima), ring of kP slots;
//   warp 3       allocates TMEM (2 x 256 columns: the epilogue of a tile overlaps the next tile's main loop);
//   warps 4-19   four groups of four: group (k-block mod 4) expands the codes to fp16 / bf16 (scale applied with one multiply per
//                pair, one rounding) into the K-major 128B-swizzled A slot it owns;
//   warps 20-23  epilogue: TMEM lane = feature, column = token.  The two 64-row groups are interleaved by 16 rows, so that with a
//                gate group and an up group in one tile a warp's two runs of 16 lanes hold gate and up of the same features.
// The signals between the two CTAs are plain arrivals: with cluster-scope release / acquire on them (a full memory fence per
// arrival) a k-block took 0.75 us instead of 0.25; what they order is shared memory, written behind a proxy fence and read by the
// tensor cores of the SM that wrote it.
// Every wait is bounded: see tc_common.cuh.
#include <type_traits>
#include "tc_pair.cuh"

namespace lowbit {
namespace gemmtc {

constexpr int kPairThreads = 32 * 24;
constexpr int kPairTok = 256;                 // most tokens of a tile
constexpr int kPairDeq0 = 4, kPairEpi0 = 20;  // first dequant / epilogue warp
constexpr int kMaxExperts = 256;

template <int QT> struct PairSmem {
    static constexpr int kGroup = PackedBlock<QT>::kGroup;
    static constexpr int kPacked = 2 * kGroup;                         // two 64-row groups, one k-block
    static constexpr int kLut = Expand<QT>::kLutBytes;
    static constexpr int kTab = 2 * (kMaxExperts + 4) * 4;             // tile prefix and row offsets of the experts
    static constexpr int kOut = 2 * 32 * 256;                          // epilogue: two chunks of 32 tokens x 128 features, 16 bits
    static constexpr int kA = 4;                                       // slots of 16 KB, one per dequant group
    static constexpr int kP = 8;                                       // see the dequant loop: twice the groups
    static constexpr int kFixed = 1024 + 512 + kTab + kLut + kOut + kA * kTileBytesAB + kP * kPacked;
    static constexpr int kX = (232448 - kFixed) / kTileBytesAB < 8 ? (232448 - kFixed) / kTileBytesAB : 8;      // slots of 128 rows x 128 bytes
    static constexpr int kTotal = kFixed + kX * kTileBytesAB;
    static_assert(kX >= 3 && kP == 2 * kA && kTotal <= 232448, "ring depths");
    static_assert((3 * kX + 2 * kP + 2 * kA + 5) * 8 + 8 <= 512, "barrier region");
};

struct PairArgs {
    const uint8_t* w;
    const uint8_t* w2;                 // MLP: the up projection (w = gate); the tile's second 64-row group
    const unsigned long long* tab;     // experts: device addresses of w / w2 per expert, row offsets [n_experts + 1]
    const unsigned long long* tab2;
    const int* offs;
    int n_experts;
    TiledGeom G;
    int M;
    int tt;                            // tokens per tile (multiple of 16); experts: chosen per expert
    int n_fp;                          // pairs of feature tiles
    int ksplit;
    int act;                           // 0: y = x W^T; 1 / 2: y = act(x W^T) * (x W2^T)
    void* y; int y_dtype;
    const void* bias; int accumulate;
    float* part;                       // ksplit > 1: [ksplit][M][N]
    Waits waits;
};

// gate (lanes 0-15) and up (lanes 16-31) of 16 features and 16 tokens -> act(gate) * up: the halves exchange one token of every two,
// so that all lanes work; out[i] is token 2 i + half
__device__ __forceinline__ void gate_up(const float (&v)[16], int act, int half, float (&out)[8]) {
#pragma unroll
    for (int j = 0; j < 16; j += 2) {
        const float got = __shfl_xor_sync(0xffffffffu, half ? v[j] : v[j + 1], 16);
        out[j >> 1] = apply_act(half ? got : v[j], act) * (half ? v[j + 1] : got);
    }
}

// GRAD: the product with the transposed weights, dx[M][K] = g[M][N] . dequant(W[N][K]), in the same loop: a k-block is 64 rows of W, a
// feature tile 128 of its columns (two k-blocks of the packed layout, side by side in memory).  The expanded tile is the same image in
// shared memory -- 64 elements of one weight row to a 128-byte line -- read as an MN-major operand, so nothing is transposed (K-major in
// its place takes the same time).  Weights are rounded once from their 32-bit value (expand_once).  What it replaces wrote the
// dequantised matrix to memory for a library product: forward and backward of 1024 rows, 11008 x 4096, through MatMulLowBit, nf4 bf16
// 193 -> 181 us, sym_int4 186 -> 159, of 20 rows, 14336 x 14336, nf4 259 -> 136; recorded, of 3000 rows, 8192 x 8192, sym_int4, 668 -> 593.
template <int QT, bool BF, bool GRAD>
__global__ void __launch_bounds__(kPairThreads, 1)
pair_kernel(const __grid_constant__ CUtensorMap xmap, const PairArgs A) {
    using E = Expand<QT>;
    using SM = PairSmem<QT>;
    constexpr int KX = SM::kX, KP = SM::kP, KA = SM::kA;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;       // 128B swizzle wants 1024-byte alignment
    const uint32_t xring = base, aring = base + KX * kTileBytesAB, pring = aring + KA * kTileBytesAB;
    const uint32_t bars = pring + KP * SM::kPacked;                    // a multiple of 16 bytes behind the packed ring
    const uint32_t lut0 = bars + 512, obuf = lut0 + SM::kLut;
    auto x_full = [&](int s) { return bars + s * 8; };
    auto x_empty = [&](int s) { return bars + (KX + s) * 8; };
    auto xp_full = [&](int s) { return bars + (2 * KX + s) * 8; };                     // CTA 0: the other half has landed
    auto p_full = [&](int s) { return bars + (3 * KX + s) * 8; };
    auto p_empty = [&](int s) { return bars + (3 * KX + KP + s) * 8; };
    auto a_full = [&](int s) { return bars + (3 * KX + 2 * KP + s) * 8; };             // CTA 0: both CTAs' tiles are expanded
    auto a_empty = [&](int s) { return bars + (3 * KX + 2 * KP + KA + s) * 8; };
    auto tmem_full = [&](int b) { return bars + (3 * KX + 2 * KP + 2 * KA + b) * 8; };
    auto tmem_empty = [&](int b) { return bars + (3 * KX + 2 * KP + 2 * KA + 2 + b) * 8; };   // CTA 0: both epilogues have drained it
    const uint32_t drained = bars + (3 * KX + 2 * KP + 2 * KA + 4) * 8;               // every MMA that was issued is done
    const uint32_t tmem_slot = drained + 8;
    int* const cum = reinterpret_cast<int*>(smem_raw + (obuf + SM::kOut - smem_u32(smem_raw)));    // experts: tiles before expert e
    int* const off = cum + kMaxExperts + 4;                                                        //          rows before expert e

    // the warp index through a shuffle: the compiler then treats everything derived from it as warp-uniform
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int rank = (int)(blockIdx.x & 1);
    const uint32_t lut = lut0 + (GRAD ? 8 * (lane & 15) : 4 * lane);
    if constexpr (E::kLutBytes > 0) {
        if (GRAD) fill_nf4_pairs(smem_raw + (lut0 - smem_u32(smem_raw)), threadIdx.x, kPairThreads);
        else E::fill_lut(smem_raw + (lut0 - smem_u32(smem_raw)), threadIdx.x, kPairThreads);
    }
    const int nb = GRAD ? (int)(A.G.rows >> 6) : (int)A.G.nb;          // k-blocks of the product

    if (threadIdx.x == 0) {
        for (int s = 0; s < KX; s++) { mbar_init(x_full(s), 1); mbar_init(x_empty(s), 1); mbar_init(xp_full(s), 1); }
        for (int s = 0; s < KP; s++) { mbar_init(p_full(s), 1); mbar_init(p_empty(s), 4); }
        for (int s = 0; s < KA; s++) { mbar_init(a_full(s), 8); mbar_init(a_empty(s), 1); }
        for (int b = 0; b < 2; b++) { mbar_init(tmem_full(b), 1); mbar_init(tmem_empty(b), 8); }
        mbar_init(drained, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // an expert's rows in tiles of at most 256 tokens, evenly cut; few rows are another kernel's
    auto tiles_of = [](int rows) { return rows > (int)kExactRows ? (rows + kPairTok - 1) / kPairTok : 0; };
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (warp == 2 && A.offs) {
        int before = 0;
        for (int e0 = 0; e0 < A.n_experts; e0 += 32) {
            const int e = e0 + lane, lo = A.offs[min(e, A.n_experts)], hi = A.offs[min(e + 1, A.n_experts)];
            int t = tiles_of(hi - lo);
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) { const int o = __shfl_up_sync(0xffffffffu, t, d); if (lane >= d) t += o; }
            if (e < A.n_experts) { cum[e + 1] = before + t; off[e + 1] = hi; }
            before += __shfl_sync(0xffffffffu, t, 31);
        }
        if (lane == 0) { cum[0] = 0; off[0] = 0; }
    }
    if (warp == 3) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync_all();                                    // both CTAs' barriers exist before anybody signals them
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    uint32_t tmem_base;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem_base) : "r"(tmem_slot));

    // ---- work units: (feature pair, token tile, K split), feature pairs fastest: the clusters running at one moment share a token
    // tile's activations in L2 and stream different weights
    const int n_tiles = A.offs ? cum[A.n_experts] : (A.M + A.tt - 1) / A.tt;
    const int n_units = n_tiles * A.n_fp * A.ksplit, stride = (int)(gridDim.x >> 1);
    struct Unit { int m0, m_end, n_tok, ft, e, ks, kb0, kb1; };
    auto decode = [&](int unit, Unit& U) {                 // units of one role come in rising order: U.e only moves forward
        const int fp = unit % A.n_fp, rest = unit / A.n_fp;
        int t = rest;
        if (A.offs) {
            while (cum[U.e + 1] <= t) U.e++;
            const int lo = off[U.e], rows = off[U.e + 1] - lo, n = tiles_of(rows);
            const int tt = ((rows + n - 1) / n + 15) & ~15;
            U.m0 = lo + (t - cum[U.e]) * tt;
            U.m_end = min(off[U.e + 1], U.m0 + tt);
            U.ks = 0;
        } else {
            t = rest % n_tiles;
            U.ks = rest / n_tiles;
            U.m0 = t * A.tt;
            U.m_end = min(A.M, U.m0 + A.tt);
        }
        U.n_tok = max(16, (U.m_end - U.m0 + 15) & ~15);
        U.ft = 2 * fp + rank;
        U.kb0 = A.ksplit == 1 ? 0 : (U.ks * nb) / A.ksplit;
        U.kb1 = A.ksplit == 1 ? nb : ((U.ks + 1) * nb) / A.ksplit;
    };
    Unit U;
    U.e = 0;
    // The next launch may start when the blocks end (the release that an exit is).  Released at the start of the last units it took SMs as they
    // happened to be free, and launches with a split K range ran 3 to 7 % longer than without any overlap: fp8_e4m3, 4096 x 14336 at 513 rows
    // 73.5 us without, 76.3 so, 71.2 now; nf4, 300 rows 46.2, 49.3, 42.7.  Where nf4's K range is whole or short the early release is the better
    // one, the next blocks fill their table meanwhile: 1024 x 1024 at 129 rows 12.3 us without, 9.2 so, 10.1 at the end
    const bool early = SM::kLut > 0 && (A.ksplit == 1 || nb <= 8 * A.ksplit);
    const uint32_t leader = elect_leader();
    int s = 0, round = 0;                                  // the two copying warps' place in their ring

    if (warp == 0) {
        // ================= activations: this CTA's half of the tile's tokens =================
        for (int unit = blockIdx.x >> 1; unit < n_units; unit += stride) {
            decode(unit, U);
            if (early && unit + stride >= n_units) asm volatile("griddepcontrol.launch_dependents;");     // the cluster's last unit
            const int half = U.n_tok >> 1, boxes = (half + 31) >> 5, row0 = U.m0 + rank * half;
            for (int kb = U.kb0; kb < U.kb1; kb++) {
                if (!mbar_wait_lim(x_empty(s), (uint32_t)((round & 1) ^ 1), A.waits)) goto done;
                mbar_expect_tx_w(x_full(s), boxes * 4096, leader);
                for (int i = 0; i < boxes; i++)
                    tma_load_2d_w(xring + s * kTileBytesAB + i * 4096, &xmap, kb * 64, row0 + i * 32, x_full(s), leader);
                if (++s == KX) { s = 0; round++; }
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            // ================= MMA issuer =================
            int sx = 0, rx = 0, it = 0, ti = 0;
            bool ready = false;
            for (int unit = blockIdx.x >> 1; unit < n_units; unit += stride, ti++) {
                decode(unit, U);
                // c F32 (1<<4), a/b format (0 f16, 1 bf16), both K-major (GRAD: A MN-major), N (>>3 at bit 17), M = 256 (>>4 at bit 24)
                const uint32_t idesc = (GRAD ? 1u << 15 : 0u) | (1u << 4) | ((BF ? 1u : 0u) << 7) | ((BF ? 1u : 0u) << 10) | (((uint32_t)U.n_tok >> 3) << 17) | ((256u >> 4) << 24);
                const int buf = ti & 1;
                if (!mbar_wait_lim(tmem_empty(buf), (uint32_t)(((ti >> 1) & 1) ^ 1), A.waits)) goto done;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t acc = tmem_base + buf * kPairTok;
                for (int kb = U.kb0; kb < U.kb1; kb++) {
                    const int sa = it & 3;
                    if (!mbar_wait3_lim(ready, x_full(sx), (uint32_t)(rx & 1), xp_full(sx), (uint32_t)(rx & 1), a_full(sa), (uint32_t)((it >> 2) & 1), A.waits)) goto done;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    uint64_t ad = make_desc(aring + sa * kTileBytesAB);
                    const uint64_t xd = make_desc(xring + sx * kTileBytesAB);
                    // MN-major: LBO = the next 64 features (8 KB), SBO = the next eight lines; a step of 16 lines
                    if (GRAD) ad = (ad & ~((uint64_t)0x3fff << 16)) | ((uint64_t)(8192 >> 4) << 16);
#pragma unroll
                    for (int k4 = 0; k4 < 4; k4++)           // the address field counts 16-byte units
                        umma2_f16_w(acc, ad + (uint64_t)((GRAD ? k4 * 2048 : k4 * 32) >> 4), xd + (uint64_t)((k4 * 32) >> 4), idesc, (kb > U.kb0 || k4 > 0) ? 1u : 0u, leader);
                    umma2_commit_w(a_empty(sa), leader);
                    umma2_commit_w(x_empty(sx), leader);
                    if (++sx == KX) { sx = 0; rx++; }
                    it++;
                    // asked here, answered while the MMAs above are being issued
                    ready = mbar_test3(x_full(sx), (uint32_t)(rx & 1), xp_full(sx), (uint32_t)(rx & 1), a_full(it & 3), (uint32_t)((it >> 2) & 1));
                }
                umma2_commit_w(tmem_full(buf), leader);
            }
        } else {
            // ================= relay: CTA 1's half has landed =================
            int sx = 0, rx = 0;
            for (int unit = blockIdx.x >> 1; unit < n_units; unit += stride) {
                decode(unit, U);
                for (int kb = U.kb0; kb < U.kb1; kb++) {
                    if (!mbar_wait_lim(x_full(sx), (uint32_t)(rx & 1), A.waits)) goto done;
                    if (lane == 0) mbar_arrive_at(xp_full(sx), 0);
                    if (++sx == KX) { sx = 0; rx++; }
                }
            }
        }
    } else if (warp == 2) {
        // ================= packed weights of this CTA's two 64-row groups =================
        const int n_rg = (int)(A.G.rows >> 6);
        for (int unit = blockIdx.x >> 1; unit < n_units; unit += stride) {
            decode(unit, U);
            const uint8_t* w0 = A.offs ? reinterpret_cast<const uint8_t*>(A.tab[U.e]) : A.w;
            const uint8_t* w1 = A.act ? (A.offs ? reinterpret_cast<const uint8_t*>(A.tab2[U.e]) : A.w2) : w0;
            // the last pair's second tile may not exist: it repeats the last group and stores nothing
            const int64_t rg0 = min(A.act ? U.ft : 2 * U.ft, n_rg - 1), rg1 = min(A.act ? U.ft : 2 * U.ft + 1, n_rg - 1);
            const int kb_end = A.waits.limit < 0 ? (U.kb0 + U.kb1) / 2 : U.kb1;
            for (int kb = U.kb0; kb < kb_end; kb++) {
                if (!mbar_wait_lim(p_empty(s), (uint32_t)((round & 1) ^ 1), A.waits)) goto done;
                mbar_expect_tx_w(p_full(s), SM::kPacked, leader);
#pragma unroll
                for (int gi = 0; gi < 2; gi++) {
                    const uint8_t* wb = gi ? w1 : w0;
                    // GRAD: row group kb, the tile's two blocks of 64 columns
                    const int64_t u = GRAD ? (int64_t)kb * A.G.nb + min(2 * (int64_t)U.ft + gi, A.G.nb - 1) : (gi ? rg1 : rg0) * nb + kb;
                    const uint32_t dst = pring + s * SM::kPacked + gi * SM::kGroup;
                    bulk_g2s_w(dst, wb + u * PackedBlock<QT>::kSuper, PackedBlock<QT>::kSuper, p_full(s), leader);
                    bulk_g2s_w(dst + PackedBlock<QT>::kSuper, wb + A.G.off_s + u * 128, 128, p_full(s), leader);
                    if (E::kHasMin) bulk_g2s_w(dst + PackedBlock<QT>::kSuper + 128, wb + A.G.off_m + u * 128, 128, p_full(s), leader);
                }
                if (++s == KP) { s = 0; round++; }
            }
            if (kb_end < U.kb1) goto done;
        }
    } else if (warp >= kPairDeq0 && warp < kPairEpi0) {
        // ================= dequant: group (warp - 4) / 4 takes every fourth k-block; a warp expands 16 rows of either row group =================
        const int grp = (warp - kPairDeq0) >> 2, dw = (warp - kPairDeq0) & 3;
        const int g = lane >> 2, t = lane & 3;
        // rows 32 dw + g, + 8; + 16, + 24 for the second group.  GRAD: lines 16 dw + g, + 8 of either block
        const uint32_t row0 = aring + grp * kTileBytesAB + (GRAD ? 2 : 4) * dw * 1024 + g * 128, row_step = GRAD ? 8192 : 2048;
        // k-blocks are numbered over all units of the cluster: `end` behind the unit's last, `it` this group's next
        int end = 0, it = grp;
        for (int unit = blockIdx.x >> 1; unit < n_units; unit += stride) {
            decode(unit, U);
            end += U.kb1 - U.kb0;
            for (; it < end; it += 4) {
                const int sp = it & (KP - 1), rp = it / KP;
                // the slot's last trip (k-block it - 8) was this group's own, so the parity is unambiguous
                if (!mbar_wait_lim(p_full(sp), (uint32_t)(rp & 1), A.waits)) goto done;
                const uint32_t pk = pring + sp * SM::kPacked;
                typename E::Codes cw[2];
                uint32_t dq[2], mq[2] = {0u, 0u};
#pragma unroll
                for (int gi = 0; gi < 2; gi++) {
                    const uint32_t gb = pk + gi * SM::kGroup;
                    E::load(gb + dw * E::kTileBytes, lane, cw[gi]);
                    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(dq[gi]) : "r"(gb + PackedBlock<QT>::kSuper + g * 16 + dw * 4));
                    if (E::kHasMin) asm volatile("ld.shared.u32 %0, [%1];" : "=r"(mq[gi]) : "r"(gb + PackedBlock<QT>::kSuper + 128 + g * 16 + dw * 4));
                }
                // expanded into registers while the MMAs still read the slot's last tile
                uint32_t lo[2][8], hi[2][8];
#pragma unroll
                for (int gi = 0; gi < 2; gi++) {
                    if constexpr (GRAD) { expand_once<QT, BF>(cw[gi], dq[gi], mq[gi], lut, lo[gi], hi[gi]); continue; }
                    const __half2 d2 = u2h(dq[gi]), m2 = u2h(mq[gi]);
                    const __half2 dlo = __low2half2(d2), dhi = __high2half2(d2);
                    const __half2 mlo = __low2half2(m2), mhi = __high2half2(m2);
#pragma unroll
                    for (int k4 = 0; k4 < 4; k4++) {
                        uint32_t a[4];
                        E::run(cw[gi], k4, dlo, dhi, mlo, mhi, lut, a);
                        if (BF) {
#pragma unroll
                            for (int i = 0; i < 4; i++) a[i] = h2_to_bf2(a[i]);
                        }
                        lo[gi][2 * k4] = a[0]; lo[gi][2 * k4 + 1] = a[2];
                        hi[gi][2 * k4] = a[1]; hi[gi][2 * k4 + 1] = a[3];
                    }
                }
                if (!mbar_wait_lim(a_empty(grp), (uint32_t)(((it >> 2) & 1) ^ 1), A.waits)) goto done;
#pragma unroll
                for (int gi = 0; gi < 2; gi++)
#pragma unroll
                    for (int q = 0; q < 2; q++) {               // k-steps 2q, 2q+1 -> one 16-byte chunk per row; 128B swizzle: chunk ^ (row & 7)
                        const uint32_t at = row0 + gi * row_step + (uint32_t)((2 * t + q) ^ g) * 16;
                        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(lo[gi][4 * q]), "r"(lo[gi][4 * q + 1]), "r"(lo[gi][4 * q + 2]), "r"(lo[gi][4 * q + 3]) : "memory");
                        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at + 1024), "r"(hi[gi][4 * q]), "r"(hi[gi][4 * q + 1]), "r"(hi[gi][4 * q + 2]), "r"(hi[gi][4 * q + 3]) : "memory");
                    }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // generic-proxy writes -> async-proxy (MMA) reads
                __syncwarp();
                // the packed slot goes back only here: the stores above used every loaded code.  An arrival right behind the expansion could
                // be issued while the second row group's loads were still under way, and the next copy then overtook them
                if (lane == 0) { mbar_arrive(p_empty(sp)); mbar_arrive_at(a_full(grp), 0); }
            }
        }
    } else if (warp >= kPairEpi0) {
        // ================= epilogue: TMEM lanes 32 * (warp % 4) .. + 31 =================
        const int quarter = warp & 3, half = lane >> 4, e_tid = threadIdx.x - 32 * kPairEpi0;
        const int64_t N = GRAD ? A.G.k : A.G.rows;
        const bool wide = A.ksplit > 1 || A.y_dtype == DT_F32;        // 32-bit results go straight to memory
        uint32_t chunk = 0;
        int ti = 0;
        for (int unit = blockIdx.x >> 1; unit < n_units; unit += stride, ti++) {
            decode(unit, U);
            const int buf = ti & 1, rows = U.m_end - U.m0;
            const int64_t f0 = (int64_t)U.ft * (A.act ? 64 : 128);
            const int64_t n = GRAD ? f0 + 32 * quarter + lane : f0 + (A.act ? 0 : 64 * half) + 16 * quarter + (lane & 15);
            const bool valid = f0 < N;                                // the last pair's second tile may not exist
            float b = 0.0f;
            if (A.bias && valid && A.ksplit == 1)
                b = A.y_dtype == DT_F32 ? ((const float*)A.bias)[n] : A.y_dtype == DT_F16 ? __half2float(((const __half*)A.bias)[n])
                                                                                          : __bfloat162float(((const __nv_bfloat16*)A.bias)[n]);
            // the four warps go on together or not at all: they meet at named barriers below
            uint32_t go = mbar_wait_lim(tmem_full(buf), (uint32_t)((ti >> 1) & 1), A.waits) ? 1u : 0u;
            asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %0, 0;\n\tbarrier.cta.red.and.pred q, 1, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "+r"(go)::"memory");
            if (!go) goto done;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t acc = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * kPairTok);
            if (wide) {
                // 32-bit results leave from the lanes: a warp stores a token's 32 features.  Conditions outside, as below
                auto unit_out = [&](auto gated, auto split) {
                    constexpr bool ACT = decltype(gated)::value, SPLIT = decltype(split)::value;
                    // partial sums: [K split][token][features], behind gate and up [gate features | up features]
                    const int64_t stride = ACT && SPLIT ? 2 * N : N;
                    float* const out = SPLIT ? A.part + ((int64_t)U.ks * A.M + U.m0) * stride + (ACT ? half * N : 0) + n : (float*)A.y + (int64_t)U.m0 * N + n;
#pragma unroll 1
                    for (int c = 0; c < rows; c += 32) {
                        float v[32];
                        tmem_ld32(acc + c, v);
                        if (!valid) continue;
                        float* p = out + c * stride;
                        if (ACT && !SPLIT) {
#pragma unroll
                            for (int h = 0; h < 2; h++) {
                                float x[16], o[8];
#pragma unroll
                                for (int j = 0; j < 16; j++) x[j] = v[16 * h + j];
                                gate_up(x, A.act, half, o);
#pragma unroll
                                for (int i = 0; i < 8; i++)
                                    if (c + 16 * h + 2 * i + half < rows) p[(16 * h + 2 * i + half) * N] = o[i];
                            }
                        } else if (!SPLIT && A.accumulate) {
#pragma unroll
                            for (int j = 0; j < 32; j++, p += stride) if (c + j < rows) *p += v[j] + b;
                        } else if (c + 32 <= rows) {
#pragma unroll
                            for (int j = 0; j < 32; j++, p += stride) *p = SPLIT ? v[j] : v[j] + b;
                        } else {
#pragma unroll
                            for (int j = 0; j < 32; j++, p += stride) if (c + j < rows) *p = SPLIT ? v[j] : v[j] + b;
                        }
                    }
                };
                const std::true_type yes;
                const std::false_type no;
                if (GRAD || !A.act) { if (A.ksplit > 1) unit_out(no, yes); else unit_out(no, no); }
                else if (A.ksplit > 1) unit_out(yes, yes);
                else unit_out(yes, no);
            } else {
                // 16-bit results: 32 tokens at a time through shared memory, so that a token's 128 (64 behind the activation) features
                // leave as one run of 16-byte stores.  The accumulators are read in the fragment shape (a thread: two tokens of features
                // g and g + 8 of 16), so that pairs of tokens are 8 x 8 matrices that stmatrix turns on their way, and gate and up of one
                // feature are registers of one thread.  When every lane stored its feature's 32 tokens in 2 bytes each, with the kinds of results
                // as conditions inside the loop (both sides computed for every value), 32 tokens took 1500 clocks beside the main loop and
                // behind it (400 so), 32-bit results of a unit of 256 tokens 12 us (3.5 so), which nothing hides behind a cluster's last
                // unit.  Recorded, short chains: 512 rows, 4096 x 11008, bf16 (K in two splits) 49.1 -> 40.6 us, fp16 44.8 -> 42.6, an MLP of 1000
                // rows, 4096 / 14336, bf16 323 -> 271, of 4000 rows 1198 -> 1099 (fewer clocks a k-block, too: 531 -> 478 beside an epilogue);
                // a stream of calls under the power cap: the MLP of 4000 rows 1263 -> 1171, 512 rows in fp16 52.7 -> 51.2.
                const bool f16 = A.y_dtype == DT_F16, y_vec = (reinterpret_cast<uintptr_t>(A.y) & 15) == 0;
                auto put = [&](uint16_t* dst, const uint4& q) {
                    if (y_vec) { *reinterpret_cast<uint4*>(dst) = q; return; }
                    const uint32_t w[4] = {q.x, q.y, q.z, q.w};          // a result that does not start on 16 bytes
#pragma unroll
                    for (int i = 0; i < 8; i++) dst[i] = (uint16_t)(w[i >> 1] >> (16 * (i & 1)));
                };
                uint16_t* const yb = (uint16_t*)A.y + (int64_t)U.m0 * N + f0;
                // 16 TMEM lanes are 16 features: which ones of the tile's
                const int first[2] = {GRAD ? 32 * quarter : 16 * quarter, GRAD ? 32 * quarter + 16 : 64 + 16 * quarter};
                // the lane's row address in four matrices: tokens 8 (lane / 16) + lane % 8 of 16, eight features of 16
                const int tok = 8 * (lane >> 4) + (lane & 7), fh8 = (lane >> 3) & 1;
                // type and activation known to the compiler: as conditions inside, both sides of them were computed for every value
                auto unit_out = [&](auto half_type, auto gated) {
                    constexpr bool F16 = decltype(half_type)::value, ACT = decltype(gated)::value;
                    constexpr int LINE = ACT ? 128 : 256, LG = ACT ? 3 : 4;                  // bytes of a token's features, its 16-byte pieces
                    auto pack = [](float x, float y) { return pack2<!F16>(x, y); };
                    float bias[2][2] = {};                            // [16 lanes][g, g + 8]
                    if (!ACT && A.bias && valid) {
#pragma unroll
                        for (int hh = 0; hh < 2; hh++)
#pragma unroll
                            for (int fh = 0; fh < 2; fh++) {
                                const int64_t f = f0 + first[hh] + 8 * fh + (lane >> 2);
                                bias[hh][fh] = F16 ? __half2float(((const __half*)A.bias)[f]) : __bfloat162float(((const __nv_bfloat16*)A.bias)[f]);
                            }
                    }
#pragma unroll 1
                    for (int c = 0; c < rows; c += 32, chunk ^= 1u) {
                        const uint32_t ob = obuf + chunk * 8192;
                        float v[2][16];
                        tmem_ld_frag32(acc + c, v[0]);
                        tmem_ld_frag32(acc + ((uint32_t)16 << 16) + c, v[1]);
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                        if (!ACT && A.accumulate && valid) {
#pragma unroll
                            for (int hh = 0; hh < 2; hh++)
#pragma unroll
                                for (int i = 0; i < 16; i++) {
                                    const int t = c + 8 * (i >> 2) + 2 * (lane & 3) + (i & 1);
                                    const uint16_t* yp = yb + (int64_t)t * N + first[hh] + 8 * ((i >> 1) & 1) + (lane >> 2);
                                    if (t < rows) v[hh][i] += F16 ? __half2float(__ushort_as_half(*yp)) : __bfloat162float(__ushort_as_bfloat16(*yp));
                                }
                        }
#pragma unroll
                        for (int hh = 0; hh < (ACT ? 1 : 2); hh++)
#pragma unroll
                            for (int p = 0; p < 2; p++) {             // 16 tokens
                                uint32_t m[4];
#pragma unroll
                                for (int j = 0; j < 4; j++) {         // tokens 8 (j / 2) of them, features 8 (j % 2) of 16
                                    const int i = 8 * p + 4 * (j >> 1) + 2 * (j & 1);
                                    m[j] = ACT ? pack(apply_act(v[0][i], A.act) * v[1][i], apply_act(v[0][i + 1], A.act) * v[1][i + 1])
                                               : pack(v[hh][i] + bias[hh][j & 1], v[hh][i + 1] + bias[hh][j & 1]);
                                }
                                const int r = 16 * p + tok, piece = (first[hh] >> 3) + fh8;
                                stmatrix4_trans(ob + (uint32_t)(r * LINE + ((piece ^ (r & 7)) << 4)), m);
                            }
                        asm volatile("barrier.cta.sync 1, 128;" ::: "memory");
                        // the other buffer is written next: everybody passes the next barrier only after this copy
                        const int n_rows = min(32, rows - c);
                        const int r0 = e_tid >> LG, p = e_tid & ((1 << LG) - 1);             // piece p: 8 features from 8 p
                        uint16_t* const to = yb + (int64_t)(c + r0) * N + p * 8;
                        constexpr int STEP = 128 >> LG;                                      // rows between a thread's pieces: 8 or 16
                        const uint32_t from = ob + (uint32_t)(r0 * LINE + ((p ^ (r0 & 7)) << 4));
                        if (valid && n_rows == 32 && y_vec) {
                            uint4 q[32 / STEP];
#pragma unroll
                            for (int i = 0; i < 32 / STEP; i++) q[i] = lds128(from + i * STEP * LINE);
#pragma unroll
                            for (int i = 0; i < 32 / STEP; i++) *reinterpret_cast<uint4*>(to + (int64_t)i * STEP * N) = q[i];
                        } else if (valid) {
                            for (int i = 0; r0 + i * STEP < n_rows; i++) put(to + (int64_t)i * STEP * N, lds128(from + i * STEP * LINE));
                        }
                    }
                };
                const std::true_type yes;
                const std::false_type no;
                if (GRAD || !A.act) { if (f16) unit_out(yes, no); else unit_out(no, no); }
                else if (f16) unit_out(yes, yes);
                else unit_out(no, yes);
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive_at(tmem_empty(buf), 0);
        }
    }
done:
    __syncwarp();
    // behind a wait that ran out copies and MMAs may still be under way: nobody leaves their memory
    if (warp == 0) drain_ring(round * KX + s, KX, x_full, A.waits);
    if (warp == 2) drain_ring(round * KP + s, KP, p_full, A.waits);
    if (warp == 1) {
        if (rank == 0) umma2_commit_w(drained, leader);    // arrives in both CTAs
        mbar_wait_lim(drained, 0u, Waits{A.waits.word, kWaitCycles});
    }
    __syncthreads();
    cluster_sync_all();                                    // nobody signals a CTA that has left, no MMA reads its memory
    if (warp == 3) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

// the same behind a split MLP: y[token][n] = act(sum of the gate partials) * (sum of the up partials)
__global__ void __launch_bounds__(256) reduce_gated_kernel(const float* part, int ksplit, int64_t m, int64_t n, void* y, int y_dtype, int act) {
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int64_t mn = m * n, n4 = n / 4;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < mn / 4; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t token = i / n4, col = (i - token * n4) * 4;
        const float* p = part + token * 2 * n + col;
        float4 g = make_float4(0.0f, 0.0f, 0.0f, 0.0f), u = g;
        for (int ks = 0; ks < ksplit; ks++, p += 2 * mn) {
            const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + n);
            g.x += a.x; g.y += a.y; g.z += a.z; g.w += a.w;
            u.x += b.x; u.y += b.y; u.z += b.z; u.w += b.w;
        }
        const float r[4] = {apply_act(g.x, act) * u.x, apply_act(g.y, act) * u.y, apply_act(g.z, act) * u.z, apply_act(g.w, act) * u.w};
#pragma unroll
        for (int j = 0; j < 4; j++) store_out(y, y_dtype, token * n + col + j, r[j], nullptr, 0, 0);
    }
}

// clusters of two that can be resident at once (one CTA per SM; an SM without a partner in its group stays idle)
template <int QT, bool BF, bool GRAD>
static int pair_clusters() {
    static int cached[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    int& n = cached[dev & 63];
    if (n) return n;
    constexpr int SMEM = PairSmem<QT>::kTotal;
    if (cudaFuncSetAttribute(pair_kernel<QT, BF, GRAD>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) != cudaSuccess) { cudaGetLastError(); return 0; }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(sm_count() & ~1)); cfg.blockDim = dim3(kPairThreads); cfg.dynamicSmemBytes = SMEM;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    int c = 0;
    if (cudaOccupancyMaxActiveClusters(&c, pair_kernel<QT, BF, GRAD>, &cfg) != cudaSuccess || c <= 0) { cudaGetLastError(); c = sm_count() / 2; }
    n = c;
    return n;
}

template <int QT, bool BF, bool GRAD>
static int pair_launch_one(const CUtensorMap& map, const PairArgs& A, int64_t units, cudaStream_t st) {
    const int clusters = pair_clusters<QT, BF, GRAD>();
    if (clusters <= 0) { set_error(LB_ERR_CUDA, "the two-SM matmul kernel cannot be configured on this device"); return LB_ERR_CUDA; }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2u * (unsigned)(units < clusters ? units : clusters)); cfg.blockDim = dim3(kPairThreads);
    cfg.dynamicSmemBytes = PairSmem<QT>::kTotal; cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = add_overlap(at, 1, launch_overlaps(st));
    cudaLaunchKernelEx(&cfg, pair_kernel<QT, BF, GRAD>, map, A);
    note_launch();
    return LB_OK;
}
template <bool GRAD = false>
static int pair_launch(int qt, bool bf, const CUtensorMap& map, const PairArgs& A, int64_t units, cudaStream_t st) {
#define PAIR_CASE(Q) case Q: return bf ? pair_launch_one<Q, true, GRAD>(map, A, units, st) : pair_launch_one<Q, false, GRAD>(map, A, units, st);
    switch (qt) { PAIR_CASE(QT_SYM_INT4) PAIR_CASE(QT_ASYM_INT4) PAIR_CASE(QT_NF4) PAIR_CASE(QT_FP8_E4M3) PAIR_CASE(QT_FP8_E5M2) PAIR_CASE(QT_FP6) }
#undef PAIR_CASE
    return LB_ERR_ARG;
}

// Token tile and K splits of a matmul, each the one that minimises rounds of the resident clusters x (k-blocks per unit x time per k-block
// + the start and end of a unit) and, when K is split, the partial sums' round trip through memory and the second launch.  A k-block takes
// a time per token once the MMAs set the pace, below that the expansion and the chain around it; sym_int4 with fp16 activations, with
// bf16, and nf4's table were measured, the other formats take sym_int4's figures.
//
// The tile changes no bit of a result.  It goes by the times under the power cap (1.6 to 1.75 GHz): 4000 rows, 4096 x 14336, with the tile
// of the split's figures / with this one: fp8_e5m2 fp16 424 (176 tokens) / 369 us (224), fp8_e4m3 412 / 386, nf4 bf16 410 (256) / 378
// (224), sym_int4 fp16 323 / 329.
//
// The split is the order of a result's 32-bit sums.  It goes by a cool GPU's times (4096 x 11008 and 4096 x 4096; partial sums at ~4 TB/s).
// Both sides of its line under the power cap, 128-token tiles of the whole K against 256-token tiles of two splits, 4096 x 11008: 512 rows
// sym_int4 fp16 48.5 / 48.1 us, bf16 52.1 / 41.7, nf4 64.1 / 42.8, 500 rows fp16 49.4 / 41.0.  Over 332 shapes and formats (65 to 1500
// rows, 1024 to 11008 features, K 2048 to 14336) the choices lie 1.6 % over the best tile and split, 12 of them more than 10 %, most of
// these because partial sums that stay in L2 cost less than is charged here (a fit over all times: 27 TB/s and 3.5 us).  Charging less moves
// which prompts are split: with the tile's figures and 4.5 TB/s the choices were 1.1 % over the best, and the logits of a decode step behind
// some prompts moved by 7e-3 (the e5m2 cache takes a low bit a long way).  0.5 % do not pay for other results.
struct PairTimes { double token, pace[3], unit, unit_token; };       // us: a k-block per token, at least (fp16, bf16, nf4); a unit, per token
constexpr PairTimes kSplitTimes = {0.0011, {0.19, 0.24, 0.29}, 1.0, 0.0}, kTileTimes = {0.0012, {0.215, 0.275, 0.35}, 1.2, 0.006};
static int pair_kind(int qt, bool bf) { return qt == QT_NF4 ? 2 : bf ? 1 : 0; }
struct PairPlan { int tt, ks; };
static PairPlan pair_plan(int kind, int64_t n_fp, int64_t nb, int64_t m, int64_t n_out, bool may_split) {
    const int64_t clusters = sm_count() / 2, nt0 = (m + kPairTok - 1) / kPairTok;
    auto best_of = [&](const PairTimes& T, int64_t ks0, int64_t ks1) {
        PairPlan best = {256, (int)ks0};
        double best_cost = 1e30;
        for (int64_t nt = nt0; nt <= nt0 + 8 && nt <= (m + 31) / 32; nt++) {
            const int64_t tt = ((m + nt - 1) / nt + 15) & ~int64_t(15);
            const double mma = T.token * (double)tt, per_kb = mma > T.pace[kind] ? mma : T.pace[kind];
            for (int64_t ks = ks0; ks <= ks1; ks++) {
                const int64_t rounds = (n_fp * nt * ks + clusters - 1) / clusters;
                double cost = (double)rounds * ((double)((nb + ks - 1) / ks) * per_kb + T.unit + T.unit_token * (double)tt);
                if (ks > 1) cost += (double)ks * (double)m * (double)n_out * 8.0 / 4.0e6 + 3.0;
                if (cost < best_cost - 1e-9) { best_cost = cost; best = {(int)tt, (int)ks}; }
            }
        }
        return best;
    };
    const int64_t most = may_split && nb >= 16 ? (nb / 8 < 8 ? nb / 8 : 8) : 1, ks = best_of(kSplitTimes, 1, most).ks;
    return best_of(kTileTimes, ks, ks);
}
static bool holds_partials(const void* workspace, size_t bytes, size_t count) {
    return workspace && ((uintptr_t)workspace & 15) == 0 && bytes >= count * sizeof(float);
}
// splits that a workspace has to hold, whatever the format and type
static int most_splits(int64_t n_fp, int64_t nb, int64_t m, int64_t n_out) {
    int ks = 1;
    for (int kind = 0; kind < 3; kind++) {
        const PairPlan p = pair_plan(kind, n_fp, nb, m, n_out, true);
        if (p.ks > ks) ks = p.ks;
    }
    return ks;
}
}  // namespace gemmtc

bool gemm_tc_supported(int qt, int64_t n_rows, int64_t k) {
    qt = canon_qtype(qt);
    const bool q = qt == QT_SYM_INT4 || qt == QT_ASYM_INT4 || qt == QT_NF4 || qt == QT_FP8_E4M3 || qt == QT_FP8_E5M2 || qt == QT_FP6;
    return q && n_rows >= 128 && (n_rows % 128) == 0 && k >= 64 && (k % 64) == 0;
}

size_t gemm_tc_workspace_size(int64_t n_rows, int64_t k, int64_t m) {
    using namespace gemmtc;
    const int ks = most_splits((n_rows / 128 + 1) / 2, k / 64, m, n_rows);
    return ks > 1 ? (size_t)ks * m * n_rows * sizeof(float) : 0;
}

int gemm_tc_launch(const void* w, int qt, int64_t n_rows, int64_t k, const void* x, int x_dtype, int64_t m, void* y,
                   int y_dtype, const void* bias, int accumulate, void* workspace, size_t workspace_bytes, cudaStream_t st) {
    using namespace gemmtc;
    qt = canon_qtype(qt);
    if (!gemm_tc_supported(qt, n_rows, k) || (x_dtype != DT_F16 && x_dtype != DT_BF16)) return LB_ERR_ARG;
    if (((uintptr_t)x & 15) || ((uintptr_t)w & 15)) return LB_ERR_ARG;
    const bool bf = x_dtype == DT_BF16;
    CUtensorMap map;
    if (const int rc = encode_rows(&map, x, bf, m, k, 32)) return rc;
    PairArgs A = {};
    if (const int rc = make_waits(&A.waits, kWaitCycles)) return rc;
    A.w = (const uint8_t*)w; A.G = make_geom(n_rows, k, qt); A.M = (int)m; A.y = y; A.y_dtype = y_dtype; A.bias = bias; A.accumulate = accumulate;
    A.n_fp = (int)((n_rows / 128 + 1) / 2);
    PairPlan p = pair_plan(pair_kind(qt, bf), A.n_fp, k / 64, m, n_rows, true);
    // a caller's workspace without room for partial sums, or not aligned for their 16-byte loads: the whole K range per unit
    if (p.ks > 1 && !holds_partials(workspace, workspace_bytes, (size_t)p.ks * m * n_rows)) p = pair_plan(pair_kind(qt, bf), A.n_fp, k / 64, m, n_rows, false);
    A.tt = p.tt; A.ksplit = p.ks; A.part = (float*)workspace;
    const int64_t units = (int64_t)A.n_fp * ((m + p.tt - 1) / p.tt) * p.ks;
    if (const int rc = pair_launch<>(qt, bf, map, A, units, st)) return rc;
    if (p.ks > 1) {
        const int64_t mn = m * n_rows;
        int rg = (int)((mn / 4 + 255) / 256); if (rg > sm_count() * 8) rg = sm_count() * 8;
        launch_behind(reduce_partials_kernel, dim3((unsigned)rg), 256, 0, st, launch_overlaps(st), A.part, p.ks, mn, n_rows, y, y_dtype, bias, accumulate);
        note_launch();
    }
    return check_launch();
}

// dx[m][k] = g[m][n_rows] . dequant(W): what a training step takes back through a frozen projection.  Whole 64-row groups (the rows behind
// the last one lie in another layout) and tiles of 128 columns
bool gemm_tc_grad_supported(int qt, int64_t n_rows, int64_t k) { return gemm_tc_supported(qt, 128, k) && n_rows >= 64 && n_rows % 64 == 0 && k % 128 == 0; }
size_t gemm_tc_grad_workspace_size(int64_t n_rows, int64_t k, int64_t m) {
    using namespace gemmtc;
    const int ks = most_splits((k / 128 + 1) / 2, n_rows / 64, m, k);
    return ks > 1 ? (size_t)ks * m * k * sizeof(float) : 0;
}
// Whether it is the better way than dequantising for a library product.  Formats but nf4: always (2000 to 6000 rows, six matrices of 4096 to
// 14336: fp8 0.88 to 1.02 of its time, the 4-bit ones 0.77 to 0.95; fewer rows or smaller matrices: less device time but for matrices under
// 5 M weights, whose 6 to 12 us no pass waits for).  nf4's table sets a pace of 0.38 us a k-block, so there it goes by cost: rounds of the plan's
// units against the matrix's way through memory (0.70 us per million weights) and the product (1590 TFLOP/s), all us, fitted to 542 times
// of 21 matrices, 16 to 4000 rows; this launch / the other way, bf16: 11008 x 4096 at 512 rows 52 / 63, 1024 rows 94 / 92 (taken), 1280
// rows 159 / 117 (not); 8192 x 8192 at 1024 rows 116 / 133 (taken), 3000 rows 393 / 332 (not); 2048 x 8192 at 2000 rows 70 / 60 (not);
// 4096 x 11008 at 1280 rows 93 / 101 (taken).  Over all of them 0.925 of the other way's time, the better of the two each time 0.916.  Below
// 40 us the pass waits for the host, which one call holds up less than two: forward and backward of 1024 rows, 4096 x 4096, 110 / 120 us
// though the GPU takes 38 / 34.
bool gemm_tc_grad_faster(int qt, int64_t n_rows, int64_t k, int64_t m) {
    using namespace gemmtc;
    if (canon_qtype(qt) != QT_NF4) return true;
    const int64_t n_fp = (k / 128 + 1) / 2, nb = n_rows / 64, clusters = sm_count() / 2;
    const PairPlan p = pair_plan(pair_kind(QT_NF4, false), n_fp, nb, m, k, true);
    const int64_t rounds = (n_fp * ((m + p.tt - 1) / p.tt) * p.ks + clusters - 1) / clusters;
    const double per_kb = 0.0019 * p.tt > 0.38 ? 0.0019 * p.tt : 0.38;
    const double here = (double)rounds * ((double)((nb + p.ks - 1) / p.ks) * per_kb + 1.5) + 8.0 + (p.ks > 1 ? 2.7 : 0.0);
    const double there = 5.5 + (double)n_rows * (double)k * (0.70e-6 + 2.0 * (double)m / 1590e6);
    return here < there || there < 40.0;
}
int gemm_tc_grad_launch(const void* w, int qt, int64_t n_rows, int64_t k, const void* g, int dtype, int64_t m, void* dx, void* workspace,
                        size_t workspace_bytes, cudaStream_t st) {
    using namespace gemmtc;
    qt = canon_qtype(qt);
    if (!gemm_tc_grad_supported(qt, n_rows, k) || (dtype != DT_F16 && dtype != DT_BF16) || (((uintptr_t)g | (uintptr_t)w) & 15)) return LB_ERR_ARG;
    const bool bf = dtype == DT_BF16;
    CUtensorMap map;
    if (const int rc = encode_rows(&map, g, bf, m, n_rows, 32)) return rc;
    PairArgs A = {};
    if (const int rc = make_waits(&A.waits, kWaitCycles)) return rc;
    A.w = (const uint8_t*)w; A.G = make_geom(n_rows, k, qt); A.M = (int)m; A.y = dx; A.y_dtype = dtype;
    A.n_fp = (int)((k / 128 + 1) / 2);
    PairPlan p = pair_plan(pair_kind(qt, bf), A.n_fp, n_rows / 64, m, k, true);
    if (p.ks > 1 && !holds_partials(workspace, workspace_bytes, (size_t)p.ks * m * k)) p = pair_plan(pair_kind(qt, bf), A.n_fp, n_rows / 64, m, k, false);
    A.tt = p.tt; A.ksplit = p.ks; A.part = (float*)workspace;
    if (const int rc = pair_launch<true>(qt, bf, map, A, (int64_t)A.n_fp * ((m + p.tt - 1) / p.tt) * p.ks, st)) return rc;
    if (p.ks > 1) {
        int rg = (int)((m * k / 4 + 255) / 256); if (rg > sm_count() * 8) rg = sm_count() * 8;
        launch_behind(reduce_partials_kernel, dim3((unsigned)rg), 256, 0, st, launch_overlaps(st), A.part, p.ks, m * k, k, dx, dtype, nullptr, 0);
        note_launch();
    }
    return check_launch();
}

// first half of an MLP at prompt sizes: y = act(x . Wgate^T) * (x . Wup^T), both products in one tile's accumulators (a gate and an
// up row group per CTA), the activation in the epilogue: the two [M][N] intermediates and their kernel do not exist
int gemm_tc_mlp_launch(const void* w_gate, const void* w_up, int act, int qt, int64_t n_rows, int64_t k, const void* x, int x_dtype,
                       int64_t m, void* y, int y_dtype, void* workspace, size_t workspace_bytes, cudaStream_t st) {
    using namespace gemmtc;
    qt = canon_qtype(qt);
    if (!gemm_tc_supported(qt, n_rows, k) || (x_dtype != DT_F16 && x_dtype != DT_BF16) || act < 1 || act > 2) return LB_ERR_ARG;
    if (((uintptr_t)x & 15) || ((uintptr_t)w_gate & 15) || ((uintptr_t)w_up & 15)) return LB_ERR_ARG;
    const bool bf = x_dtype == DT_BF16;
    CUtensorMap map;
    if (const int rc = encode_rows(&map, x, bf, m, k, 32)) return rc;
    PairArgs A = {};
    if (const int rc = make_waits(&A.waits, kWaitCycles)) return rc;
    A.w = (const uint8_t*)w_gate; A.w2 = (const uint8_t*)w_up; A.act = act; A.G = make_geom(n_rows, k, qt); A.M = (int)m; A.y = y; A.y_dtype = y_dtype;
    A.n_fp = (int)((n_rows / 64 + 1) / 2);
    PairPlan p = pair_plan(pair_kind(qt, bf), A.n_fp, k / 64, m, 2 * n_rows, true);
    if (p.ks > 1 && !holds_partials(workspace, workspace_bytes, (size_t)p.ks * m * 2 * n_rows)) p = pair_plan(pair_kind(qt, bf), A.n_fp, k / 64, m, 2 * n_rows, false);
    A.tt = p.tt; A.ksplit = p.ks; A.part = (float*)workspace;
    if (const int rc = pair_launch<>(qt, bf, map, A, (int64_t)A.n_fp * ((m + A.tt - 1) / A.tt) * p.ks, st)) return rc;
    if (p.ks > 1) {
        int rg = (int)((m * n_rows / 4 + 255) / 256); if (rg > sm_count() * 8) rg = sm_count() * 8;
        launch_behind(reduce_gated_kernel, dim3((unsigned)rg), 256, 0, st, launch_overlaps(st), A.part, p.ks, m, n_rows, y, y_dtype, act);
        note_launch();
    }
    return check_launch();
}
size_t gemm_tc_mlp_workspace_size(int64_t n_rows, int64_t k, int64_t m) {
    using namespace gemmtc;
    const int ks = most_splits((n_rows / 64 + 1) / 2, k / 64, m, 2 * n_rows);
    return ks > 1 ? (size_t)ks * m * 2 * n_rows * sizeof(float) : 256;
}

// the same kernel over every expert's rows: x [rows][k] sorted by expert, offs [n_experts + 1] row offsets on the device, tab /
// tab2 device addresses of the experts' weights (tab2: the up projections, act in the epilogue; or NULL).  Experts of at most
// kExactRows rows are left out
int gemm_tc_experts_launch(const unsigned long long* tab, const unsigned long long* tab2, int act, const int* offs, int n_experts, int qt,
                           int64_t n_rows, int64_t k, const void* x, int x_dtype, int64_t rows, void* y, int y_dtype, cudaStream_t st) {
    using namespace gemmtc;
    qt = canon_qtype(qt);
    if (!gemm_tc_supported(qt, n_rows, k) || (x_dtype != DT_F16 && x_dtype != DT_BF16) || n_experts > kMaxExperts || ((uintptr_t)x & 15)) return LB_ERR_ARG;
    const bool bf = x_dtype == DT_BF16;
    CUtensorMap map;
    if (const int rc = encode_rows(&map, x, bf, rows, k, 32)) return rc;
    PairArgs A = {};
    if (const int rc = make_waits(&A.waits, kWaitCycles)) return rc;
    A.tab = tab; A.tab2 = tab2; A.act = tab2 ? act : 0; A.offs = offs; A.n_experts = n_experts;
    A.G = make_geom(n_rows, k, qt); A.M = (int)rows; A.y = y; A.y_dtype = y_dtype; A.ksplit = 1; A.tt = kPairTok;
    A.n_fp = (int)((n_rows / (tab2 ? 64 : 128) + 1) / 2);
    const int64_t most = (rows < n_experts ? rows : n_experts) + rows / kPairTok;        // tiles: one per used expert and one per 256 rows
    if (const int rc = pair_launch<>(qt, bf, map, A, most * A.n_fp, st)) return rc;
    return check_launch();
}

}  // namespace lowbit
