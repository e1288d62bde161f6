// gemm_tc.cu -- kernel (c'): dequant-GEMM of small batches on the 5th-generation tensor cores (17 <= M <= 64 activation rows:
// batched decode, short prefills).  The EXPANDED WEIGHTS are the 128-row A operand and the tokens are the N dimension
// (32 / 48 / 64), so nothing is padded to a 128-token tile, an activation stage is NTOK x 256 bytes and the accumulator is NTOK TMEM columns.
//   * work = the linear sequence of (128-feature tile, PAIR of k-blocks) items, cut into gridDim.x contiguous ranges of
//     equal length (stream-K): every SM expands the same number of blocks whatever the matrix shape; a range that crosses
//     a tile boundary produces one partial result per tile it touches (fp32, in the workspace) and a second,
//     programmatic-dependent launch adds a tile's partials in CTA order (deterministic) and applies bias / accumulate;
//   * an item is 128 k: the barrier handshakes, the MMA thread's loop and the bulk copies are per item;
//   * warp 0 streams PACKED weights through a ring of stages (in a recorded step, where they are complete, in front of
//     griddepcontrol.wait); a stage is free again when its codes have been expanded.  A warp of its own brings the activations' k-slices
//     through a ring of two to four;
//   * 16 dequant warps in two groups take alternate items; a group fills 128 x 128 K-major 128B-swizzled A tiles (two 16 KB atoms each),
//     two in turn, and every warp expands its 16 rows of both k-blocks: a group goes on while the MMAs of its last tile run, and its
//     waits, LDS / STS latency and proxy fence overlap the other group's arithmetic;
//   * warp 1 issues tcgen05.mma M = 128, N = NTOK, K = 16 (8 per item) into one of two TMEM accumulators; ONE commit per
//     item frees both the activations (for their warp) and the A tile;  4 epilogue warps read TMEM (lane = feature,
//     column = token).
// Bound by shared memory: an item of 64 tokens moves 32 KB of expanded weights in and out, 16 KB of activations twice and 9 KB of codes
// twice, about 850 of its 128-byte wavefronts, 0.45 us; 8.6 us of 12.2 are there without expansion and MMAs.  40 rows, 11008 x 4096,
// asym_int4: kernel 13.8 -> 12.2 us (one tile per group, activations and weights in one ring before), its reduction 5.4 -> 4.0 (below);
// 60 rows, 4096 x 14336, fp8_e4m3: 19.9 + 7.8 -> 18.9 + 5.0.
#include "tc_common.cuh"

namespace lowbit {
namespace gemmtc {

constexpr int kSkStagesMax = 12;
constexpr int kSkDeqWarps = 16;
constexpr int kSkThreads = 64 + 32 * kSkDeqWarps + 128 + 32;

#ifdef LOWBIT_SK_TIMESTAMPS
__device__ unsigned long long g_sk_ts[6][64];
#define SKTS(row, it) do { if (blockIdx.x == 0 && lane == 0 && (it) < 64) { unsigned long long t_; asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_)); g_sk_ts[row][it] = t_; } } while (0)
#else
#define SKTS(row, it) do { } while (0)
#endif

struct SkinnyArgs {
    const uint8_t* w;
    const uint8_t* w2;       // fused MLP: a second matrix of the same shape; its feature tiles follow w's in the item sequence
    TiledGeom G;
    int M;
    float* part;             // [gridDim.x * max_seg][NTOK][128] fp32 partial tiles
    int max_seg;
    int pdl;                 // launched as a programmatic dependent: 1 in a recorded step (the weights are complete), 2 outside one
};

template <int QT, int NTOK> struct SkSmem {
    static constexpr int kSuper = PackedBlock<QT>::kSuper;
    static constexpr int kAux = Expand<QT>::kHasMin ? 512 : 256;                // scales (+ minima) of the two k-blocks
    static constexpr int kGroup = 2 * kSuper + kAux;                            // one 64-row group, two k-blocks
    static constexpr int kX = NTOK * 256;                                       // two [NTOK][64] atoms
    static constexpr int kW = (2 * kGroup + 127) / 128 * 128;
    static constexpr int kTiles = 4;                                            // expanded tiles, two atoms each: two per group
    static constexpr int kFree = 232448 - 1024 - 512 - kTiles * 2 * kTileBytesAB - Expand<QT>::kLutBytes;
    static constexpr int kXStages = NTOK <= 32 ? 4 : kFree - 3 * kX >= 3 * kW ? 3 : 2;
    static constexpr int kFit = (kFree - kXStages * kX) / kW;
    static constexpr int kStages = kFit < kSkStagesMax ? kFit : kSkStagesMax;   // of packed weights
    static constexpr int kTotal = 1024 + 512 + kTiles * 2 * kTileBytesAB + kXStages * kX + kStages * kW + Expand<QT>::kLutBytes;
};

template <int N> __device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, float (&v)[N]);
template <> __device__ __forceinline__ void tmem_ld_cols<32>(uint32_t taddr, float (&v)[32]) { tmem_ld32(taddr, v); }
template <> __device__ __forceinline__ void tmem_ld_cols<16>(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

template <int QT, bool BF, int NTOK>
__global__ void __launch_bounds__(kSkThreads, 1)
skinny_kernel(const __grid_constant__ CUtensorMap xmap, const SkinnyArgs A) {
    using E = Expand<QT>;
    using SM = SkSmem<QT, NTOK>;
    constexpr int NS = SM::kStages, NX = SM::kXStages, NA = SM::kTiles;
    // A group waits for its own items only, and a barrier tells apart two rounds: with an odd ring of stages the rounds of a stage alternate
    // between the groups, so the barriers go round at twice its length
    constexpr int NF = (NS & 1) ? 2 * NS : NS;
    // an activation stage is waited for by the tile of the item NX before: not more stages than tiles, else that tile's barrier may be two
    // rounds on; and a group's tiles are every second one
    static_assert(NS >= 2 && NX >= 2 && NX <= 4 && NX <= NA && NA % 2 == 0, "ring depth");
    constexpr uint32_t ACC_COLS = NTOK, TMEM_COLS = NTOK <= 32 ? 64 : 128;   // a power of two
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t atiles = base, xring = atiles + NA * 2 * kTileBytesAB, ring = xring + NX * SM::kX, bars = ring + NS * SM::kW;
    auto full_bar = [&](int i) { return bars + i * 8; };                          // weights have come (NF)
    auto free_bar = [&](int s) { return bars + (2 * kSkStagesMax + s) * 8; };     // they have been expanded
    auto xfull_bar = [&](int s) { return bars + (3 * kSkStagesMax + s) * 8; };
    auto afull_bar = [&](int t) { return bars + (3 * kSkStagesMax + 4 + t) * 8; };
    auto done_bar = [&](int t) { return bars + (3 * kSkStagesMax + 8 + t) * 8; }; // the MMAs that read tile t (and its item's activations)
    auto tmem_full = [&](int b) { return bars + (3 * kSkStagesMax + 12 + b) * 8; };
    auto tmem_empty = [&](int b) { return bars + (3 * kSkStagesMax + 14 + b) * 8; };
    const uint32_t tmem_slot = bars + (3 * kSkStagesMax + 16) * 8;

    // the warp index through a shuffle: the compiler then treats everything derived from it as warp-uniform
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const uint32_t lut = bars + 512 + 4 * lane;
    if constexpr (E::kLutBytes > 0) E::fill_lut(smem_raw + (bars + 512 - smem_u32(smem_raw)), threadIdx.x, kSkThreads);
    const int nb = (int)A.G.nb, np = nb >> 1;                // k-blocks / pairs of k-blocks per tile (nb is even)
    const int n_ft1 = (int)(A.G.rows / kTileN);                    // feature tiles of one matrix
    const int64_t total = (int64_t)(A.w2 ? 2 * n_ft1 : n_ft1) * np;
    const int64_t i_begin = (int64_t)blockIdx.x * total / gridDim.x, i_end = (int64_t)(blockIdx.x + 1) * total / gridDim.x;
    const int n_items = (int)(i_end - i_begin);
    const int ft0 = (int)(i_begin / np), p_first = (int)(i_begin - (int64_t)ft0 * np);

    if (threadIdx.x == 0) {
        for (int i = 0; i < NF; i++) mbar_init(full_bar(i), 1);
        for (int s = 0; s < NS; s++) mbar_init(free_bar(s), kSkDeqWarps / 2);
        for (int s = 0; s < NX; s++) mbar_init(xfull_bar(s), 1);
        for (int t = 0; t < NA; t++) { mbar_init(afull_bar(t), 32 * (kSkDeqWarps / 2)); mbar_init(done_bar(t), 1); }
        for (int b = 0; b < 2; b++) { mbar_init(tmem_full(b), 1); mbar_init(tmem_empty(b), 128); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    uint32_t tmem_base;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem_base) : "r"(tmem_slot));

    auto locate = [&](int it, int& ft, int& kb) {
        int p = p_first + it;
        ft = ft0;
        while (p >= np) { p -= np; ft++; }
        kb = 2 * p;
    };
    if (warp == 0) {
        // ================= packed weights: the whole warp runs the loop, one elected lane issues the copies.  The first round does not
        // depend on the previous kernel and is not held up by it
        const uint32_t leader = elect_leader();
        if (A.pdl == 2) asm volatile("griddepcontrol.wait;" ::: "memory");
        for (int it = 0; it < n_items; it++) {
            const int s = it % NS;
            if (it >= NS) mbar_wait(free_bar(s), (uint32_t)((it / NS - 1) & 1));
            SKTS(0, it);
            int ft, kb;
            locate(it, ft, kb);
            const uint32_t bar = full_bar(it % NF);
            mbar_expect_tx_w(bar, 2 * SM::kGroup, leader);
#pragma unroll
            for (int gi = 0; gi < 2; gi++) {
                const uint8_t* wb = ft < n_ft1 ? A.w : A.w2;
                const int64_t u = ((int64_t)(ft < n_ft1 ? ft : ft - n_ft1) * 2 + gi) * nb + kb;   // units kb and kb + 1 are adjacent in memory
                const uint32_t dst = ring + s * SM::kW + gi * SM::kGroup;
                bulk_g2s_w(dst, wb + u * SM::kSuper, 2 * SM::kSuper, bar, leader);
                bulk_g2s_w(dst + 2 * SM::kSuper, wb + A.G.off_s + u * 128, 256, bar, leader);
                if (E::kHasMin) bulk_g2s_w(dst + 2 * SM::kSuper + 256, wb + A.G.off_m + u * 128, 256, bar, leader);
            }
        }
    } else if (warp == 2 + kSkDeqWarps + 4) {
        // ================= the k-slices of the activations: 2 x [NTOK tokens] x [64]
        const uint32_t leader = elect_leader();
        if (A.pdl) asm volatile("griddepcontrol.wait;" ::: "memory");
        for (int it = 0; it < n_items; it++) {
            const int s = it % NX, j = it - NX;
            if (j >= 0) mbar_wait(done_bar(j % NA), (uint32_t)((j / NA) & 1));
            int ft, kb;
            locate(it, ft, kb);
            mbar_expect_tx_w(xfull_bar(s), SM::kX, leader);
            tma_load_2d_w(xring + s * SM::kX, &xmap, kb * 64, 0, xfull_bar(s), leader);
            tma_load_2d_w(xring + s * SM::kX + NTOK * 128, &xmap, kb * 64 + 64, 0, xfull_bar(s), leader);
        }
    } else if (warp == 1) {
        // ================= MMA issuer: the whole warp runs the loop, one elected lane issues =================
        {
            const uint32_t leader = elect_leader();
            // c F32 (1<<4), a/b format (0 f16, 1 bf16), both K-major, N = NTOK (>>3 at bit 17), M = 128 (>>4 at bit 24)
            const uint32_t idesc = (1u << 4) | ((BF ? 1u : 0u) << 7) | ((BF ? 1u : 0u) << 10) | (((uint32_t)NTOK >> 3) << 17) | ((128u >> 4) << 24);
            int p = p_first, seg = 0;
            bool fresh = true;
            if (n_items > 0) {
                mbar_wait(tmem_empty(0), 1u);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            }
            for (int it = 0; it < n_items; it++) {
                const int s = it % NX, t = it % NA;
                mbar_wait(xfull_bar(s), (uint32_t)((it / NX) & 1));
                mbar_wait(afull_bar(t), (uint32_t)((it / NA) & 1));
                SKTS(1, it);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t acc = tmem_base + (uint32_t)(seg & 1) * ACC_COLS;
                const uint64_t ad = make_desc(atiles + t * (2 * kTileBytesAB)), xd = make_desc(xring + s * SM::kX);
#pragma unroll
                for (int kk = 0; kk < 2; kk++)
#pragma unroll
                    for (int k4 = 0; k4 < 4; k4++)           // the address field counts 16-byte units
                        umma_f16_w(acc, ad + (uint64_t)((kk * kTileBytesAB + k4 * 32) >> 4), xd + (uint64_t)((kk * NTOK * 128 + k4 * 32) >> 4),
                                   idesc, (!fresh || kk > 0 || k4 > 0) ? 1u : 0u, leader);
                fresh = false;
                umma_commit_w(done_bar(t), leader);          // frees the tile (dequant warps) and the activations
                SKTS(2, it);
                if (++p == np || it + 1 == n_items) {        // the tile (or this CTA's part of it) is complete
                    umma_commit_w(tmem_full(seg & 1), leader);
                    p = 0; seg++; fresh = true;
                    if (it + 1 < n_items) {
                        mbar_wait(tmem_empty(seg & 1), (uint32_t)(((seg >> 1) & 1) ^ 1));
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    }
                }
            }
        }
    } else if (warp < 2 + kSkDeqWarps) {
        // ================= dequant warps: group q = (warp - 2) / 8 takes the items of its parity, its tiles in turn =================
        const int q = (warp - 2) >> 3, w8 = (warp - 2) & 7;
        const int dw = w8 & 3, gi = w8 >> 2;                 // tile r = dw of row group gi, both k-blocks
        const int g = lane >> 2, t = lane & 3;
        const int f_lo = 64 * gi + 16 * dw + g;
        const uint32_t row0 = atiles + (f_lo >> 3) * 1024 + (f_lo & 7) * 128;
        for (int it = q; it < n_items; it += 2) {
            const int s = it % NS;
            mbar_wait(full_bar(it % NF), (uint32_t)((it / NF) & 1));
            const uint32_t grp = ring + s * SM::kW + gi * SM::kGroup;
            uint32_t dq[2], mq[2] = {0u, 0u};
            typename E::Codes cw[2];
#pragma unroll
            for (int kk = 0; kk < 2; kk++) {
                asm volatile("ld.shared.u32 %0, [%1];" : "=r"(dq[kk]) : "r"(grp + 2 * SM::kSuper + kk * 128 + g * 16 + dw * 4));
                if (E::kHasMin) asm volatile("ld.shared.u32 %0, [%1];" : "=r"(mq[kk]) : "r"(grp + 2 * SM::kSuper + 256 + kk * 128 + g * 16 + dw * 4));
                E::load(grp + kk * SM::kSuper + dw * E::kTileBytes, lane, cw[kk]);
            }
            const int tile = it % NA;
            if (it >= NA) mbar_wait(done_bar(tile), (uint32_t)((it / NA - 1) & 1));           // the MMAs that read the tile last
            const uint32_t row_lo0 = row0 + tile * (2 * kTileBytesAB);
            if (w8 == 0) SKTS(3, it);
#pragma unroll
            for (int kk = 0; kk < 2; kk++) {
                const __half2 d2 = u2h(dq[kk]), m2 = u2h(mq[kk]);
                const __half2 dlo = __low2half2(d2), dhi = __high2half2(d2);
                const __half2 mlo = __low2half2(m2), mhi = __high2half2(m2);
                const uint32_t row_lo = row_lo0 + kk * kTileBytesAB, row_hi = row_lo + 1024;
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    uint32_t va[4], vb[4];
                    E::run(cw[kk], 2 * h, dlo, dhi, mlo, mhi, lut, va);
                    E::run(cw[kk], 2 * h + 1, dlo, dhi, mlo, mhi, lut, vb);
                    if (BF) {
#pragma unroll
                        for (int i = 0; i < 4; i++) { va[i] = h2_to_bf2(va[i]); vb[i] = h2_to_bf2(vb[i]); }
                    }
                    const uint32_t chunk = (uint32_t)((2 * t + h) ^ g) * 16;
                    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(row_lo + chunk), "r"(va[0]), "r"(va[2]), "r"(vb[0]), "r"(vb[2]) : "memory");
                    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(row_hi + chunk), "r"(va[1]), "r"(va[3]), "r"(vb[1]), "r"(vb[3]) : "memory");
                }
            }
            if (w8 == 0) SKTS(4, it);
            // only now are the codes surely in registers: an arrival behind the loads alone, before anything used them, let the next copy
            // overtake a load now and then
            __syncwarp();
            if (lane == 0) mbar_arrive(free_bar(s));
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            mbar_arrive(afull_bar(tile));
            if (w8 == 0) SKTS(5, it);
        }
    } else {
        // ================= epilogue warps: TMEM lanes 32 * (warp % 4) .. + 31 = features, columns = tokens =================
        const int quarter = warp & 3;
        const int n_seg = n_items > 0 ? (int)((i_end - 1) / np) - ft0 + 1 : 0;
        if (A.pdl) asm volatile("griddepcontrol.wait;" ::: "memory");      // the workspace may still be read by the previous reduction
        for (int seg = 0; seg < n_seg; seg++) {
            mbar_wait(tmem_full(seg & 1), (uint32_t)((seg >> 1) & 1));
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // the reduction may be scheduled while the last tiles are stored: it waits for this grid's end.  Calls in a row, launched
            // behind the grid -> so: 40 rows, 11008 x 4096 20.5 -> 18.6 us, 17 rows, 1024 x 1024 16.5 -> 12.4, an MLP of 60 rows, 4096 /
            // 14336, 74.4 -> 68.0.  (From the kernel's start the waiting blocks cost the recorded MLP 2 %.)
            if (seg + 1 == n_seg) asm volatile("griddepcontrol.launch_dependents;");
            float* dst = A.part + ((int64_t)blockIdx.x * A.max_seg + seg) * (NTOK * 128) + quarter * 32 + lane;
            constexpr int CH = NTOK % 32 ? 16 : 32;
#pragma unroll 1
            for (int c = 0; c < NTOK; c += CH) {
                float v[CH];
                tmem_ld_cols<CH>(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)((seg & 1) * ACC_COLS + c), v);
#pragma unroll
                for (int j = 0; j < CH; j++)
                    if (c + j < A.M) dst[(c + j) * 128] = v[j];          // a warp writes 128 contiguous bytes per token
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            mbar_arrive(tmem_empty(seg & 1));
        }
    }
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}

// y[token][feature] = sum over the CTAs whose range touches the feature's tile, in CTA order, + bias (+ y).
// grid = (feature tiles, ceil(M / 8)); a block adds eight tokens of one tile, thread = feature.
struct SkReduceArgs {
    const float* part; int max_seg, grid, np, ntok, M;
    int64_t total, n_cols;
    void* y; int y_dtype; const void* bias; int accumulate; int pdl;
    int mlp_act, n_ft1;      // mlp_act != 0: y = act(tile ft) * (tile ft + n_ft1), the fused MLP's two matrices (1 SiLU, 2 GELU)
};
__global__ void __launch_bounds__(128) skinny_reduce_kernel(const SkReduceArgs A) {
    if (A.pdl) asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int ft = blockIdx.x, f = threadIdx.x;
    // CTA of item i = the largest c with c * total / grid <= i
    auto cta_of = [&](int64_t i) { return (int)(((i + 1) * A.grid + A.total - 1) / A.total - 1); };
    const int t0 = blockIdx.y * 8;
    auto tile_sum = [&](int tile, float (&v)[8]) {       // the partial tiles of `tile`, in CTA order
        const int c_lo = cta_of((int64_t)tile * A.np), c_hi = cta_of((int64_t)(tile + 1) * A.np - 1);
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = 0.0f;
        auto part_of = [&](int c) {
            const int seg = tile - (int)(((int64_t)c * A.total / A.grid) / A.np);
            return A.part + ((int64_t)c * A.max_seg + seg) * (A.ntok * 128) + t0 * 128 + f;
        };
        for (int c = c_lo; c <= c_hi; c += 3) {          // three are asked for at once: one by one each waits for the memory in turn
            const float *const p0 = part_of(c), *const p1 = part_of(c + 1 > c_hi ? c : c + 1), *const p2 = part_of(c + 2 > c_hi ? c : c + 2);
            float a0[8], a1[8], a2[8];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const bool there = t0 + j < A.M;
                a0[j] = there ? p0[j * 128] : 0.0f;
                a1[j] = there && c + 1 <= c_hi ? p1[j * 128] : 0.0f;
                a2[j] = there && c + 2 <= c_hi ? p2[j * 128] : 0.0f;
            }
#pragma unroll
            for (int j = 0; j < 8; j++) {
                v[j] += a0[j];
                if (c + 1 <= c_hi) v[j] += a1[j];
                if (c + 2 <= c_hi) v[j] += a2[j];
            }
        }
    };
    float v[8];
    tile_sum(ft, v);
    if (A.mlp_act) {                                     // fused MLP: act(gate) * up
        float u[8];
        tile_sum(ft + A.n_ft1, u);
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = apply_act(v[j], A.mlp_act) * u[j];
    }
    const int64_t col = (int64_t)ft * kTileN + f;
    float b = 0.0f;
    if (A.bias) b = A.y_dtype == DT_F32 ? ((const float*)A.bias)[col]
                  : A.y_dtype == DT_F16 ? __half2float(((const __half*)A.bias)[col]) : __bfloat162float(((const __nv_bfloat16*)A.bias)[col]);
#pragma unroll
    for (int j = 0; j < 8; j++) {
        if (t0 + j >= A.M) break;
        const int64_t idx = (int64_t)(t0 + j) * A.n_cols + col;
        const float r = v[j] + b;
        if (A.y_dtype == DT_F32) { float* p = (float*)A.y + idx; *p = A.accumulate ? *p + r : r; }
        else if (A.y_dtype == DT_F16) { __half* p = (__half*)A.y + idx; *p = __float2half_rn(A.accumulate ? __half2float(*p) + r : r); }
        else { __nv_bfloat16* p = (__nv_bfloat16*)A.y + idx; *p = __float2bfloat16_rn(A.accumulate ? __bfloat162float(*p) + r : r); }
    }
}

template <int QT, bool BF, int NTOK>
static int sk_launch_one(const CUtensorMap& map, const SkinnyArgs& A, int grid, cudaStream_t st) {
    constexpr int SMEM = SkSmem<QT, NTOK>::kTotal;
    static bool configured_dev[64] = {};
    int dev_id = 0;
    cudaGetDevice(&dev_id);
    bool& configured = configured_dev[dev_id & 63];
    if (!configured) {
        cudaFuncSetAttribute(skinny_kernel<QT, BF, NTOK>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
        configured = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid); cfg.blockDim = dim3(kSkThreads); cfg.dynamicSmemBytes = SMEM; cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = A.pdl ? 1 : 0;
    cudaLaunchKernelEx(&cfg, skinny_kernel<QT, BF, NTOK>, map, A);
    return 0;
}
template <int QT>
static int sk_launch_qt(bool bf, int ntok, const CUtensorMap& map, const SkinnyArgs& A, int grid, cudaStream_t st) {
#define SK_CASE(N) case N: return bf ? sk_launch_one<QT, true, N>(map, A, grid, st) : sk_launch_one<QT, false, N>(map, A, grid, st);
    switch (ntok) { SK_CASE(32) SK_CASE(48) SK_CASE(64) }
#undef SK_CASE
    return LB_ERR_ARG;
}
// 48 columns for 33 to 48 rows: 64 move a third more activations through shared memory.  48 rows against 49, 14336 x 4096: sym_int4 16.3 / 17.4 us,
// asym_int4 16.3 / 16.8, nf4 19.8 / 21.0, fp8_e4m3 19.2 / 19.6, fp6 17.2 / 19.6
static int sk_ntok(int64_t m) { return m <= 32 ? 32 : m <= 48 ? 48 : 64; }
static int sk_grid(int64_t total) { const int sms = sm_count(); return (int)(total < sms ? total : sms); }
static int sk_max_seg(int64_t total, int grid, int64_t np) { return (int)(((total + grid - 1) / grid + np - 1) / np + 1); }
}  // namespace gemmtc

#ifdef LOWBIT_SK_TIMESTAMPS
extern "C" int lowbit_debug_skinny_timestamps(unsigned long long* out) {
    return (int)cudaMemcpyFromSymbol(out, gemmtc::g_sk_ts, sizeof(gemmtc::g_sk_ts));
}
#endif
// ---- skinny variant (at most 64 rows, fp16 / bf16 activations): see gemmtc::skinny_kernel
bool gemm_skinny_supported(int qt, int64_t n_rows, int64_t k, int64_t m, int x_dtype) {
    return (x_dtype == DT_F16 || x_dtype == DT_BF16) && m >= 1 && m <= 64 && gemm_tc_supported(qt, n_rows, k) && (n_rows % 128) == 0 &&
           (k % 128) == 0;                                 // an item is a pair of k-blocks
}
size_t gemm_skinny_workspace_size(int64_t n_rows, int64_t k, int64_t m) {
    using namespace gemmtc;
    const int64_t np = k / 128, total = (n_rows / 128) * np;
    const int grid = sk_grid(total);
    return (size_t)grid * sk_max_seg(total, grid, np) * sk_ntok(m) * 128 * sizeof(float);
}
static int skinny_launch_impl(const void* w, const void* w2, int mlp_act, int qt, int64_t n_rows, int64_t k, const void* x, int x_dtype,
                              int64_t m, void* y, int y_dtype, const void* bias, int accumulate, void* workspace, size_t workspace_bytes,
                              cudaStream_t st, int pdl);
int gemm_skinny_launch(const void* w, int qt, int64_t n_rows, int64_t k, const void* x, int x_dtype, int64_t m, void* y, int y_dtype,
                       const void* bias, int accumulate, void* workspace, size_t workspace_bytes, cudaStream_t st, int pdl) {
    return skinny_launch_impl(w, nullptr, 0, qt, n_rows, k, x, x_dtype, m, y, y_dtype, bias, accumulate, workspace, workspace_bytes, st, pdl);
}
// fused MLP front half for 17..64 rows: y = act(x . Wgate^T) * (x . Wup^T); both matrices in ONE stream-K pass (their feature
// tiles follow each other in the item sequence), the activation and the product in the reduction launch.  act: 1 SiLU, 2 GELU
size_t gemm_skinny_mlp_workspace_size(int64_t n_rows, int64_t k, int64_t m) {
    using namespace gemmtc;
    const int64_t np = k / 128, total = 2 * (n_rows / 128) * np;
    const int grid = sk_grid(total);
    return (size_t)grid * sk_max_seg(total, grid, np) * sk_ntok(m) * 128 * sizeof(float);
}
int gemm_skinny_mlp_launch(const void* w_gate, const void* w_up, int act, int qt, int64_t n_rows, int64_t k, const void* x, int x_dtype,
                           int64_t m, void* y, int y_dtype, void* workspace, size_t workspace_bytes, cudaStream_t st, int pdl) {
    if (!w_up || act < 1 || act > 2 || ((uintptr_t)w_up & 15)) return LB_ERR_ARG;
    return skinny_launch_impl(w_gate, w_up, act, qt, n_rows, k, x, x_dtype, m, y, y_dtype, nullptr, 0, workspace, workspace_bytes, st, pdl);
}
static int skinny_launch_impl(const void* w, const void* w2, int mlp_act, int qt, int64_t n_rows, int64_t k, const void* x, int x_dtype,
                              int64_t m, void* y, int y_dtype, const void* bias, int accumulate, void* workspace, size_t workspace_bytes,
                              cudaStream_t st, int pdl) {
    using namespace gemmtc;
    qt = canon_qtype(qt);
    if (!gemm_skinny_supported(qt, n_rows, k, m, x_dtype)) return LB_ERR_ARG;
    if (((uintptr_t)x & 15) || ((uintptr_t)w & 15)) return LB_ERR_ARG;
    if (!workspace || workspace_bytes < (w2 ? gemm_skinny_mlp_workspace_size(n_rows, k, m) : gemm_skinny_workspace_size(n_rows, k, m))) return LB_ERR_WORKSPACE;
    const bool bf = x_dtype == DT_BF16;
    const int ntok = sk_ntok(m);
    CUtensorMap map;
    if (const int rc = encode_rows(&map, x, bf, m, k, ntok)) return rc;
    SkinnyArgs A;
    A.w = (const uint8_t*)w; A.w2 = (const uint8_t*)w2; A.G = make_geom(n_rows, k, qt); A.M = (int)m;
    const int64_t np = k / 128, total = (w2 ? 2 : 1) * (n_rows / 128) * np;
    const int grid = sk_grid(total);
    A.part = (float*)workspace; A.max_seg = sk_max_seg(total, grid, np); A.pdl = pdl;
    int rc;
    switch (qt) {
        case QT_SYM_INT4:  rc = sk_launch_qt<QT_SYM_INT4>(bf, ntok, map, A, grid, st); break;
        case QT_NF4:       rc = sk_launch_qt<QT_NF4>(bf, ntok, map, A, grid, st); break;
        case QT_ASYM_INT4: rc = sk_launch_qt<QT_ASYM_INT4>(bf, ntok, map, A, grid, st); break;
        case QT_FP8_E4M3:  rc = sk_launch_qt<QT_FP8_E4M3>(bf, ntok, map, A, grid, st); break;
        case QT_FP8_E5M2:  rc = sk_launch_qt<QT_FP8_E5M2>(bf, ntok, map, A, grid, st); break;
        case QT_FP6:       rc = sk_launch_qt<QT_FP6>(bf, ntok, map, A, grid, st); break;
        default: return LB_ERR_ARG;
    }
    if (rc) return rc;
    note_launch();
    SkReduceArgs R;
    R.part = A.part; R.max_seg = A.max_seg; R.grid = grid; R.np = (int)np; R.ntok = ntok; R.M = (int)m;
    R.total = total; R.n_cols = n_rows; R.y = y; R.y_dtype = y_dtype; R.bias = bias; R.accumulate = accumulate; R.pdl = pdl;
    R.mlp_act = w2 ? mlp_act : 0; R.n_ft1 = (int)(n_rows / 128);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(n_rows / 128), (unsigned)((m + 7) / 8)); cfg.blockDim = dim3(128); cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = 1;                         // whatever the switch for the launches around this one says
    cudaLaunchKernelEx(&cfg, skinny_reduce_kernel, R);
    note_launch();
    return check_launch();
}

}  // namespace lowbit
