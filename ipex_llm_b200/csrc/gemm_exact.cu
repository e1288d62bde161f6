// gemm_exact.cu -- the fp32 matmul of a prompt on the 5th-generation tensor cores: y[M][N] (+)= x[M][K] . dequant(W[N][K])^T with 32-bit
// activations kept to 2^-24, the fp32-in / fp32-out contract of ggml_compute_forward_mul_mat_q_fp32 (reference
// low_bit_linear.py:494-529), for more than 32 rows.
//
// The arithmetic is the exact GEMV's (gemv_kernel.cuh): the CODES (4-bit offsets, e4m3 / e5m2 / e3m2 values) are exact in bf16, an
// activation is the sum of three bf16 planes, so every product is exact in 32 bits; a 64-element block's sum leaves the tensor cores
// after 12 steps and is multiplied by the block's scale and added in 32-bit floats.  asym_int4's minima multiply the
// activations' sums per block, which split3_kernel leaves; nf4's table is the sum of two bf16 planes (2^-17), as there.
//
// Layout of the work as in gemm_pair.cu: a cluster of two CTAs computes 256 features x up to 128 tokens with tcgen05.mma.cta_group::2,
// codes expanded to bf16 = A operand, the token planes = B, each CTA staging half of the tokens (boxes of 32 rows, three planes per
// k-block).  Every k-block has a TMEM buffer of its own; eight epilogue warps drain it: lane = feature, so a block's scale is one value
// per lane, and a thread keeps half of the tile's tokens' sums in registers over the unit's K range.
//   warp 0 token planes (TMA), warp 1 MMAs / relay, warp 2 packed weights, warp 3 TMEM, then two or three expansion groups of four
//   warps, then eight warps of epilogue.
// Tiles of 64 tokens alone (the first form) read A from shared memory for every 32 clocks of MMAs (N = 64 of twelve steps) and took 900
// clocks a k-block: 500 of them four barrier tests one after the other (asked together and ahead now), then the MMAs themselves; at 128
// tokens a step's math covers its operands.  All three planes in one step of N = 192 halved the MMA time but made the epilogue read
// three times as much TMEM: 600 clocks a k-block, slower than either.  The kernel starts while split3_kernel runs and waits only in
// front of the planes.  sym_int4, GEMV passes of 32 rows -> 64-token tiles -> now: 4096 x 4096 at 33 rows 33.8 -> 17.7 -> 15.6 us, 64 rows
// 50.4 -> 18.1 -> 15.6, 200 rows 161 -> 38.0 -> 26.8, 512 rows 400 -> 69.9 -> 40.4; 11008 x 4096 at 512 rows 938 -> 160 -> 105; 1024 x 1024
// at 33 rows 18.2 -> 12.5 -> 10.9.  asym_int4 (passes -> now): 4096 x 4096 at 33 rows 46.1 -> 25.6, 200 rows 198 -> 44.0, 1000 rows 915 ->
// 128, 31232 x 9280 at 506 rows 3812 -> 804; the minima's loads straight from L2, two blocks under way, took 1422 there.
// nf4: 56.4 -> 29.7, 245 -> 48.1, 1166 -> 142, 5013 -> 1084.  Error against 64 bits, relative to the result's norm: the GEMV 4.8e-7, here 1.2e-7 to 1.5e-7
// (sym_int4, 4096 x 4096).  At 512 rows the MMAs' twelve steps are 3/4 of the time; below 100 rows it is the three launches' ends.
#include "tc_pair.cuh"

namespace lowbit {
namespace gemmtc {

constexpr int kExTok = 128, kExDeq0 = 4;     // most tokens of a tile; first expanding warp

// nf4's table is held as two bf16 planes, the GEMV's: a k-block is two A tiles and 24 MMA steps into one TMEM buffer, on the same packed
// weights and token planes.  A tile's values come out of registers, four codes to a byte permutation of the table's low and high halves (the
// shared table that the 16-bit kernel reads costs 32 KB a plane, which the token planes' ring needs).
template <int QT> struct ExWeights {
    static constexpr int kPlanes = 1;
    struct Table {};
    __device__ static __forceinline__ void table(bool, Table&) {}
};
template <> struct ExWeights<QT_NF4> {
    static constexpr int kPlanes = 2;
    struct Table { uint32_t lo[4], hi[4]; };                           // low and high bytes of 16 bf16 values
    __device__ static __forceinline__ void table(bool rest, Table& T) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            T.lo[i] = T.hi[i] = 0;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float v = kNF4Table[4 * i + j];
                const __nv_bfloat16 h = __float2bfloat16_rn(v);
                const uint32_t b = __bfloat16_as_ushort(rest ? __float2bfloat16_rn(v - __bfloat162float(h)) : h);
                T.lo[i] |= (b & 0xffu) << (8 * j); T.hi[i] |= (b >> 8) << (8 * j);
            }
        }
    }
    // byte b of the lane's word is the code pair of out[b]
    __device__ static __forceinline__ void expand(const Table& T, uint32_t w, uint32_t (&out)[4]) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const uint32_t c = w >> (16 * h), at = c & 0x7777u, upper = __byte_perm(0xff00u, 0u, (c >> 3) & 0x1111u);
            const uint32_t lo = (__byte_perm(T.lo[0], T.lo[1], at) & ~upper) | (__byte_perm(T.lo[2], T.lo[3], at) & upper);
            const uint32_t hi = (__byte_perm(T.hi[0], T.hi[1], at) & ~upper) | (__byte_perm(T.hi[2], T.hi[3], at) & upper);
            out[2 * h] = __byte_perm(lo, hi, 0x5140u);
            out[2 * h + 1] = __byte_perm(lo, hi, 0x7362u);
        }
    }
};

// TOK: 64 tokens or 128.  A thread of the epilogue keeps half of them, so the larger tile leaves registers for two expansion groups only;
// its MMAs take that long.
template <int QT, int TOK> struct ExShape {
    static constexpr int kGroups = TOK == 64 ? 3 : 2, kEpi0 = kExDeq0 + 4 * kGroups, kThreads = 32 * (kEpi0 + 8);
    static constexpr int kSteps = ExWeights<QT>::kPlanes;              // A tiles of a k-block
    static constexpr int kBufs = 512 / TOK;                            // TMEM: one for every k-block in flight
    static constexpr int kGroup = PackedBlock<QT>::kGroup, kPacked = 2 * kGroup;
    static constexpr int kA = TOK == 64 ? 3 : 4, kP = 6, kX = TOK == 64 ? 6 : 4;
    static constexpr int kXPlane = TOK * 64, kXSlot = 3 * kXPlane;     // half of the tokens' rows of 128 bytes
    static constexpr int kTotal = 1024 + 512 + kA * kTileBytesAB + kP * kPacked + kX * kXSlot + (Expand<QT>::kHasMin ? 8 * TOK * 4 : 0);
    static_assert(kTotal <= 232448, "shared memory");
    static_assert(kP % kGroups == 0 && (3 * kX + 2 * kP + 2 * kA + 2 * kBufs + 1) * 8 + 8 <= 512, "barrier region");
};

struct ExactArgs {
    const uint8_t* w;
    TiledGeom G;
    int M, tt, n_fp, ksplit;
    float* y; const float* bias; int accumulate;
    float* part;
    const float* sums; int sum_rows;        // minima: [k-block][sum_rows] the activations' sums, tokens padded to whole 16
    Waits waits;
};

template <int QT, int TOK>
__global__ void __launch_bounds__(ExShape<QT, TOK>::kThreads, 1)
exact_kernel(const __grid_constant__ CUtensorMap xmap, const ExactArgs A) {
    using E = Expand<QT>;
    using SM = ExShape<QT, TOK>;
    constexpr int KX = SM::kX, KP = SM::kP, KA = SM::kA, GROUPS = SM::kGroups, BUFS = SM::kBufs, STEPS = SM::kSteps;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t xring = base, aring = base + KX * SM::kXSlot, pring = aring + KA * kTileBytesAB, bars = base + SM::kTotal - 1536;
    auto x_full = [&](int s) { return bars + s * 8; };
    auto x_empty = [&](int s) { return bars + (KX + s) * 8; };
    auto xp_full = [&](int s) { return bars + (2 * KX + s) * 8; };                     // CTA 0: the other half has landed
    auto p_full = [&](int s) { return bars + (3 * KX + s) * 8; };
    auto p_empty = [&](int s) { return bars + (3 * KX + KP + s) * 8; };
    auto a_full = [&](int s) { return bars + (3 * KX + 2 * KP + s) * 8; };             // CTA 0: both CTAs' tiles are expanded
    auto a_empty = [&](int s) { return bars + (3 * KX + 2 * KP + KA + s) * 8; };
    auto t_full = [&](int b) { return bars + (3 * KX + 2 * KP + 2 * KA + b) * 8; };
    auto t_empty = [&](int b) { return bars + (3 * KX + 2 * KP + 2 * KA + BUFS + b) * 8; };   // CTA 0: both epilogues have read it
    const uint32_t drained = bars + (3 * KX + 2 * KP + 2 * KA + 2 * BUFS) * 8;      // every MMA that was issued is done
    const uint32_t tmem_slot = drained + 8;
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31, rank = (int)(blockIdx.x & 1);
    const int nb = (int)A.G.nb;
    if (threadIdx.x == 0) {
        for (int s = 0; s < KX; s++) { mbar_init(x_full(s), 1); mbar_init(x_empty(s), 1); mbar_init(xp_full(s), 1); }
        for (int s = 0; s < KP; s++) { mbar_init(p_full(s), 1); mbar_init(p_empty(s), 4 * STEPS); }
        for (int s = 0; s < KA; s++) { mbar_init(a_full(s), 8); mbar_init(a_empty(s), 1); }
        for (int b = 0; b < BUFS; b++) { mbar_init(t_full(b), 1); mbar_init(t_empty(b), 16); }
        mbar_init(drained, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 3) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync_all();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    uint32_t tmem_base;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem_base) : "r"(tmem_slot));

    const int n_tiles = (A.M + A.tt - 1) / A.tt, n_units = n_tiles * A.n_fp * A.ksplit, stride = (int)(gridDim.x >> 1);
    struct Unit { int m0, rows, n_tok, ft, ks, kb0, kb1; };
    auto decode = [&](int unit, Unit& U) {
        const int fp = unit % A.n_fp, rest = unit / A.n_fp;
        U.m0 = (rest % n_tiles) * A.tt;
        U.rows = min(A.M, U.m0 + A.tt) - U.m0;
        U.n_tok = (U.rows + 15) & ~15;
        U.ft = 2 * fp + rank;
        U.ks = rest / n_tiles;
        U.kb0 = (U.ks * nb) / A.ksplit;
        U.kb1 = ((U.ks + 1) * nb) / A.ksplit;
    };
    Unit U;
    const uint32_t leader = elect_leader();
    int s = 0, round = 0;                                  // the two copying warps' place in their ring

    if (warp == 0) {
        // ================= token planes: this CTA's half of the tile's tokens =================
        asm volatile("griddepcontrol.wait;" ::: "memory");     // split3_kernel's; the weights' copies and expansion have begun meanwhile
        for (int unit = blockIdx.x >> 1; unit < n_units; unit += stride) {
            decode(unit, U);
            if (unit + stride >= n_units) asm volatile("griddepcontrol.launch_dependents;");     // the cluster's last unit
            const int row0 = U.m0 + rank * (U.n_tok >> 1), boxes = ((U.n_tok >> 1) + 31) >> 5;
            for (int kb = U.kb0; kb < U.kb1; kb++) {
                if (!mbar_wait_lim(x_empty(s), (uint32_t)((round & 1) ^ 1), A.waits)) goto done;
                mbar_expect_tx_w(x_full(s), 3 * boxes * 4096, leader);
                // rows of a plane beyond the last token belong to the next plane (or read zero): columns that nothing stores
                for (int p = 0; p < 3; p++)
                    for (int i = 0; i < boxes; i++) tma_load_2d_w(xring + s * SM::kXSlot + p * SM::kXPlane + i * 4096, &xmap, kb * 64, p * A.M + row0 + 32 * i, x_full(s), leader);
                if (++s == KX) { s = 0; round++; }
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            // ================= MMA issuer: 3 planes x 4 steps per k-block, into the k-block's own TMEM buffer =================
            int sx = 0, rx = 0, sa = 0, ra = 0, tb = 0, rt = 0;
            bool ready = false;
            for (int unit = blockIdx.x >> 1; unit < n_units; unit += stride) {
                decode(unit, U);
                const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (((uint32_t)U.n_tok >> 3) << 17) | ((256u >> 4) << 24);
                for (int kb = STEPS * U.kb0; kb < STEPS * U.kb1; kb++) {
                    if (!mbar_wait4_lim(ready, t_empty(tb), (uint32_t)((rt & 1) ^ 1), x_full(sx), (uint32_t)(rx & 1), xp_full(sx), (uint32_t)(rx & 1), a_full(sa),
                                        (uint32_t)(ra & 1), A.waits)) goto done;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t ad = make_desc(aring + sa * kTileBytesAB), xd = make_desc(xring + sx * SM::kXSlot);
#pragma unroll
                    for (int p = 2; p >= 0; p--)             // the small planes first
#pragma unroll
                        for (int k4 = 0; k4 < 4; k4++)
                            umma2_f16_w(tmem_base + tb * TOK, ad + (uint64_t)((k4 * 32) >> 4), xd + (uint64_t)((p * SM::kXPlane + k4 * 32) >> 4), idesc,
                                        (p < 2 || k4 > 0 || kb % STEPS) ? 1u : 0u, leader);
                    umma2_commit_w(a_empty(sa), leader);
                    if (++sa == KA) { sa = 0; ra++; }
                    if (kb % STEPS == STEPS - 1) {
                        umma2_commit_w(x_empty(sx), leader);
                        umma2_commit_w(t_full(tb), leader);
                        if (++sx == KX) { sx = 0; rx++; }
                        if (++tb == BUFS) { tb = 0; rt++; }
                    }
                    // asked here, answered while the MMAs above are being issued
                    ready = mbar_test4(t_empty(tb), (uint32_t)((rt & 1) ^ 1), x_full(sx), (uint32_t)(rx & 1), xp_full(sx), (uint32_t)(rx & 1), a_full(sa), (uint32_t)(ra & 1));
                }
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
            const int kb_end = A.waits.limit < 0 ? (U.kb0 + U.kb1) / 2 : U.kb1;
            for (int kb = U.kb0; kb < kb_end; kb++) {
                if (!mbar_wait_lim(p_empty(s), (uint32_t)((round & 1) ^ 1), A.waits)) goto done;
                mbar_expect_tx_w(p_full(s), 2 * PackedBlock<QT>::kSuper, leader);
#pragma unroll
                for (int gi = 0; gi < 2; gi++) {
                    const int64_t u = (int64_t)min(2 * U.ft + gi, n_rg - 1) * nb + kb;      // a tile that does not exist repeats the last group
                    bulk_g2s_w(pring + s * SM::kPacked + gi * SM::kGroup, A.w + u * PackedBlock<QT>::kSuper, PackedBlock<QT>::kSuper, p_full(s), leader);
                }
                if (++s == KP) { s = 0; round++; }
            }
            if (kb_end < U.kb1) goto done;
        }
    } else if (warp >= kExDeq0 && warp < SM::kEpi0) {
        // ================= expansion: group (warp - 4) / 4 takes every second (third) k-block =================
        const int grp = (warp - kExDeq0) >> 2, dw = (warp - kExDeq0) & 3, g = lane >> 2, t = lane & 3;
        int end = 0, it = grp, sp = grp / STEPS, rp = 0;      // `it` counts A tiles, STEPS to a k-block: the rest of a table's values first
        typename ExWeights<QT>::Table values, others;
        ExWeights<QT>::table(grp % 2 == 0, values);
        ExWeights<QT>::table(grp % 2 == 1, others);
        for (int unit = blockIdx.x >> 1; unit < n_units; unit += stride) {
            decode(unit, U);
            end += STEPS * (U.kb1 - U.kb0);
            for (; it < end; it += GROUPS) {
                const int sa = it % KA;
                const uint32_t row0 = aring + sa * kTileBytesAB + 4 * dw * 1024 + g * 128;     // rows interleaved by 16 as in gemm_pair.cu
                // the slot's earlier trip (KP k-blocks before) was this group's own too
                if (!mbar_wait_lim(p_full(sp), (uint32_t)(rp & 1), A.waits)) goto done;
                typename E::Codes cw[2];
#pragma unroll
                for (int gi = 0; gi < 2; gi++) E::load(pring + sp * SM::kPacked + gi * SM::kGroup + dw * E::kTileBytes, lane, cw[gi]);
                uint32_t lo[2][8], hi[2][8];
#pragma unroll
                for (int gi = 0; gi < 2; gi++)
#pragma unroll
                    for (int k4 = 0; k4 < 4; k4++) {
                        uint32_t a[4];
                        if constexpr (STEPS == 2) {
                            const uint32_t w = k4 == 0 ? cw[gi].q.x : k4 == 1 ? cw[gi].q.y : k4 == 2 ? cw[gi].q.z : cw[gi].q.w;
                            ExWeights<QT>::expand(values, w, a);
                        } else {
                            E::bf16(cw[gi], k4, a);
                        }
                        lo[gi][2 * k4] = a[0]; lo[gi][2 * k4 + 1] = a[2];
                        hi[gi][2 * k4] = a[1]; hi[gi][2 * k4 + 1] = a[3];
                    }
                if (!mbar_wait_lim(a_empty(sa), (uint32_t)(((it / KA) & 1) ^ 1), A.waits)) goto done;
#pragma unroll
                for (int gi = 0; gi < 2; gi++)
#pragma unroll
                    for (int q = 0; q < 2; q++) {
                        const uint32_t at = row0 + gi * 2048 + (uint32_t)((2 * t + q) ^ g) * 16;
                        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(lo[gi][4 * q]), "r"(lo[gi][4 * q + 1]), "r"(lo[gi][4 * q + 2]), "r"(lo[gi][4 * q + 3]) : "memory");
                        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at + 1024), "r"(hi[gi][4 * q]), "r"(hi[gi][4 * q + 1]), "r"(hi[gi][4 * q + 2]), "r"(hi[gi][4 * q + 3]) : "memory");
                    }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) { mbar_arrive(p_empty(sp)); mbar_arrive_at(a_full(sa), 0); }      // behind the stores: the codes have been used
                if (STEPS == 1) {
                    if ((sp += GROUPS) >= KP) { sp -= KP; rp++; }
                } else {
                    sp = (it + GROUPS) / STEPS % KP; rp = (it + GROUPS) / STEPS / KP;
                    if (GROUPS % 2) { const auto t = values; values = others; others = t; }
                }
            }
        }
    } else if (warp >= SM::kEpi0) {
        // ================= epilogue: TMEM lanes 32 * (warp % 4) .., half `part` of the tile's tokens =================
        const int quarter = warp & 3, part = (warp - SM::kEpi0) >> 2, half = lane >> 4;
        const int64_t N = A.G.rows;
        int tb = 0, rt = 0;
        for (int unit = blockIdx.x >> 1; unit < n_units; unit += stride) {
            decode(unit, U);
            const int64_t f0 = (int64_t)U.ft * 128, n = f0 + 64 * half + 16 * quarter + (lane & 15);
            const bool valid = f0 < N;
            // the lane's scales: row 16 quarter + (lane & 15) of 64-row group 2 ft + half, one fp16 per k-block, 128 bytes apart
            const int64_t rg = valid ? 2 * U.ft + half : 0;
            const __half* sp = reinterpret_cast<const __half*>(A.w + A.G.off_s + (rg * nb) * 128) + (lane & 7) * 8 + quarter * 2 + ((lane >> 3) & 1);
            constexpr int TOKS = TOK / 2;
            const int t0 = TOKS * part;
            float acc[TOKS];
#pragma unroll
            for (int i = 0; i < TOKS; i++) acc[i] = 0.0f;
            // value = (code - 8) d + (min + 8 d) with minima: the second part times the block's activations' sums, in the time that a wait for
            // the block's MMAs takes; a block's scale and minimum are kept as they are stored
            if (E::kHasMin && unit == (int)(blockIdx.x >> 1)) asm volatile("griddepcontrol.wait;" ::: "memory");
            auto block = [&](int kb) {
                __half2 h = __half2half2(__ushort_as_half(0));
                if (kb < U.kb1) {
                    h.x = sp[(int64_t)kb * 64];
                    if constexpr (E::kHasMin) h.y = sp[(int64_t)kb * 64 + (A.G.off_m - A.G.off_s) / 2];
                }
                return h;
            };
            // the warp's tokens' sums of a block, loaded one block ahead and handed round through shared memory
            const uint32_t sums_at = pring + KP * SM::kPacked + (uint32_t)(warp - SM::kEpi0) * (2 * TOKS * 4);
            auto sums = [&](int kb) {
                constexpr int kEach = TOKS / 32;
                float2 v = make_float2(0.0f, 0.0f);
                if (E::kHasMin && kb < U.kb1 && t0 + kEach * lane < U.rows) {
                    const float* const at = A.sums + (int64_t)kb * A.sum_rows + U.m0 + t0 + kEach * lane;
                    if constexpr (kEach == 2) v = *reinterpret_cast<const float2*>(at);
                    else v.x = *at;
                }
                return v;
            };
            float2 ahead = sums(U.kb0);
            __syncwarp();                                        // the last unit's reads lie before the first writes
            constexpr int kAhead = E::kHasMin ? 2 : 4;           // blocks' scales loaded ahead; with sums the registers are full
            __half2 next[kAhead];
#pragma unroll
            for (int i = 0; i < kAhead; i++) next[i] = block(U.kb0 + i);
            for (int kb = U.kb0; kb < U.kb1; kb += kAhead) {
                __half2 now[kAhead];
#pragma unroll
                for (int i = 0; i < kAhead; i++) now[i] = next[i];
#pragma unroll
                for (int i = 0; i < kAhead; i++) next[i] = block(kb + kAhead + i);
#pragma unroll
                for (int i = 0; i < kAhead; i++) {
                    if (kb + i >= U.kb1) break;
                    const float d = __low2float(now[i]);
                    if constexpr (E::kHasMin) {
                        const float least = fmaf(8.0f, d, __high2float(now[i]));
                        const uint32_t held = sums_at + (uint32_t)((kb + i) & 1) * (TOKS * 4);
                        if constexpr (TOKS == 64) asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(held + lane * 8), "f"(ahead.x), "f"(ahead.y) : "memory");
                        else asm volatile("st.shared.f32 [%0], %1;" ::"r"(held + lane * 4), "f"(ahead.x) : "memory");
                        __syncwarp();                            // the one of the next block lies between these reads and the next writes here
                        ahead = sums(kb + i + 1);
#pragma unroll
                        for (int c = 0; c < TOKS; c += 16) {
                            if (t0 + c >= U.rows) break;
#pragma unroll
                            for (int j = 0; j < 16; j += 4) {
                                float4 v;
                                asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(held + (c + j) * 4) : "memory");
                                acc[c + j] = fmaf(least, v.x, acc[c + j]); acc[c + j + 1] = fmaf(least, v.y, acc[c + j + 1]);
                                acc[c + j + 2] = fmaf(least, v.z, acc[c + j + 2]); acc[c + j + 3] = fmaf(least, v.w, acc[c + j + 3]);
                            }
                        }
                    }
                    if (!mbar_wait_lim(t_full(tb), (uint32_t)(rt & 1), A.waits)) goto done;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                    for (int c = 0; c < TOKS; c += 16) {
                        if (t0 + c >= U.rows) break;
                        float v[16];
                        tmem_ld16(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(tb * TOK + t0 + c), v);
#pragma unroll
                        for (int j = 0; j < 16; j++) acc[c + j] = fmaf(d, v[j], acc[c + j]);
                    }
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive_at(t_empty(tb), 0);
                    if (++tb == BUFS) { tb = 0; rt++; }
                }
            }
            if (valid && t0 < U.rows) {
                const int64_t at = (int64_t)(U.m0 + t0) * N + n;
                const float b = A.bias && A.ksplit == 1 ? A.bias[n] : 0.0f;
                float* const dst = A.ksplit > 1 ? A.part + (int64_t)U.ks * A.M * N + at : A.y + at;
#pragma unroll
                for (int c = 0; c < TOKS; c += 16) {
                    float v[16];
#pragma unroll
                    for (int j = 0; j < 16; j++) v[j] = acc[c + j];
                    store_feature(dst + c * N, N, v, U.rows - t0 - c, b, A.ksplit == 1 && A.accumulate);
                }
            }
            __syncwarp();
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
    cluster_sync_all();
    if (warp == 3) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

// fp32 activations -> three bf16 planes whose sum reproduces them to 2^-24, four elements a thread; `sums`: those of 64 elements, for minima
__global__ void __launch_bounds__(256) split3_kernel(const float4* x, uint2* out, int64_t n4, float* sums, int k4, int sum_rows) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");     // not before the wait: the matmul reads its weights ahead of its own
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n4; i += (int64_t)gridDim.x * blockDim.x) {
        const float4 q = x[i];
        float r[4] = {q.x, q.y, q.z, q.w};
        if (sums) {                                        // 16 lanes hold a block of 64, and all of them are here
            float v = (q.x + q.y) + (q.z + q.w);
#pragma unroll
            for (int d = 1; d < 16; d <<= 1) v += __shfl_xor_sync(0xffffu << (threadIdx.x & 16), v, d);
            const int64_t token = i / k4;
            if ((threadIdx.x & 15) == 0) sums[((i - token * k4) >> 4) * sum_rows + token] = v;
        }
#pragma unroll
        for (int p = 0; p < 3; p++) {
            uint32_t b[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const __nv_bfloat16 h = __float2bfloat16_rn(r[j]);
                b[j] = __bfloat16_as_ushort(h);
                r[j] -= __bfloat162float(h);
            }
            out[p * n4 + i] = make_uint2(b[0] | (b[1] << 16), b[2] | (b[3] << 16));
        }
    }
}

template <int QT, int TOK> static int exact_launch_tile(const CUtensorMap& map, const ExactArgs& A, int64_t units, cudaStream_t st) {
    constexpr int SMEM = ExShape<QT, TOK>::kTotal;
    static int cached[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    int& clusters = cached[dev & 63];
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(sm_count() & ~1)); cfg.blockDim = dim3(ExShape<QT, TOK>::kThreads); cfg.dynamicSmemBytes = SMEM; cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    if (!clusters) {
        int c = 0;
        if (cudaFuncSetAttribute(exact_kernel<QT, TOK>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) != cudaSuccess) {
            cudaGetLastError();
            set_error(LB_ERR_CUDA, "the two-SM fp32 matmul cannot be configured on this device");
            return LB_ERR_CUDA;
        }
        if (cudaOccupancyMaxActiveClusters(&c, exact_kernel<QT, TOK>, &cfg) != cudaSuccess || c <= 0) { cudaGetLastError(); c = sm_count() / 2; }
        clusters = c;
    }
    cfg.gridDim = dim3(2u * (unsigned)(units < clusters ? units : clusters));
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = 2;
    cudaLaunchKernelEx(&cfg, exact_kernel<QT, TOK>, map, A);
    note_launch();
    return LB_OK;
}
template <int QT> static int exact_launch_one(const CUtensorMap& map, const ExactArgs& A, int64_t units, cudaStream_t st) {
    return A.tt <= 64 ? exact_launch_tile<QT, 64>(map, A, units, st) : exact_launch_tile<QT, 128>(map, A, units, st);
}

// Token tile and K splits: rounds of the resident clusters x (k-blocks per unit + a unit's start and end), + the partial sums' round trip and
// its launch.  Fitted to 918 times (33 to 512 rows, 1024 to 11008 features, K 2048 to 11008, sym_int4 and fp8): a k-block 0.40 us in tiles of
// up to 64 tokens, 0.52 above (its MMAs, 0.0031 us a token, are 3/4 of that at 128), a unit 1.2 us and 0.014 a token, partial sums 6.6 TB/s
// and 2.7 us.  Over 120 shapes the choice lies 0.4 % over the best tile and split; with 0.33 us for either tile it was 1.6 %.  sym_int4, its
// tile then / now: 65 rows, 2048 x 2048 14.2 us (80 tokens) / 12.6 (48), 512 rows 24.0 (96) / 20.5 (64); 48 rows, 11008 x 4096 33.1 (K
// whole) / 30.4 (three splits); at 128 rows, 4096 x 11008, tiles of 64 take 47.5, of 128 37.2, as then.  asym_int4 and nf4, whose k-blocks take
// longer (another pass over the accumulators, 24 MMA steps for 12), are not among the fitted times: they take the plan of the others
struct ExactPlan { int tt, ks; };
static ExactPlan exact_plan(int64_t n_rows, int64_t nb, int64_t m) {
    const int64_t clusters = sm_count() / 2, n_fp = (n_rows / 128 + 1) / 2, nt0 = (m + kExTok - 1) / kExTok;
    ExactPlan best = {kExTok, 1};
    double best_cost = 1e30;
    for (int64_t nt = nt0; nt <= nt0 + 4 && nt <= (m + 31) / 32; nt++) {
        const int64_t tt = ((m + nt - 1) / nt + 15) & ~int64_t(15);
        const double per_kb = tt <= 64 ? 0.40 : 0.52;
        for (int64_t ks = 1; ks == 1 || (ks <= 8 && nb / ks >= 8); ks++) {
            const int64_t rounds = (n_fp * nt * ks + clusters - 1) / clusters;
            double cost = (double)rounds * ((double)((nb + ks - 1) / ks) * per_kb + 1.2 + 0.014 * (double)tt);
            if (ks > 1) cost += (double)ks * (double)m * (double)n_rows * 8.0 / 6.6e6 + 2.7;
            if (cost < best_cost - 1e-9) { best_cost = cost; best = {(int)tt, (int)ks}; }
        }
    }
    return best;
}
static size_t exact_planes_bytes(int64_t k, int64_t m) { return ((size_t)3 * m * k * 2 + 255) / 256 * 256; }
static int64_t exact_sum_rows(int64_t m) { return (m + 15) / 16 * 16; }
static size_t exact_sums_bytes(int64_t k, int64_t m) { return ((size_t)(k / 64) * exact_sum_rows(m) * 4 + 255) / 256 * 256; }
}  // namespace gemmtc

bool gemm_exact_supported(int qt, int64_t n_rows, int64_t k, int64_t m) {
    qt = canon_qtype(qt);
    return (qt == QT_SYM_INT4 || qt == QT_ASYM_INT4 || qt == QT_NF4 || qt == QT_FP8_E4M3 || qt == QT_FP8_E5M2 || qt == QT_FP6) && gemm_tc_supported(qt, n_rows, k) && 3 * m < 0x7fffffff;
}
size_t gemm_exact_workspace_size(int qt, int64_t n_rows, int64_t k, int64_t m) {
    using namespace gemmtc;
    const ExactPlan p = exact_plan(n_rows, k / 64, m);
    return exact_planes_bytes(k, m) + (canon_qtype(qt) == QT_ASYM_INT4 ? exact_sums_bytes(k, m) : 0) +
           (p.ks > 1 ? (size_t)p.ks * m * n_rows * sizeof(float) : 0);
}
int gemm_exact_launch(const void* w, int qt, int64_t n_rows, int64_t k, const void* x, int64_t m, void* y, const void* bias, int accumulate,
                      void* workspace, size_t workspace_bytes, cudaStream_t st) {
    using namespace gemmtc;
    qt = canon_qtype(qt);
    if (!gemm_exact_supported(qt, n_rows, k, m) || (((uintptr_t)x | (uintptr_t)w | (uintptr_t)workspace) & 15)) return LB_ERR_ARG;
    if (!workspace || workspace_bytes < gemm_exact_workspace_size(qt, n_rows, k, m)) return LB_ERR_WORKSPACE;
    float* const sums = qt == QT_ASYM_INT4 ? (float*)((char*)workspace + exact_planes_bytes(k, m)) : nullptr;
    const int64_t n4 = m * k / 4;                                       // k is a multiple of 64
    int sg = (int)((n4 + 255) / 256); if (sg > sm_count() * 8) sg = sm_count() * 8;
    launch_behind(split3_kernel, dim3((unsigned)sg), 256, 0, st, launch_overlaps(st), (const float4*)x, (uint2*)workspace, n4, sums, (int)(k / 4), (int)exact_sum_rows(m));
    note_launch();
    CUtensorMap map;
    if (const int rc = encode_rows(&map, workspace, true, 3 * m, k, 32)) return rc;
    const ExactPlan p = exact_plan(n_rows, k / 64, m);
    ExactArgs A = {};
    if (const int rc = make_waits(&A.waits, kWaitCycles)) return rc;
    A.w = (const uint8_t*)w; A.G = make_geom(n_rows, k, qt); A.M = (int)m; A.tt = p.tt; A.n_fp = (int)((n_rows / 128 + 1) / 2); A.ksplit = p.ks;
    A.y = (float*)y; A.bias = (const float*)bias; A.accumulate = accumulate; A.part = (float*)((char*)workspace + exact_planes_bytes(k, m) + (sums ? exact_sums_bytes(k, m) : 0));
    A.sums = sums; A.sum_rows = (int)exact_sum_rows(m);
    const int64_t units = (int64_t)A.n_fp * ((m + p.tt - 1) / p.tt) * p.ks;
    int rc = LB_ERR_ARG;
    switch (qt) {
        case QT_SYM_INT4: rc = exact_launch_one<QT_SYM_INT4>(map, A, units, st); break;
        case QT_ASYM_INT4: rc = exact_launch_one<QT_ASYM_INT4>(map, A, units, st); break;
        case QT_NF4:      rc = exact_launch_one<QT_NF4>(map, A, units, st); break;
        case QT_FP8_E4M3: rc = exact_launch_one<QT_FP8_E4M3>(map, A, units, st); break;
        case QT_FP8_E5M2: rc = exact_launch_one<QT_FP8_E5M2>(map, A, units, st); break;
        case QT_FP6:      rc = exact_launch_one<QT_FP6>(map, A, units, st); break;
    }
    if (rc) return rc;
    if (p.ks > 1) {
        const int64_t mn = m * n_rows;
        int rg = (int)((mn / 4 + 255) / 256); if (rg > sm_count() * 8) rg = sm_count() * 8;
        launch_behind(reduce_partials_kernel, dim3((unsigned)rg), 256, 0, st, launch_overlaps(st), A.part, p.ks, mn, n_rows, y, DT_F32, bias, accumulate);
        note_launch();
    }
    return check_launch();
}

}  // namespace lowbit
