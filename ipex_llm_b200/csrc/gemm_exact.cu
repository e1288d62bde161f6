// gemm_exact.cu -- the fp32 matmul of a prompt on the 5th-generation tensor cores: y[M][N] (+)= x[M][K] . dequant(W[N][K])^T with 32-bit
// activations kept to 2^-24, the fp32-in / fp32-out contract of ggml_compute_forward_mul_mat_q_fp32 (reference
// low_bit_linear.py:494-529), for more than 32 rows.
//
// The arithmetic is the exact GEMV's (gemv_kernel.cuh): the CODES (4-bit offsets, e4m3 / e5m2 / e3m2 values) are exact in bf16, an
// activation is the sum of three bf16 planes, so every product is exact in 32 bits; a 64-element block's sum leaves the tensor cores
// after 12 steps and is multiplied by the block's scale and added in 32-bit floats.  Formats whose value is not code x scale (asym_int4's
// minima, nf4's table) stay on the GEMV.
//
// Layout of the work as in gemm_pair.cu: a cluster of two CTAs computes 256 features x up to 64 tokens with tcgen05.mma.cta_group::2, codes
// expanded to bf16 = A operand, the token planes = B, each CTA staging half of the tokens (three boxes of 32 rows per k-block).  Every
// k-block has a TMEM buffer of its own (eight of 64 columns); eight epilogue warps drain it: lane = feature, so a block's scale is one
// value per lane, and a thread keeps 32 tokens' sums in registers over the unit's K range.
//   warp 0 token planes (TMA), warp 1 MMAs / relay, warp 2 packed weights, warp 3 TMEM, warps 4-15 three expansion groups, 16-23 epilogue.
// What it replaces ran chunks of 32 rows on the GEMV's mma.sync path, every chunk reading the weights again.  sym_int4, before -> now:
// 4096 x 4096 at 33 rows 33.8 -> 17.4 us, 64 rows 50.4 -> 18.0, 200 rows 161 -> 37.7, 512 rows 400 -> 67.6; 11008 x 4096 at 512 rows
// 938 -> 153; 1024 x 1024 at 33 rows 18.2 -> 12.4 (the smallest shape that reaches this kernel also gains).  Error against 64 bits,
// relative to the result's norm: 4.8e-7 -> 1.5e-7 (sym_int4, 4096 x 4096), 2.5e-7 -> 1.6e-7 (e4m3).  A k-block costs 0.28 us at one unit
// per pair: bound by the latency of staging and expansion, as in gemm_pair.cu; 12 MMA steps instead of 4 fit under it.
#include "tc_pair.cuh"

namespace lowbit {
namespace gemmtc {

constexpr int kExThreads = 32 * 24, kExTok = 64, kExBufs = 8, kExGroups = 3;
constexpr int kExDeq0 = 4, kExEpi0 = 16;

template <int QT> struct ExSmem {
    static constexpr int kGroup = PackedBlock<QT>::kGroup, kPacked = 2 * kGroup;
    static constexpr int kA = kExGroups, kP = 2 * kExGroups, kX = 6;
    static constexpr int kXSlot = 3 * 4096;                            // three planes x 32 rows x 128 bytes
    static constexpr int kTotal = 1024 + 512 + kA * kTileBytesAB + kP * kPacked + kX * kXSlot;
    static_assert(kTotal <= 232448, "shared memory");
    static_assert((3 * kX + 2 * kP + 2 * kA + 2 * kExBufs + 1) * 8 + 8 <= 512, "barrier region");
};

struct ExactArgs {
    const uint8_t* w;
    TiledGeom G;
    int M, tt, n_fp, ksplit;
    float* y; const float* bias; int accumulate;
    float* part;
    Waits waits;
};

template <int QT>
__global__ void __launch_bounds__(kExThreads, 1)
exact_kernel(const __grid_constant__ CUtensorMap xmap, const ExactArgs A) {
    using E = Expand<QT>;
    using SM = ExSmem<QT>;
    constexpr int KX = SM::kX, KP = SM::kP, KA = SM::kA;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t xring = base, aring = base + KX * SM::kXSlot, pring = aring + KA * kTileBytesAB, bars = pring + KP * SM::kPacked;
    auto x_full = [&](int s) { return bars + s * 8; };
    auto x_empty = [&](int s) { return bars + (KX + s) * 8; };
    auto xp_full = [&](int s) { return bars + (2 * KX + s) * 8; };                     // CTA 0: the other half has landed
    auto p_full = [&](int s) { return bars + (3 * KX + s) * 8; };
    auto p_empty = [&](int s) { return bars + (3 * KX + KP + s) * 8; };
    auto a_full = [&](int s) { return bars + (3 * KX + 2 * KP + s) * 8; };             // CTA 0: both CTAs' tiles are expanded
    auto a_empty = [&](int s) { return bars + (3 * KX + 2 * KP + KA + s) * 8; };
    auto t_full = [&](int b) { return bars + (3 * KX + 2 * KP + 2 * KA + b) * 8; };
    auto t_empty = [&](int b) { return bars + (3 * KX + 2 * KP + 2 * KA + kExBufs + b) * 8; };   // CTA 0: both epilogues have read it
    const uint32_t drained = bars + (3 * KX + 2 * KP + 2 * KA + 2 * kExBufs) * 8;      // every MMA that was issued is done
    const uint32_t tmem_slot = drained + 8;
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31, rank = (int)(blockIdx.x & 1);
    const int nb = (int)A.G.nb;
    if (threadIdx.x == 0) {
        for (int s = 0; s < KX; s++) { mbar_init(x_full(s), 1); mbar_init(x_empty(s), 1); mbar_init(xp_full(s), 1); }
        for (int s = 0; s < KP; s++) { mbar_init(p_full(s), 1); mbar_init(p_empty(s), 4); }
        for (int s = 0; s < KA; s++) { mbar_init(a_full(s), 8); mbar_init(a_empty(s), 1); }
        for (int b = 0; b < kExBufs; b++) { mbar_init(t_full(b), 1); mbar_init(t_empty(b), 16); }
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
        for (int unit = blockIdx.x >> 1; unit < n_units; unit += stride) {
            decode(unit, U);
            const int row0 = U.m0 + rank * (U.n_tok >> 1);
            for (int kb = U.kb0; kb < U.kb1; kb++) {
                if (!mbar_wait_lim(x_empty(s), (uint32_t)((round & 1) ^ 1), A.waits)) goto done;
                mbar_expect_tx_w(x_full(s), SM::kXSlot, leader);
                // rows of a plane beyond the last token belong to the next plane (or read zero): columns that nothing stores
                for (int p = 0; p < 3; p++) tma_load_2d_w(xring + s * SM::kXSlot + p * 4096, &xmap, kb * 64, p * A.M + row0, x_full(s), leader);
                if (++s == KX) { s = 0; round++; }
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            // ================= MMA issuer: 3 planes x 4 steps per k-block, into the k-block's own TMEM buffer =================
            int sx = 0, rx = 0, sa = 0, ra = 0, tb = 0, rt = 0;
            for (int unit = blockIdx.x >> 1; unit < n_units; unit += stride) {
                decode(unit, U);
                const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (((uint32_t)U.n_tok >> 3) << 17) | ((256u >> 4) << 24);
                for (int kb = U.kb0; kb < U.kb1; kb++) {
                    if (!mbar_wait_lim(t_empty(tb), (uint32_t)((rt & 1) ^ 1), A.waits)) goto done;
                    if (!mbar_wait_lim(x_full(sx), (uint32_t)(rx & 1), A.waits)) goto done;
                    if (!mbar_wait_lim(xp_full(sx), (uint32_t)(rx & 1), A.waits)) goto done;
                    if (!mbar_wait_lim(a_full(sa), (uint32_t)(ra & 1), A.waits)) goto done;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t ad = make_desc(aring + sa * kTileBytesAB), xd = make_desc(xring + sx * SM::kXSlot);
#pragma unroll
                    for (int p = 2; p >= 0; p--)             // the small planes first
#pragma unroll
                        for (int k4 = 0; k4 < 4; k4++)
                            umma2_f16_w(tmem_base + tb * kExTok, ad + (uint64_t)((k4 * 32) >> 4), xd + (uint64_t)((p * 4096 + k4 * 32) >> 4), idesc,
                                        (p < 2 || k4 > 0) ? 1u : 0u, leader);
                    umma2_commit_w(a_empty(sa), leader);
                    umma2_commit_w(x_empty(sx), leader);
                    umma2_commit_w(t_full(tb), leader);
                    if (++sx == KX) { sx = 0; rx++; }
                    if (++sa == KA) { sa = 0; ra++; }
                    if (++tb == kExBufs) { tb = 0; rt++; }
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
    } else if (warp >= kExDeq0 && warp < kExEpi0) {
        // ================= expansion: group (warp - 4) / 4 takes every third k-block =================
        const int grp = (warp - kExDeq0) >> 2, dw = (warp - kExDeq0) & 3, g = lane >> 2, t = lane & 3;
        const uint32_t row0 = aring + grp * kTileBytesAB + 4 * dw * 1024 + g * 128;        // rows interleaved by 16 as in gemm_pair.cu
        const __half2 one = __floats2half2_rn(1.0f, 1.0f), zero = __floats2half2_rn(0.0f, 0.0f);
        int it = 0, turn = 0, sp = 0, rp = 0, ra = 0;
        for (int unit = blockIdx.x >> 1; unit < n_units; unit += stride) {
            decode(unit, U);
            for (int kb = U.kb0; kb < U.kb1; kb++, it++, (++turn == kExGroups ? turn = 0 : 0), (++sp == KP ? (sp = 0, rp++) : 0)) {
                if (turn != grp) continue;
                // at its last k-block this group waited for the MMAs of k-block it - 6 = it - KP: the packed slot's earlier trips are over
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
                        E::run(cw[gi], k4, one, one, zero, zero, 0u, a);                  // the codes' values, exact in fp16 and in bf16
                        lo[gi][2 * k4] = h2_to_bf2(a[0]); lo[gi][2 * k4 + 1] = h2_to_bf2(a[2]);
                        hi[gi][2 * k4] = h2_to_bf2(a[1]); hi[gi][2 * k4 + 1] = h2_to_bf2(a[3]);
                    }
                if (!mbar_wait_lim(a_empty(grp), (uint32_t)((ra & 1) ^ 1), A.waits)) goto done;
                ra++;
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
                if (lane == 0) { mbar_arrive(p_empty(sp)); mbar_arrive_at(a_full(grp), 0); }      // behind the stores: the codes have been used
            }
        }
    } else if (warp >= kExEpi0) {
        // ================= epilogue: TMEM lanes 32 * (warp % 4) .., tokens 32 * part .. + 31 =================
        const int quarter = warp & 3, part = (warp - kExEpi0) >> 2, half = lane >> 4;
        const int64_t N = A.G.rows;
        int tb = 0, rt = 0;
        for (int unit = blockIdx.x >> 1; unit < n_units; unit += stride) {
            decode(unit, U);
            const int64_t f0 = (int64_t)U.ft * 128, n = f0 + 64 * half + 16 * quarter + (lane & 15);
            const bool valid = f0 < N;
            // the lane's scales: row 16 quarter + (lane & 15) of 64-row group 2 ft + half, one fp16 per k-block, 128 bytes apart
            const int64_t rg = valid ? 2 * U.ft + half : 0;
            const __half* sp = reinterpret_cast<const __half*>(A.w + A.G.off_s + (rg * nb) * 128) + (lane & 7) * 8 + quarter * 2 + ((lane >> 3) & 1);
            const int t0 = 32 * part;
            float acc[32];
#pragma unroll
            for (int i = 0; i < 32; i++) acc[i] = 0.0f;
            float next[4];
#pragma unroll
            for (int i = 0; i < 4; i++) next[i] = U.kb0 + i < U.kb1 ? __half2float(sp[(int64_t)(U.kb0 + i) * 64]) : 0.0f;
            for (int kb = U.kb0; kb < U.kb1; kb += 4) {
                float d[4];
#pragma unroll
                for (int i = 0; i < 4; i++) d[i] = next[i];
#pragma unroll
                for (int i = 0; i < 4; i++) next[i] = kb + 4 + i < U.kb1 ? __half2float(sp[(int64_t)(kb + 4 + i) * 64]) : 0.0f;
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    if (kb + i >= U.kb1) break;
                    if (!mbar_wait_lim(t_full(tb), (uint32_t)(rt & 1), A.waits)) goto done;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                    for (int c = 0; c < 32; c += 16) {
                        if (t0 + c >= U.rows) break;
                        float v[16];
                        tmem_ld16(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(tb * kExTok + t0 + c), v);
#pragma unroll
                        for (int j = 0; j < 16; j++) acc[c + j] = fmaf(d[i], v[j], acc[c + j]);
                    }
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive_at(t_empty(tb), 0);
                    if (++tb == kExBufs) { tb = 0; rt++; }
                }
            }
            if (valid && t0 < U.rows) {
                const int64_t at = (int64_t)(U.m0 + t0) * N + n;
                const float b = A.bias && A.ksplit == 1 ? A.bias[n] : 0.0f;
                float* const dst = A.ksplit > 1 ? A.part + (int64_t)U.ks * A.M * N + at : A.y + at;
#pragma unroll
                for (int c = 0; c < 32; c += 16) {
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

// fp32 activations -> three bf16 planes whose sum reproduces them to 2^-24, four elements a thread
__global__ void __launch_bounds__(256) split3_kernel(const float4* __restrict__ x, uint2* __restrict__ out, int64_t n4) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n4; i += (int64_t)gridDim.x * blockDim.x) {
        const float4 q = x[i];
        float r[4] = {q.x, q.y, q.z, q.w};
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

template <int QT> static int exact_launch_one(const CUtensorMap& map, const ExactArgs& A, int64_t units, cudaStream_t st) {
    constexpr int SMEM = ExSmem<QT>::kTotal;
    static int cached[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    int& clusters = cached[dev & 63];
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(sm_count() & ~1)); cfg.blockDim = dim3(kExThreads); cfg.dynamicSmemBytes = SMEM; cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    if (!clusters) {
        int c = 0;
        if (cudaFuncSetAttribute(exact_kernel<QT>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) != cudaSuccess) {
            cudaGetLastError();
            set_error(LB_ERR_CUDA, "the two-SM fp32 matmul cannot be configured on this device");
            return LB_ERR_CUDA;
        }
        if (cudaOccupancyMaxActiveClusters(&c, exact_kernel<QT>, &cfg) != cudaSuccess || c <= 0) { cudaGetLastError(); c = sm_count() / 2; }
        clusters = c;
    }
    cfg.gridDim = dim3(2u * (unsigned)(units < clusters ? units : clusters));
    cudaLaunchKernelEx(&cfg, exact_kernel<QT>, map, A);
    note_launch();
    return LB_OK;
}

// K splits: rounds of the resident clusters x k-blocks per unit at 0.33 us, + the partial sums' round trip and its launch
struct ExactPlan { int tt, ks; };
static ExactPlan exact_plan(int64_t n_rows, int64_t nb, int64_t m) {
    const int64_t clusters = sm_count() / 2, n_fp = (n_rows / 128 + 1) / 2, nt = (m + kExTok - 1) / kExTok;
    ExactPlan best = {(int)(((m + nt - 1) / nt + 15) & ~int64_t(15)), 1};
    double best_cost = 1e30;
    for (int64_t ks = 1; ks == 1 || (ks <= 8 && nb / ks >= 8); ks++) {
        const int64_t rounds = (n_fp * nt * ks + clusters - 1) / clusters;
        double cost = (double)rounds * ((double)((nb + ks - 1) / ks) * 0.33 + 1.0);
        if (ks > 1) cost += (double)ks * (double)m * (double)n_rows * 8.0 / 4.0e6 + 2.0;
        if (cost < best_cost - 1e-9) { best_cost = cost; best.ks = (int)ks; }
    }
    return best;
}
static size_t exact_planes_bytes(int64_t k, int64_t m) { return ((size_t)3 * m * k * 2 + 255) / 256 * 256; }
}  // namespace gemmtc

bool gemm_exact_supported(int qt, int64_t n_rows, int64_t k, int64_t m) {
    qt = canon_qtype(qt);
    return (qt == QT_SYM_INT4 || qt == QT_FP8_E4M3 || qt == QT_FP8_E5M2 || qt == QT_FP6) && gemm_tc_supported(qt, n_rows, k) && 3 * m < 0x7fffffff;
}
size_t gemm_exact_workspace_size(int64_t n_rows, int64_t k, int64_t m) {
    using namespace gemmtc;
    const ExactPlan p = exact_plan(n_rows, k / 64, m);
    return exact_planes_bytes(k, m) + (p.ks > 1 ? (size_t)p.ks * m * n_rows * sizeof(float) : 0);
}
int gemm_exact_launch(const void* w, int qt, int64_t n_rows, int64_t k, const void* x, int64_t m, void* y, const void* bias, int accumulate,
                      void* workspace, size_t workspace_bytes, cudaStream_t st) {
    using namespace gemmtc;
    qt = canon_qtype(qt);
    if (!gemm_exact_supported(qt, n_rows, k, m) || (((uintptr_t)x | (uintptr_t)w | (uintptr_t)workspace) & 15)) return LB_ERR_ARG;
    if (!workspace || workspace_bytes < gemm_exact_workspace_size(n_rows, k, m)) return LB_ERR_WORKSPACE;
    const int64_t n4 = m * k / 4;                                       // k is a multiple of 64
    int sg = (int)((n4 + 255) / 256); if (sg > sm_count() * 8) sg = sm_count() * 8;
    split3_kernel<<<sg, 256, 0, st>>>((const float4*)x, (uint2*)workspace, n4);
    note_launch();
    CUtensorMap map;
    if (const int rc = encode_rows(&map, workspace, true, 3 * m, k, 32)) return rc;
    const ExactPlan p = exact_plan(n_rows, k / 64, m);
    ExactArgs A = {};
    if (const int rc = make_waits(&A.waits, kWaitCycles)) return rc;
    A.w = (const uint8_t*)w; A.G = make_geom(n_rows, k, qt); A.M = (int)m; A.tt = p.tt; A.n_fp = (int)((n_rows / 128 + 1) / 2); A.ksplit = p.ks;
    A.y = (float*)y; A.bias = (const float*)bias; A.accumulate = accumulate; A.part = (float*)((char*)workspace + exact_planes_bytes(k, m));
    const int64_t units = (int64_t)A.n_fp * ((m + p.tt - 1) / p.tt) * p.ks;
    int rc = LB_ERR_ARG;
    switch (qt) {
        case QT_SYM_INT4: rc = exact_launch_one<QT_SYM_INT4>(map, A, units, st); break;
        case QT_FP8_E4M3: rc = exact_launch_one<QT_FP8_E4M3>(map, A, units, st); break;
        case QT_FP8_E5M2: rc = exact_launch_one<QT_FP8_E5M2>(map, A, units, st); break;
        case QT_FP6:      rc = exact_launch_one<QT_FP6>(map, A, units, st); break;
    }
    if (rc) return rc;
    if (p.ks > 1) {
        const int64_t mn = m * n_rows;
        int rg = (int)((mn / 4 + 255) / 256); if (rg > sm_count() * 8) rg = sm_count() * 8;
        reduce_partials_kernel<<<rg, 256, 0, st>>>(A.part, p.ks, mn, n_rows, y, DT_F32, bias, accumulate);
        note_launch();
    }
    return check_launch();
}

}  // namespace lowbit
