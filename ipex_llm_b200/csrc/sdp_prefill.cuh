// sdp_prefill.cuh -- included by kvcache.cu (inside namespace lowbit::{anonymous}, after sdp_mma.cuh).
// Attention of MANY query tokens over the e5m2 cache -- xe_addons.sdp_fp8_causal / sdp_fp8_non_causal of the reference
// (models/common.py:264-286: the prefill, where key.dtype == uint8 because DynamicFp8Cache.update returned the cache).
//
// fp16 / bf16 queries, head_dim 128, both products on the 5th-generation tensor cores.  One CTA = NT tiles of 128 query rows of one
// (sequence, query head), walking the keys in tiles of 128:
//   S_t = Q_t . K^T   tcgen05.mma M = 128, N = 128, K = 16, both operands in shared memory, S in TMEM (lane = query row);
//   softmax           four warps per tile, one thread per row, P (two fp16 values each) back into TMEM over S;
//   O_t += P_t . V    A operand = P in TMEM, B operand = V as it lies in the cache (rows = keys: the MN-major descriptor).
// Warps 0 .. 4 NT - 1: softmax; the next four read the cache (16 bytes a thread, coalesced), expand e5m2 -> fp16 (one byte permute
// per pair) and write K and V into a ring of four 32 KB swizzled tiles; the last warp issues the MMAs and owns TMEM.
// With two tiles a CTA their softmax and MMAs alternate: P_t . V, then Q_t . K of the next keys, of one tile run while the other is in
// its softmax, and every key tile is expanded once for 256 rows.  P lies over S, so a tile's next Q . K waits for its P . V (a commit,
// not the issue order); P . V of the first 64 keys of a tile starts while the softmax works on the others.
// P is hi + lo, both fp16, and both multiply V: with one fp16 value the result carried the rounding of every probability, where the
// kernel before this one (64 rows a CTA, mma.sync) rounded to fp16 too, but relative to a maximum that followed the keys 32 at a time,
// so that the largest of them stayed exact.  Error against 64 bits of fp32 results, scale 128^-1/2 / 1.0 (2000 tokens): before 1.5e-4 /
// 3.3e-5; one value with this kernel's lagging reference 1.6e-4 / 5.0e-5; the exact maximum as reference, O rescaled with nearly every
// key tile, 1.5e-4 / 3.5e-5; hi + lo 1.1e-6 / 0.9e-6.
// What bounds it: the chain Q.K -> softmax -> P.V of one tile, beside 3072 clocks of MMAs and 2048 of ex2 (16 a clock) per 128 keys and
// 256 rows (2000 tokens: tensor pipe 46 % busy, XU 31 %, issue slots 39 %).  4000 causal tokens, 32 heads over 8, the call: 609 us
// before, 160 with one value, 176 with one value and the exact maximum, 195 so: 672 TFLOP/s, each product counted once (6000 tokens:
// 418 while P . V waited for a tile's 128 keys, 392 now).
// Causal: query token s (0-based among the S new ones) sees keys <= L - S + s; key tiles beyond a tile's last row are skipped.  An
// additive mask [B][1|Hq][S][L] is honoured.  A value row that is not finite reaches the rows of its key tile that do not see it, as 0
// times it.  Softmax and accumulation in 32 bits; Q enters the MMAs as fp16.  P is kept relative to a reference 2^8 below fp16's
// comfortable range (values up to 2^14), and the reference follows the row's maximum only when that grew by more than 2^6: O is then
// rescaled in TMEM, which is rarely.

constexpr int SP_ROWS = 128, SP_KEYS = 128, SP_SLOTS = 4;
constexpr int SP_TILE = 128 * 256;                                    // 128 rows x 128 fp16, as two swizzled halves of 64 columns
constexpr int SP_BARS = 256;
__host__ __device__ constexpr int sp_smem(int nt) { return 1024 + (nt + SP_SLOTS) * SP_TILE + SP_BARS; }
constexpr int sp_threads(int nt) { return 32 * (4 * nt + 5); }

__device__ __forceinline__ void sp_tmem_ld32(uint32_t taddr, float* v) {
    uint32_t* r = reinterpret_cast<uint32_t*>(v);
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}
__device__ __forceinline__ void sp_tmem_st32(uint32_t taddr, const uint32_t* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
          "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
          "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]) : "memory");
}
__device__ __forceinline__ void sp_umma_ts_w(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate, uint32_t leader) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(leader) : "memory");
}
// two probabilities as two fp16 values each, hi + lo
__device__ __forceinline__ void sp_split2(float a, float b, uint32_t& hi, uint32_t& lo) {
    asm("{\n\t.reg .b16 p, q, m;\n\t.reg .f32 x, y;\n\t"
        "cvt.rn.f16x2.f32 %0, %3, %2;\n\t"
        "mov.b32 {p, q}, %0;\n\t"
        "mov.b16 m, 0xbc00;\n\t"
        "fma.rn.f32.f16 x, p, m, %2;\n\t"
        "fma.rn.f32.f16 y, q, m, %3;\n\t"
        "cvt.rn.f16x2.f32 %1, y, x;\n\t}" : "=&r"(hi), "=r"(lo) : "f"(a), "f"(b));
}
__device__ __forceinline__ void sp_sts128(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}

template <int NT, bool MASK>
__global__ void __launch_bounds__(sp_threads(NT), 1)
sdp_fp8_prompt_kernel(const SdpArgs A, int n_qt) {
    using namespace gemmtc;
    extern __shared__ uint8_t sp_raw[];
    const uint32_t base = (smem_u32(sp_raw) + 1023u) & ~1023u;
    const uint32_t qs = base, ring = base + NT * SP_TILE, bars = ring + SP_SLOTS * SP_TILE;
    auto kv_full = [&](int s) { return bars + s * 8; };
    auto kv_empty = [&](int s) { return bars + 32 + s * 8; };
    auto s_full = [&](int t) { return bars + 64 + t * 8; };
    auto p_full = [&](int t, int c) { return bars + 80 + (2 * t + c) * 8; };      // P of 64 keys
    auto pv_done = [&](int t) { return bars + 112 + t * 8; };
    const uint32_t drained = bars + 128;                               // every MMA that was issued is done
    const uint32_t tmem_slot = bars + 136;
    constexpr uint32_t TMEM_COLS = NT * 256;                           // S_t at 128 t, O_t behind all S
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int hq = blockIdx.x % A.Hq, b = blockIdx.x / A.Hq, hkv = hq / (A.Hq / A.Hkv);
    const int q0 = (n_qt - 1 - (int)blockIdx.y) * NT * SP_ROWS;        // the longest tiles of a causal prompt start first
    const int L = A.L, S = A.S;
    // key tiles that the rows of tile t need (0: no rows)
    auto tiles_of = [&](int t) {
        const int first = q0 + t * SP_ROWS;
        if (first >= S) return 0;
        const int last = min(first + SP_ROWS, S) - 1;
        const int end = A.causal ? min(L, L - S + last + 1) : L;
        return (end + SP_KEYS - 1) / SP_KEYS;
    };
    int nk = tiles_of(0);
    if (NT == 2) nk = max(nk, tiles_of(1));
    asm volatile("griddepcontrol.wait;" ::: "memory");

    // ---- before the barriers exist: the queries into their tiles, the first keys on their way
    if (warp < 4 * NT) {
        const int t = warp >> 2, r = 32 * (warp & 3) + lane, row = q0 + t * SP_ROWS + r;
        if (tiles_of(t) > 0) {
            // the row as fp16 into the swizzled operand tile (rows beyond S: zeros), in front of the block's first barrier
            const uint4* qrow = reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(A.q) + b * A.q_sb + hq * A.q_sh + (int64_t)row * A.q_ss);
            const uint32_t qd = qs + t * SP_TILE + r * 128;
#pragma unroll 8
            for (int c = 0; c < 16; c++) {
                uint4 w = make_uint4(0u, 0u, 0u, 0u);
                if (row < S) {
                    w = qrow[c];
                    if (A.q_dtype != DT_F16) {
                        uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            const __half2 h = __floats2half2_rn(__uint_as_float(u[i] << 16), __uint_as_float(u[i] & 0xffff0000u));
                            u[i] = *reinterpret_cast<const uint32_t*>(&h);
                        }
                        w = make_uint4(u[0], u[1], u[2], u[3]);
                    }
                }
                sp_sts128(qd + (c >> 3) * (SP_TILE / 2) + (((c & 7) ^ (r & 7)) << 4), w.x, w.y, w.z, w.w);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
    }
    const int tid = threadIdx.x - 128 * NT, piece = tid & 7, r0 = tid >> 3;       // loader warps: rows r0, r0 + 16, ... of a tile, piece of 16 columns
    uint4 w[8];
    auto fetch = [&](int item) {                                                  // item 2 j = keys of tile j, 2 j + 1 = its values
        const uint8_t* p = (item & 1) ? A.v + b * A.v_sb + hkv * A.v_sh + 16 * piece : A.k + b * A.k_sb + hkv * A.k_sh + 16 * piece;
        const int64_t ss = (item & 1) ? A.v_ss : A.k_ss;
        const int k0 = (item >> 1) * SP_KEYS + r0;
#pragma unroll
        for (int i = 0; i < 8; i++) w[i] = k0 + 16 * i < L ? *reinterpret_cast<const uint4*>(p + (k0 + 16 * i) * ss) : make_uint4(0u, 0u, 0u, 0u);
    };
    if (warp >= 4 * NT && warp < 4 * NT + 4 && nk > 0) fetch(0);

    if (threadIdx.x == 0) {
        for (int s = 0; s < SP_SLOTS; s++) { mbar_init(kv_full(s), 4); mbar_init(kv_empty(s), 1); }
        for (int t = 0; t < 2; t++) { mbar_init(s_full(t), 1); mbar_init(p_full(t, 0), 4); mbar_init(p_full(t, 1), 4); mbar_init(pv_done(t), 1); }
        mbar_init(drained, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 4 * NT + 4) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    uint32_t tmem;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(tmem_slot));
    // not before every block holds its columns: a dependent that allocates in front of its wait must find nobody who still wants some
    asm volatile("griddepcontrol.launch_dependents;");

    const uint32_t leader = elect_leader();
    if (warp < 4 * NT) {
        // ================= softmax: thread = query row =================
        const int t = warp >> 2, quarter = warp & 3, r = 32 * quarter + lane, row = q0 + t * SP_ROWS + r;
        const int nkt = tiles_of(t);
        if (nkt > 0) {
            const uint32_t lanes = (uint32_t)(32 * quarter) << 16;
            const uint32_t st = tmem + lanes + t * 128, ot = tmem + lanes + (NT + t) * 128;
            const int n_vis = row >= S ? 0 : A.causal ? min(L, L - S + row + 1) : L;                    // keys the row sees
            const int plain_end = MASK ? -1 : A.causal ? min(L, L - S + q0 + t * SP_ROWS + 32 * quarter + 1) : L;   // keys below: visible to the whole warp
            const int64_t mbase = b * A.m_sb + hq * A.m_sh + (int64_t)row * A.m_ss;
            float m_ref = -CUDART_INF_F, sum = 0.0f;
            for (int j = 0; j < nkt; j++) {
                if (!mbar_wait_lim(s_full(t), (uint32_t)(j & 1), A.waits)) goto done;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const int k0 = j * SP_KEYS;
                const bool plain = k0 + SP_KEYS <= plain_end;
                const float mul = MASK ? 1.0f : A.scale_log2e;
                // the row's scores pass through the registers twice, 64 at a time (maximum, then exponentials): holding all 128 spilled
                auto load = [&](int c, float (&x)[64]) {
                    sp_tmem_ld32(st + 64 * c, x);
                    sp_tmem_ld32(st + 64 * c + 32, x + 32);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (MASK) {
#pragma unroll
                        for (int i = 0; i < 64; i++) {
                            const int key = k0 + 64 * c + i;
                            x[i] = key < n_vis ? x[i] * A.scale_log2e + load_as_float(A.mask, A.mask_dtype, mbase + key) * 1.4426950408889634f : -CUDART_INF_F;
                        }
                    } else if (!plain) {
                        const int left = n_vis - k0 - 64 * c;
#pragma unroll
                        for (int i = 0; i < 64; i++) x[i] = i < left ? x[i] : -CUDART_INF_F;
                    }
                };
                float mx = -CUDART_INF_F;
#pragma unroll 1
                for (int c = 0; c < 2; c++) {
                    float x[64];
                    load(c, x);
                    float m0 = x[0], m1 = x[1], m2 = x[2], m3 = x[3];
#pragma unroll
                    for (int i = 4; i < 64; i += 4) { m0 = fmaxf(m0, x[i]); m1 = fmaxf(m1, x[i + 1]); m2 = fmaxf(m2, x[i + 2]); m3 = fmaxf(m3, x[i + 3]); }
                    mx = fmaxf(mx, fmaxf(fmaxf(m0, m1), fmaxf(m2, m3)));
                }
                mx *= mul;
                const bool grow = mx > m_ref + 6.0f;                                // -inf: any visible key
                if (__any_sync(0xffffffffu, grow)) {
                    const float m_new = grow ? mx : m_ref;
                    if (j > 0) {
                        // the P . V before this Q . K is done: O is at rest
                        const float corr = grow ? ex2_approx(m_ref - m_new) : 1.0f;
                        sum *= corr;
#pragma unroll 1
                        for (int c = 0; c < 128; c += 32) {
                            float o[32];
                            sp_tmem_ld32(ot + c, o);
                            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                            for (int i = 0; i < 32; i++) o[i] *= corr;
                            sp_tmem_st32(ot + c, reinterpret_cast<const uint32_t*>(o));
                        }
                    }
                    m_ref = m_new;
                }
                const float shift = 8.0f - (m_ref == -CUDART_INF_F ? 0.0f : m_ref);
                float a0 = 0.0f, a1 = 0.0f, a2 = 0.0f, a3 = 0.0f;
                // P of keys 64 c .. 64 c + 63 goes where their scores were: the high parts to the first 32 columns, the low parts to the others
#pragma unroll 1
                for (int c = 0; c < 2; c++) {
                    float x[64];
                    load(c, x);
                    uint32_t hi[32], lo[32];
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        const float p0 = ex2_approx(fmaf(x[2 * i], mul, shift)), p1 = ex2_approx(fmaf(x[2 * i + 1], mul, shift));
                        const float p2 = ex2_approx(fmaf(x[2 * i + 2], mul, shift)), p3 = ex2_approx(fmaf(x[2 * i + 3], mul, shift));
                        a0 += p0; a1 += p1; a2 += p2; a3 += p3;
                        sp_split2(p0, p1, hi[i], lo[i]);
                        sp_split2(p2, p3, hi[i + 1], lo[i + 1]);
                    }
                    sp_tmem_st32(st + 64 * c, hi);
                    sp_tmem_st32(st + 64 * c + 32, lo);
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(p_full(t, c));
                }
                sum += (a0 + a1) + (a2 + a3);
            }
            if (!mbar_wait_lim(pv_done(t), (uint32_t)((nkt - 1) & 1), A.waits)) goto done;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const float inv = sum > 0.0f ? 1.0f / sum : 0.0f;                       // a row with every key masked gives zeros
            const int64_t oi = (int64_t)b * A.o_sb + (int64_t)hq * A.o_sh + (int64_t)row * A.o_ss;
#pragma unroll 1
            for (int c = 0; c < 128; c += 32) {
                float o[32];
                sp_tmem_ld32(ot + c, o);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (row < S) {
                    if (A.out_dtype == DT_F32) {
                        float4* p = reinterpret_cast<float4*>((float*)A.out + oi + c);
#pragma unroll
                        for (int i = 0; i < 8; i++) p[i] = make_float4(o[4 * i] * inv, o[4 * i + 1] * inv, o[4 * i + 2] * inv, o[4 * i + 3] * inv);
                    } else {
                        uint4* p = reinterpret_cast<uint4*>((uint16_t*)A.out + oi + c);
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            uint32_t w[4];
#pragma unroll
                            for (int k = 0; k < 4; k++) {
                                const float x = o[8 * i + 2 * k] * inv, y = o[8 * i + 2 * k + 1] * inv;
                                if (A.out_dtype == DT_F16) { const __half2 v = __floats2half2_rn(x, y); w[k] = *reinterpret_cast<const uint32_t*>(&v); }
                                else { const __nv_bfloat162 v = __floats2bfloat162_rn(x, y); w[k] = *reinterpret_cast<const uint32_t*>(&v); }
                            }
                            p[i] = make_uint4(w[0], w[1], w[2], w[3]);
                        }
                    }
                }
                __syncwarp();
            }
        }
    } else if (warp < 4 * NT + 4) {
        // ================= the cache: expanded into the ring, item by item =================
        // a thread's 16 elements are two chunks of one row's half; lanes of the second half write them in the other order, so that a
        // quarter warp (one row) meets every bank once
        const int half = piece >> 2, c0 = 2 * (piece & 3) + half;
        const int items = A.waits.limit < 0 ? nk : 2 * nk;
        for (int item = 0; item < items; item++) {
            const int s = item % SP_SLOTS, round = item / SP_SLOTS;
            if (!mbar_wait_lim(kv_empty(s), (uint32_t)((round & 1) ^ 1), A.waits)) goto done;
            const uint32_t dst = ring + s * SP_TILE + half * (SP_TILE / 2);
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int r = r0 + 16 * i;
                const uint32_t lo0 = __byte_perm(w[i].x, 0u, 0x1404u), lo1 = __byte_perm(w[i].x, 0u, 0x3424u), lo2 = __byte_perm(w[i].y, 0u, 0x1404u),
                               lo3 = __byte_perm(w[i].y, 0u, 0x3424u), hi0 = __byte_perm(w[i].z, 0u, 0x1404u), hi1 = __byte_perm(w[i].z, 0u, 0x3424u),
                               hi2 = __byte_perm(w[i].w, 0u, 0x1404u), hi3 = __byte_perm(w[i].w, 0u, 0x3424u);
                const uint32_t a = dst + r * 128 + ((c0 ^ (r & 7)) << 4), z = dst + r * 128 + (((c0 ^ 1) ^ (r & 7)) << 4);
                if (half) { sp_sts128(a, hi0, hi1, hi2, hi3); sp_sts128(z, lo0, lo1, lo2, lo3); }
                else { sp_sts128(a, lo0, lo1, lo2, lo3); sp_sts128(z, hi0, hi1, hi2, hi3); }
            }
            if (item + 1 < 2 * nk) fetch(item + 1);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(kv_full(s));
        }
    } else {
        // ================= MMA issuer: the whole warp runs the loop, one elected lane issues =================
        // c F32, a / b fp16, N = 128, M = 128; S: both operands K-major; O: A in TMEM, B (values) MN-major (bit 16)
        const uint32_t id_s = (1u << 4) | ((128u >> 3) << 17) | ((128u >> 4) << 24), id_o = id_s | (1u << 16);
        const int nk0 = tiles_of(0), nk1 = NT == 2 ? tiles_of(1) : 0;
        auto scores = [&](int t, int j) {
            const uint64_t qd = make_desc(qs + t * SP_TILE), kd = make_desc(ring + ((2 * j) % SP_SLOTS) * SP_TILE);
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const uint64_t step = (uint64_t)(((k >> 2) * (SP_TILE / 2) + (k & 3) * 32) >> 4);
                umma_f16_w(tmem + t * 128, qd + step, kd + step, id_s, k > 0 ? 1u : 0u, leader);
            }
            umma_commit_w(s_full(t), leader);
        };
        auto values = [&](int t, int j, int c) {             // 64 keys
            // V tile: element (d, key) at half(d / 64), row key: LBO = the next 64 d, SBO = the next 8 keys; 16 keys a step
            const uint64_t vd = (make_desc(ring + ((2 * j + 1) % SP_SLOTS) * SP_TILE) & ~((uint64_t)0x3fff << 16)) | ((uint64_t)((SP_TILE / 2) >> 4) << 16);
#pragma unroll
            for (int k = 0; k < 4; k++)
#pragma unroll
                for (int lo = 1; lo >= 0; lo--)              // the small parts first
                    sp_umma_ts_w(tmem + (NT + t) * 128, tmem + t * 128 + c * 64 + lo * 32 + k * 8, vd + (uint64_t)(((4 * c + k) * 2048) >> 4), id_o,
                                 (j > 0 || c > 0 || k > 0 || lo == 0) ? 1u : 0u, leader);
        };
        if (nk > 0) {
            if (!mbar_wait_lim(kv_full(0), 0u, A.waits)) goto done;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int t = 0; t < NT; t++) {
                if ((t == 0 ? nk0 : nk1) == 0) continue;
                scores(t, 0);
            }
            umma_commit_w(kv_empty(0), leader);
        }
        for (int j = 0; j < nk; j++) {
            const int vi = 2 * j + 1, ki = 2 * j + 2;
            if (!mbar_wait_lim(kv_full(vi % SP_SLOTS), (uint32_t)((vi / SP_SLOTS) & 1), A.waits)) goto done;
            if (j + 1 < nk && !mbar_wait_lim(kv_full(ki % SP_SLOTS), (uint32_t)((ki / SP_SLOTS) & 1), A.waits)) goto done;
            const int last = NT == 2 && j < nk1 ? 1 : 0;
            for (int t = 0; t < NT; t++) {
                const int nkt = t == 0 ? nk0 : nk1;
                if (j >= nkt) continue;
                for (int c = 0; c < 2; c++) {
                    if (!mbar_wait_lim(p_full(t, c), (uint32_t)(j & 1), A.waits)) goto done;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    values(t, j, c);
                }
                umma_commit_w(pv_done(t), leader);
                if (t == last) umma_commit_w(kv_empty(vi % SP_SLOTS), leader);
                if (j + 1 < nkt) {
                    if (!mbar_wait_lim(pv_done(t), (uint32_t)(j & 1), A.waits)) goto done;         // S and P share their columns
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    scores(t, j + 1);
                }
            }
            if (j + 1 < nk) umma_commit_w(kv_empty(ki % SP_SLOTS), leader);
        }
    }
done:
    __syncwarp();
    if (warp == 4 * NT + 4) {
        // behind a wait that ran out MMAs may still be under way: nobody leaves their memory
        umma_commit_w(drained, leader);
        mbar_wait_lim(drained, 0u, Waits{A.waits.word, kWaitCycles});
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 4 * NT + 4) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    }
}

template <int NT, bool MASK> int sdp_prompt_launch_nt(const SdpArgs& A, cudaStream_t st) {
    static bool configured_dev[64] = {};                                  // the attribute is per device context
    int dev = 0;
    cudaGetDevice(&dev);
    if (!configured_dev[dev & 63]) {
        cudaFuncSetAttribute(sdp_fp8_prompt_kernel<NT, MASK>, cudaFuncAttributeMaxDynamicSharedMemorySize, sp_smem(NT));
        configured_dev[dev & 63] = true;
    }
    const int n_qt = (A.S + NT * SP_ROWS - 1) / (NT * SP_ROWS);
    launch_behind(sdp_fp8_prompt_kernel<NT, MASK>, dim3((unsigned)(A.B * A.Hq), (unsigned)n_qt), sp_threads(NT), sp_smem(NT), st, launch_overlaps(st), A, n_qt);
    note_launch();
    return check_launch();
}
// 256 rows a CTA share every key tile's expansion, 128 spread a short prompt over twice the SMs: two tiles once they fill the chip
int sdp_prompt_launch(SdpArgs A, cudaStream_t st) {
    if (const int rc = make_waits(&A.waits, gemmtc::kWaitCycles)) return rc;
    const int64_t two = (int64_t)A.B * A.Hq * ((A.S + 2 * SP_ROWS - 1) / (2 * SP_ROWS));
    if (A.mask) return two >= sm_count() ? sdp_prompt_launch_nt<2, true>(A, st) : sdp_prompt_launch_nt<1, true>(A, st);
    return two >= sm_count() ? sdp_prompt_launch_nt<2, false>(A, st) : sdp_prompt_launch_nt<1, false>(A, st);
}
