// Gated delta rule over a prompt, 32 tokens at a time.
//
//   M <- g M;  u = beta (v - M^T k);  M <- M + k u^T;  o = M^T q          (M [dim, vdim]; see recurrence.cu)
//
// With C_t = the product of the decays of the chunk's tokens up to t and M0 the state in front of the chunk, the chunk's updates solve a
// unit lower triangular system that does not contain M0:
//   u_t + beta_t sum_{j < t} (C_t / C_j) (k_j . k_t) u_j = beta_t (v_t - C_t M0^T k_t)          U = T (V - C o (K M0)),  T = (I + L)^-1 diag(beta)
//   o_t = C_t M0^T q_t + sum_{j <= t} (C_t / C_j) (k_j . q_t) u_j                                O = C o (Q M0) + A U
//   M   = C_last M0 + sum_j (C_last / C_j) k_j u_j^T
// T, A and the unit vectors need nothing from earlier chunks: delta_gram_kernel forms them for all chunks at once.  What stays serial
// is four small products per chunk and block of 16 value columns (delta_walk_kernel).  The token-by-token walk it replaces for
// prompts was bound by the chain of one token (two dot products, three exchanges, the update: 590 clocks): 2048 tokens, 16 heads,
// 128 x 128: 632 us.
// Everything is 32-bit; the quotients C_t / C_j come from sums of logarithms held, and raised, in double precision (a quotient of 32-bit
// products would carry the rounding of both).
#include "mixers_common.cuh"

namespace {

constexpr int DC = 32;                                  // tokens per chunk
constexpr int DV = 16;                                  // value columns per block of the walk
constexpr int DT = 256;                                 // threads of the first kernel, and of the walk beside its loading warp
constexpr int D_STAGES = 3;                             // chunks in shared memory
constexpr int D_TRI = DC + 4;                           // padded rows of T and A
constexpr int D_SIDE = 2 * DC * D_TRI + 2 * DC;         // per (head, chunk): T, A, C_t, C_last / C_t
// keys, then queries, as three bf16 planes whose sum is the 32-bit value to 2^-24; rows padded: eight of them start in eight different
// groups of four banks.  In floats
template <int D> __host__ __device__ constexpr int d_ld() { return D + 8; }
template <int D> __host__ __device__ constexpr int d_rows() { return 3 * 2 * DC * d_ld<D>() / 2; }

struct ChunkArgs {
    const void* conv; const void* proj; const void* A_log; const void* dt_bias;
    int B, S, kv_heads, heads, dim, vdim, ld_proj, off_b, off_a, slot0, n_chunks;
    int seq;                                            // tokens from one sequence to the next: S, or more when S is a portion of them
    const int32_t* pad;
    float* rows;                                        // [B][kv_heads][n_chunks][3 planes][2][DC][D + 8] bf16
    float* side;                                        // [B][heads][n_chunks][D_SIDE]
    float* state; float* o;
};

__device__ __forceinline__ int first_token(const ChunkArgs& a, int b) {
    const int f = a.pad ? a.pad[b] - a.slot0 : 0;
    return f < 0 ? 0 : f > a.S ? a.S : f;
}

// v = hi + mid + lo in bf16, two values at a time
__device__ __forceinline__ void split3(float a, float b, uint32_t (&out)[3]) {
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
        out[p] = *reinterpret_cast<const uint32_t*>(&h);
        a -= __low2float(h); b -= __high2float(h);
    }
}

// grid (chunks, key/value heads, batch)
template <typename T, int D>
__global__ void __launch_bounds__(DT) delta_gram_kernel(const ChunkArgs a) {
    constexpr int LD = D + 4;
    extern __shared__ __align__(16) float sh[];
    float* const ks = sh;                               // [DC][LD]
    float* const qs = ks + DC * LD;
    float* const kk = qs + DC * LD;                     // [DC][DC] k_i . k_j
    float* const qk = kk + DC * DC;                     // [DC][DC] q_i . k_j
    float* const tri = qk + DC * DC;                    // [8 warps][DC][DC] L of the warp's head
    const int c = blockIdx.x, g = blockIdx.y, b = blockIdx.z;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int t0 = first_token(a, b) + c * DC, nt = min(DC, a.S - t0);
    if (nt <= 0) return;
    const int ld = 2 * a.kv_heads * a.dim + a.heads * a.vdim;
    const double q_scale = 1.0 / sqrt((double)a.dim);
    // unit vectors, a warp per token
    for (int t = warp; t < DC; t += DT / 32) {
        const T* row = (const T*)a.conv + ((long)b * a.seq + t0 + (t < nt ? t : 0)) * ld;
        float kv[D / 32], qv[D / 32], sk = 0.0f, sq = 0.0f;
#pragma unroll
        for (int e = 0; e < D / 32; ++e) {
            const int i = lane + 32 * e;
            const bool ok = t < nt && i < a.dim;
            qv[e] = ok ? to_f(row[g * a.dim + i]) : 0.0f;
            kv[e] = ok ? to_f(row[(a.kv_heads + g) * a.dim + i]) : 0.0f;
            sq += qv[e] * qv[e]; sk += kv[e] * kv[e];
        }
        sq = warp_sum(sq); sk = warp_sum(sk);
        const float nq = (float)(q_scale / sqrt((double)sq + 1e-6)), nk = (float)(1.0 / sqrt((double)sk + 1e-6));
#pragma unroll
        for (int e = 0; e < D / 32; ++e) { ks[t * LD + lane + 32 * e] = kv[e] * nk; qs[t * LD + lane + 32 * e] = qv[e] * nq; }
    }
    __syncthreads();
    float* const rows = a.rows + (((long)b * a.kv_heads + g) * a.n_chunks + c) * d_rows<D>();
    for (int i = tid; i < 2 * DC * D / 2; i += DT) {
        const int row = i / (D / 2), d = 2 * (i % (D / 2));
        const float2 x = *reinterpret_cast<const float2*>(ks + row * LD + d);
        uint32_t pl[3];
        split3(x.x, x.y, pl);
#pragma unroll
        for (int p = 0; p < 3; ++p) reinterpret_cast<uint32_t*>(rows)[((p * 2 * DC + row) * d_ld<D>() + d) / 2] = pl[p];
    }
    // the two Gram matrices, 2 x 2 of each per thread
    {
        const int i0 = tid >> 4, j0 = tid & 15;
        // eight sums per dot product: what their rounding leaves sets the error of a chunk's outputs
        float x[2][2][8] = {}, y[2][2][8] = {};
#pragma unroll 1
        for (int d = 0; d < D; d += 8) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                float4 ki[2], qi[2], kj[2];
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    ki[r] = *reinterpret_cast<const float4*>(ks + (i0 + 16 * r) * LD + d + 4 * q);
                    qi[r] = *reinterpret_cast<const float4*>(qs + (i0 + 16 * r) * LD + d + 4 * q);
                    kj[r] = *reinterpret_cast<const float4*>(ks + (j0 + 16 * r) * LD + d + 4 * q);
                }
#pragma unroll
                for (int r = 0; r < 2; ++r)
#pragma unroll
                    for (int s = 0; s < 2; ++s) {
                        x[r][s][4 * q] += ki[r].x * kj[s].x; x[r][s][4 * q + 1] += ki[r].y * kj[s].y; x[r][s][4 * q + 2] += ki[r].z * kj[s].z; x[r][s][4 * q + 3] += ki[r].w * kj[s].w;
                        y[r][s][4 * q] += qi[r].x * kj[s].x; y[r][s][4 * q + 1] += qi[r].y * kj[s].y; y[r][s][4 * q + 2] += qi[r].z * kj[s].z; y[r][s][4 * q + 3] += qi[r].w * kj[s].w;
                    }
            }
        }
        auto sum8 = [](const float (&v)[8]) { return ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7])); };
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int s = 0; s < 2; ++s) { kk[(i0 + 16 * r) * DC + j0 + 16 * s] = sum8(x[r][s]); qk[(i0 + 16 * r) * DC + j0 + 16 * s] = sum8(y[r][s]); }
    }
    __syncthreads();
    // a warp per head of the group: lane = token for the gates, then lane = column of the inverse
    const int n_rep = a.heads / a.kv_heads;
    float* const L = tri + warp * DC * DC;
    for (int hi = warp; hi < n_rep; hi += DT / 32) {
        const int h = g * n_rep + hi;
        const T* pr = (const T*)a.proj + ((long)b * a.seq + t0 + (lane < nt ? lane : 0)) * a.ld_proj;
        // the gates in double: a decay's error counts as often as there are tokens behind it
        const double z = (double)to_f(pr[a.off_a + h]) + (double)to_f(((const T*)a.dt_bias)[h]);
        double lg = -exp((double)to_f(((const T*)a.A_log)[h])) * (z > 20.0 ? z : log1p(exp(z)));
        lg = lg < -200.0 ? -200.0 : lg;                 // e^-200 is zero in 32 bits; an infinite logarithm would not cancel in a quotient
        const float beta = lane < nt ? (float)(1.0 / (1.0 + exp(-(double)to_f(pr[a.off_b + h])))) : 0.0f;
        double cum = lane < nt ? lg : 0.0;
#pragma unroll
        for (int m = 1; m < 32; m <<= 1) { const double v = __shfl_up_sync(0xffffffffu, cum, m); if (lane >= m) cum += v; }
        const double end = __shfl_sync(0xffffffffu, cum, 31);
        float* const side = a.side + (((long)b * a.heads + h) * a.n_chunks + c) * D_SIDE;
        for (int i = 0; i < DC; ++i) {                  // row i, lane = column j
            const double ci = __shfl_sync(0xffffffffu, cum, i);
            const float bi = __shfl_sync(0xffffffffu, beta, i);
            const float ratio = lane <= i ? (float)exp(ci - cum) : 0.0f;
            L[i * DC + lane] = lane < i ? bi * ratio * kk[i * DC + lane] : 0.0f;
            side[(DC + i) * D_TRI + lane] = lane <= i ? ratio * qk[i * DC + lane] : 0.0f;
        }
        side[2 * DC * D_TRI + lane] = (float)exp(cum);
        side[2 * DC * D_TRI + DC + lane] = (float)exp(end - cum);
        __syncwarp();
        float x[DC];
#pragma unroll
        for (int i = 0; i < DC; ++i) {
            float s0 = i == lane ? 1.0f : 0.0f, s1 = 0.0f;
#pragma unroll
            for (int m = 0; m < i; ++m) { if (m & 1) s1 -= L[i * DC + m] * x[m]; else s0 -= L[i * DC + m] * x[m]; }
            x[i] = s0 + s1;
            side[i * D_TRI + lane] = x[i] * beta;
        }
        __syncwarp();
    }
}

__device__ __forceinline__ void cp16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t at) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], uint32_t at) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// the six products of two three-plane numbers above 2^-25 of the largest, smallest first
__device__ constexpr int kPlaneA[6] = {2, 0, 1, 1, 0, 0}, kPlaneB[6] = {0, 2, 1, 0, 1, 0};

// row 4 warp + r of a lower triangular matrix times two columns: later tokens are left out, not multiplied by zero (an infinity or a NaN
// among them stays theirs); four sums each
__device__ __forceinline__ float2 lower_row(const float* row, const float* y, int warp, int r) {
    float s[2][4] = {};
#pragma unroll 2
    for (int j = 0; j < 4 * warp; j += 4) {
        const float4 x = *reinterpret_cast<const float4*>(row + j);
        const float f[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float2 v = *reinterpret_cast<const float2*>(y + (j + q) * DV);
            s[0][q] += f[q] * v.x; s[1][q] += f[q] * v.y;
        }
    }
    const float4 x = *reinterpret_cast<const float4*>(row + 4 * warp);
    const float f[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float2 v = *reinterpret_cast<const float2*>(y + (4 * warp + q) * DV);
        if (q <= r) { s[0][q] += f[q] * v.x; s[1][q] += f[q] * v.y; }
    }
    return make_float2((s[0][0] + s[0][1]) + (s[0][2] + s[0][3]), (s[1][0] + s[1][1]) + (s[1][2] + s[1][3]));
}

// grid (blocks of DV value columns, heads, batch); warps 0-7 compute, warp 8 brings the chunks in.
// The two large products (K M0 / Q M0 of 64 rows, and the state's update) bound the walk: from shared memory every operand of a 32-bit
// fma costs its 4 bytes of the 128 that reach the registers per clock, 4500 of a chunk's 6900 clocks with tiles of 8 x 4 and 4 x 2 per
// lane.  They go to mma.sync as six products of bf16 planes (each exact, sums in 32 bits; see kPlaneA).  The state stays in registers,
// transposed: a warp owns 16 of its rows, updated as the accumulators of mma tiles [16 columns x 8 rows], and those are, split into
// planes, the operand tiles of the next chunk's products, so between the two stands no barrier and no store.
// Measured, both kernels, 2048 tokens, 16 heads, 128 x 128: 245 us when all warps staged the chunks (1130 clocks of 7300 a chunk) and
// multiplied with scalar fmas, 232 with a loading warp and two fmas per instruction, 159 so.  Error of the outputs against 64 bits,
// relative to their norm: 1.05e-7 (token by token 1.23e-7, norms and gates in 32 bits there).
template <typename T, int D>
__global__ void __launch_bounds__(DT + 32) delta_walk_kernel(const ChunkArgs a) {
    constexpr int LD = d_ld<D>(), STAGE = d_rows<D>() + D_SIDE, SL = D / 16, MT = 4 * SL / 8, UE = DC + 8;
    extern __shared__ __align__(16) float sh[];
    float* const part = sh + D_STAGES * STAGE;          // [SL slices][2 DC rows][DV] partial K M0, Q M0, halves of rows 2, 3, 6, 7, .. swapped
    float* const w = part + SL * 2 * DC * DV;           // [DC][DV] V - C o (K M0)
    float* const u = w + DC * DV;                       // [DC][DV]
    __nv_bfloat16* const ue = reinterpret_cast<__nv_bfloat16*>(u + DC * DV);             // [3 planes][DV][UE] U times C_last / C_t, transposed
    const int col0 = blockIdx.x * DV, h = blockIdx.y, b = blockIdx.z, g = h / (a.heads / a.kv_heads);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int first = first_token(a, b), n = (a.S - first + DC - 1) / DC;
    const int cols = min(DV, a.vdim - col0);

    if (warp == 8) {
        const float* const rows = a.rows + ((long)b * a.kv_heads + g) * a.n_chunks * d_rows<D>();
        const float* const side = a.side + ((long)b * a.heads + h) * a.n_chunks * D_SIDE;
        auto stage = [&](int c) {
            if (c < n) {
                float* const dst = sh + (c % D_STAGES) * STAGE;
                for (int i = lane; i < d_rows<D>() / 4; i += 32) cp16(dst + 4 * i, rows + (long)c * d_rows<D>() + 4 * i);
                for (int i = lane; i < D_SIDE / 4; i += 32) cp16(dst + d_rows<D>() + 4 * i, side + (long)c * D_SIDE + 4 * i);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        stage(0);
        stage(1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        for (int c = 0; c < n; ++c) {
            asm volatile("cp.async.wait_group 0;" ::: "memory");         // chunk c + 1
            __syncthreads();                            // the third barrier of chunk c: everybody has left chunk c - 1
            stage(c + 2);                               // into its slot
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        return;
    }

    const int ld = 2 * a.kv_heads * a.dim + a.heads * a.vdim, off_v = 2 * a.kv_heads * a.dim + h * a.vdim + col0;
    float* const ob = a.o + (((long)b * a.seq) * a.heads + h) * a.vdim + col0;
    const long o_ld = (long)a.heads * a.vdim;
    for (int i = tid; i < first * DV; i += DT) if (i % DV < cols) ob[(i / DV) * o_ld + i % DV] = 0.0f;

    // a slice of 16 rows of the state per warp (dim 64: per two warps, which take half of the products' rows each); the lane's part:
    // rows k0 + 8 kt + 2 tq, + 1 of columns gq (m[kt][0], [1]) and gq + 8 ([2], [3])
    const int slice = warp % SL, mt0 = (warp / SL) * MT, k0 = 16 * slice, gq = lane >> 2, tq = lane & 3;
    float* const stg = a.state + ((long)b * a.heads + h) * a.dim * a.vdim + col0;
    float m[2][4];
#pragma unroll
    for (int kt = 0; kt < 2; ++kt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int i = k0 + 8 * kt + 2 * tq + (e & 1), col = gq + 8 * (e >> 1);
            m[kt][e] = i < a.dim && col < cols ? stg[(long)i * a.vdim + col] : 0.0f;
        }
    const uint32_t row_at = (uint32_t)(((lane & 15) * LD + 8 * (lane >> 4)) * 2);        // the lane's row of a 16 x 16 tile of a plane
    const uint32_t ue_at = (uint32_t)__cvta_generic_to_shared(ue) + (uint32_t)(((lane & 15) * UE + 8 * (lane >> 4)) * 2);
    // the lane's two results of a chunk, in K M0, U and the outputs alike: token orow, columns op and op + 1
    const int orow = 4 * warp + (lane >> 3), op = 2 * (lane & 7), pp = op ^ (((orow >> 1) & 1) << 3);
    T v[2];
    auto values = [&](int c) {                          // as they are stored: a conversion here would wait for the loads
        const int t = first + c * DC + orow;
#pragma unroll
        for (int e = 0; e < 2; ++e)
            if (c < n && t < a.S && op + e < cols) v[e] = ((const T*)a.conv)[((long)b * a.seq + t) * ld + off_v + op + e];
    };
    v[0] = v[1] = from_f<T>(0.0f);
    values(0);
    __syncthreads();
    auto meet = [] { asm volatile("barrier.cta.sync 1, 256;" ::: "memory"); };
    for (int c = 0; c < n; ++c) {
        const float* const stage = sh + (c % D_STAGES) * STAGE;
        const uint32_t kq = (uint32_t)__cvta_generic_to_shared(stage) + row_at + (uint32_t)(k0 * 2);   // the slice's columns of keys, then queries
        const float* const tm = stage + d_rows<D>();
        const float* const am = tm + DC * D_TRI;
        const float* const cd = am + DC * D_TRI;        // C_t, then C_last / C_t
        // ---- K M0 and Q M0 over the slice's rows of M0
        {
            uint32_t bp[2][2][3];                       // [rows' half][columns' half][plane]
#pragma unroll
            for (int kt = 0; kt < 2; ++kt)
#pragma unroll
                for (int nt = 0; nt < 2; ++nt) split3(m[kt][2 * nt], m[kt][2 * nt + 1], bp[kt][nt]);
#pragma unroll
            for (int mi = 0; mi < MT; ++mi) {
                uint32_t ap[3][4];
#pragma unroll
                for (int p = 0; p < 3; ++p) ldsm4(ap[p], kq + (uint32_t)((p * 2 * DC + 16 * (mt0 + mi)) * LD * 2));
                float acc[2][4] = {};
#pragma unroll
                for (int q = 0; q < 6; ++q)
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt) mma_bf16(acc[nt], ap[kPlaneA[q]], bp[0][nt][kPlaneB[q]], bp[1][nt][kPlaneB[q]]);
                float* const to = part + (slice * 2 * DC + 16 * (mt0 + mi) + gq) * DV;
                const int swap = ((gq >> 1) & 1) << 3;
#pragma unroll
                for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                    for (int hf = 0; hf < 2; ++hf)
                        *reinterpret_cast<float2*>(to + 8 * hf * DV + ((8 * nt + 2 * tq) ^ swap)) = make_float2(acc[nt][2 * hf], acc[nt][2 * hf + 1]);
            }
        }
        meet();
        float2 read;                                    // Q M0, times C_t
        {
            float2 p[2][SL];
#pragma unroll
            for (int i = 0; i < SL; ++i) {
                p[0][i] = *reinterpret_cast<const float2*>(part + (i * 2 * DC + orow) * DV + pp);
                p[1][i] = *reinterpret_cast<const float2*>(part + (i * 2 * DC + DC + orow) * DV + pp);
            }
#pragma unroll
            for (int step = SL / 2; step > 0; step >>= 1)
#pragma unroll
                for (int i = 0; i < step; ++i)
#pragma unroll
                    for (int q = 0; q < 2; ++q) { p[q][i].x += p[q][i + step].x; p[q][i].y += p[q][i + step].y; }
            const float ct = cd[orow];
            const bool live = first + c * DC + orow < a.S;
            const float v0 = live && op < cols ? to_f(v[0]) : 0.0f, v1 = live && op + 1 < cols ? to_f(v[1]) : 0.0f;
            *reinterpret_cast<float2*>(w + orow * DV + op) = make_float2(v0 - ct * p[0][0].x, v1 - ct * p[0][0].y);
            read = make_float2(ct * p[1][0].x, ct * p[1][0].y);
        }
        values(c + 1);
        meet();
        // ---- U = T W
        {
            const float2 sum = lower_row(tm + orow * D_TRI, w + op, warp, lane >> 3);
            const float u0 = sum.x, u1 = sum.y, e = cd[DC + orow];
            *reinterpret_cast<float2*>(u + orow * DV + op) = make_float2(u0, u1);
            uint32_t pl[3];
            split3(e * u0, e * u1, pl);
#pragma unroll
            for (int p = 0; p < 3; ++p) {
                ue[(p * DV + op) * UE + orow] = __ushort_as_bfloat16((unsigned short)pl[p]);
                ue[(p * DV + op + 1) * UE + orow] = __ushort_as_bfloat16((unsigned short)(pl[p] >> 16));
            }
        }
        __syncthreads();
        // ---- the state: C_last M0 + K^T (U C_last / C_t)
        {
            float add[2][4] = {};
            uint32_t ap[2][3][4], bp[2][3][4];          // [tokens' half][plane]
#pragma unroll
            for (int th = 0; th < 2; ++th)
#pragma unroll
                for (int p = 0; p < 3; ++p) {
                    ldsm4(ap[th][p], ue_at + (uint32_t)((p * DV * UE + 16 * th) * 2));
                    ldsm4t(bp[th][p], kq + (uint32_t)((p * 2 * DC + 16 * th) * LD * 2));
                }
#pragma unroll
            for (int q = 0; q < 6; ++q)
#pragma unroll
                for (int th = 0; th < 2; ++th)
#pragma unroll
                    for (int kt = 0; kt < 2; ++kt) mma_bf16(add[kt], ap[th][kPlaneA[q]], bp[th][kPlaneB[q]][2 * kt], bp[th][kPlaneB[q]][2 * kt + 1]);
            const float decay = cd[DC - 1];
#pragma unroll
            for (int kt = 0; kt < 2; ++kt)
#pragma unroll
                for (int e = 0; e < 4; ++e) m[kt][e] = decay * m[kt][e] + add[kt][e];
        }
        // ---- outputs: C_t Q M0 + A U
        {
            const float2 sum = lower_row(am + orow * D_TRI, u + op, warp, lane >> 3);
            const int slot = first + c * DC + orow;
            if (slot < a.S) {
                if (op < cols) ob[slot * o_ld + op] = read.x + sum.x;
                if (op + 1 < cols) ob[slot * o_ld + op + 1] = read.y + sum.y;
            }
        }
    }
    if (mt0 == 0)
#pragma unroll
        for (int kt = 0; kt < 2; ++kt)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int i = k0 + 8 * kt + 2 * tq + (e & 1), col = gq + 8 * (e >> 1);
                if (i < a.dim && col < cols) stg[(long)i * a.vdim + col] = m[kt][e];
            }
}

template <typename T, int D> int launch_chunks(const ChunkArgs& a, cudaStream_t st) {
    constexpr int gram = (2 * DC * (D + 4) + 2 * DC * DC + (DT / 32) * DC * DC) * 4;
    constexpr int walk = (D_STAGES * (d_rows<D>() + D_SIDE) + (D / 16) * 2 * DC * DV + 2 * DC * DV) * 4 + 3 * DV * (DC + 8) * 2;
    static_assert(walk <= 232448, "shared memory");
    static bool configured_dev[64] = {};                // the attributes are per device context
    int dev = 0;
    cudaGetDevice(&dev);
    if (!configured_dev[dev & 63]) {
        cudaFuncSetAttribute(delta_gram_kernel<T, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, gram);
        cudaFuncSetAttribute(delta_walk_kernel<T, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, walk);
        configured_dev[dev & 63] = true;
    }
    delta_gram_kernel<T, D><<<dim3(a.n_chunks, a.kv_heads, a.B), DT, gram, st>>>(a);
    delta_walk_kernel<T, D><<<dim3((a.vdim + DV - 1) / DV, a.heads, a.B), DT + 32, walk, st>>>(a);
    return mixers_status();
}

}  // namespace

// Scratch of a call at most (or one chunk's, where that is more): 11 KB a token at 4 / 16 heads of 128, 22 KB at 8 / 32.  Longer prompts
// run in portions of whole chunks, the state carried through memory as between two calls
namespace {
constexpr long kDeltaScratch = 512l << 20;
long chunk_bytes(int B, int kv_heads, int heads, int dim) { return 4l * B * (kv_heads * (dim <= 64 ? d_rows<64>() : d_rows<128>()) + (long)heads * D_SIDE); }
// chunks of one portion: portions of equal length
long portion_chunks(int B, int S, int kv_heads, int heads, int dim) {
    const long n = ((long)S + DC - 1) / DC, fit = kDeltaScratch / chunk_bytes(B, kv_heads, heads, dim), most = fit > 1 ? fit : 1;
    const long portions = (n + most - 1) / most;
    return (n + portions - 1) / portions;
}
}  // namespace

extern "C" long mixers_gated_delta_chunks_workspace(int B, int S, int kv_heads, int heads, int dim) {
    if (B <= 0 || S <= 0 || dim <= 0 || dim > 128 || kv_heads <= 0 || kv_heads > 65535 || heads > 65535 || B > 65535) return -1;
    return portion_chunks(B, S, kv_heads, heads, dim) * chunk_bytes(B, kv_heads, heads, dim);
}

template <typename T> static int run_portions(ChunkArgs a, cudaStream_t st) {
    const int S = a.S, slot0 = a.slot0, step = DC * (int)portion_chunks(a.B, S, a.kv_heads, a.heads, a.dim);
    const long ld = 2 * a.kv_heads * a.dim + a.heads * a.vdim;
    const T *const conv = (const T*)a.conv, *const proj = (const T*)a.proj;
    float* const o = a.o;
    a.seq = S;
    a.side = a.rows + (long)a.B * a.kv_heads * (step / DC) * (a.dim <= 64 ? d_rows<64>() : d_rows<128>());
    for (long at = 0; at < S; at += step) {
        a.S = (int)(S - at < step ? S - at : step);
        a.n_chunks = (a.S + DC - 1) / DC;
        a.slot0 = slot0 + (int)at;
        a.conv = conv + at * ld; a.proj = proj + at * a.ld_proj; a.o = o + at * a.heads * a.vdim;
        if (const int rc = a.dim <= 64 ? launch_chunks<T, 64>(a, st) : launch_chunks<T, 128>(a, st)) return rc;
    }
    return 0;
}

extern "C" int mixers_gated_delta_chunks(int dtype, const void* conv, int B, int S, int kv_heads, int heads, int dim, int vdim, const void* proj, int ld,
                                         int off_b, int off_a, const void* A_log, const void* dt_bias, float* state, int slot0, const int32_t* pad, float* o,
                                         float* workspace, mixers_stream_t stream) {
    if (B <= 0 || S <= 0) return 0;
    if (kv_heads <= 0 || heads % kv_heads != 0 || mixers_gated_delta_chunks_workspace(B, S, kv_heads, heads, dim) < 0 || !workspace || ((uintptr_t)workspace & 15)) return (int)cudaErrorInvalidValue;
    ChunkArgs a = {};
    a.conv = conv; a.proj = proj; a.A_log = A_log; a.dt_bias = dt_bias;
    a.B = B; a.S = S; a.kv_heads = kv_heads; a.heads = heads; a.dim = dim; a.vdim = vdim; a.ld_proj = ld; a.off_b = off_b; a.off_a = off_a;
    a.slot0 = slot0; a.pad = pad; a.state = state; a.o = o; a.rows = workspace;
    MIXERS_DISPATCH(dtype, return run_portions<T>(a, (cudaStream_t)stream));
    return 0;
}
