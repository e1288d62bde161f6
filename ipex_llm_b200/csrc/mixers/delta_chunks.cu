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
// Everything is 32-bit, the quotients C_t / C_j come from sums of logarithms held in double precision (a quotient of 32-bit products
// would carry the rounding of both).
#include "mixers_common.cuh"

namespace {

constexpr int DC = 32;                                  // tokens per chunk
constexpr int DV = 16;                                  // value columns per block of the walk
constexpr int DT = 256;                                 // threads of both kernels
constexpr int D_SIDE = 2 * DC * DC + 2 * DC;            // per (head, chunk): T, A, C_t, C_last / C_t
template <int D> __host__ __device__ constexpr int d_row() { return D + 4; }        // padded: eight rows start in eight different banks
template <int D> __host__ __device__ constexpr int d_rows() { return 2 * DC * d_row<D>(); }       // keys, then queries

struct ChunkArgs {
    const void* conv; const void* proj; const void* A_log; const void* dt_bias;
    int B, S, kv_heads, heads, dim, vdim, ld_proj, off_b, off_a, slot0, n_chunks;
    const int32_t* pad;
    float* rows;                                        // [B][kv_heads][n_chunks][2][DC][D + 4]
    float* side;                                        // [B][heads][n_chunks][D_SIDE]
    float* state; float* o;
};

__device__ __forceinline__ int first_token(const ChunkArgs& a, int b) {
    const int f = a.pad ? a.pad[b] - a.slot0 : 0;
    return f < 0 ? 0 : f > a.S ? a.S : f;
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
    const float q_scale = rsqrtf((float)a.dim);
    // unit vectors, a warp per token
    for (int t = warp; t < DC; t += DT / 32) {
        const T* row = (const T*)a.conv + ((long)b * a.S + t0 + (t < nt ? t : 0)) * ld;
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
        const float nq = q_scale / sqrtf(sq + 1e-6f), nk = 1.0f / sqrtf(sk + 1e-6f);
#pragma unroll
        for (int e = 0; e < D / 32; ++e) { ks[t * LD + lane + 32 * e] = kv[e] * nk; qs[t * LD + lane + 32 * e] = qv[e] * nq; }
    }
    __syncthreads();
    float* const rows = a.rows + (((long)b * a.kv_heads + g) * a.n_chunks + c) * d_rows<D>();
    for (int i = tid; i < d_rows<D>() / 4; i += DT) reinterpret_cast<float4*>(rows)[i] = reinterpret_cast<const float4*>(ks)[i];
    // the two Gram matrices, 2 x 2 of each per thread
    {
        const int i0 = tid >> 4, j0 = tid & 15;
        float x[2][2] = {}, y[2][2] = {};
        for (int d = 0; d < D; d += 4) {
            float4 ki[2], qi[2], kj[2];
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                ki[r] = *reinterpret_cast<const float4*>(ks + (i0 + 16 * r) * LD + d);
                qi[r] = *reinterpret_cast<const float4*>(qs + (i0 + 16 * r) * LD + d);
                kj[r] = *reinterpret_cast<const float4*>(ks + (j0 + 16 * r) * LD + d);
            }
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int s = 0; s < 2; ++s) {
                    x[r][s] += ki[r].x * kj[s].x + ki[r].y * kj[s].y + ki[r].z * kj[s].z + ki[r].w * kj[s].w;
                    y[r][s] += qi[r].x * kj[s].x + qi[r].y * kj[s].y + qi[r].z * kj[s].z + qi[r].w * kj[s].w;
                }
        }
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int s = 0; s < 2; ++s) { kk[(i0 + 16 * r) * DC + j0 + 16 * s] = x[r][s]; qk[(i0 + 16 * r) * DC + j0 + 16 * s] = y[r][s]; }
    }
    __syncthreads();
    // a warp per head of the group: lane = token for the gates, then lane = column of the inverse
    const int n_rep = a.heads / a.kv_heads;
    float* const L = tri + warp * DC * DC;
    for (int hi = warp; hi < n_rep; hi += DT / 32) {
        const int h = g * n_rep + hi;
        const T* pr = (const T*)a.proj + ((long)b * a.S + t0 + (lane < nt ? lane : 0)) * a.ld_proj;
        const float neg_exp_a = -expf(to_f(((const T*)a.A_log)[h]));
        float lg = neg_exp_a * softplus_f(to_f(pr[a.off_a + h]) + to_f(((const T*)a.dt_bias)[h]));
        lg = lg < -200.0f ? -200.0f : lg;               // e^-200 is zero in 32 bits; an infinite logarithm would not cancel in a quotient
        const float beta = lane < nt ? sigmoid_f(to_f(pr[a.off_b + h])) : 0.0f;
        double cum = lane < nt ? (double)lg : 0.0;
#pragma unroll
        for (int m = 1; m < 32; m <<= 1) { const double v = __shfl_up_sync(0xffffffffu, cum, m); if (lane >= m) cum += v; }
        const double end = __shfl_sync(0xffffffffu, cum, 31);
        float* const side = a.side + (((long)b * a.heads + h) * a.n_chunks + c) * D_SIDE;
        for (int i = 0; i < DC; ++i) {                  // row i, lane = column j
            const double ci = __shfl_sync(0xffffffffu, cum, i);
            const float bi = __shfl_sync(0xffffffffu, beta, i);
            const float ratio = lane <= i ? expf((float)(ci - cum)) : 0.0f;
            L[i * DC + lane] = lane < i ? bi * ratio * kk[i * DC + lane] : 0.0f;
            side[DC * DC + i * DC + lane] = lane <= i ? ratio * qk[i * DC + lane] : 0.0f;
        }
        side[2 * DC * DC + lane] = expf((float)cum);
        side[2 * DC * DC + DC + lane] = expf((float)(end - cum));
        __syncwarp();
        float x[DC];
#pragma unroll
        for (int i = 0; i < DC; ++i) {
            float s0 = i == lane ? 1.0f : 0.0f, s1 = 0.0f;
#pragma unroll
            for (int m = 0; m < i; ++m) { if (m & 1) s1 -= L[i * DC + m] * x[m]; else s0 -= L[i * DC + m] * x[m]; }
            x[i] = s0 + s1;
            side[i * DC + lane] = x[i] * beta;
        }
        __syncwarp();
    }
}

__device__ __forceinline__ void cp16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// grid (blocks of DV value columns, heads, batch); the state block lives in registers between chunks and in shared memory for K M0 / Q M0
template <typename T, int D>
__global__ void __launch_bounds__(DT) delta_walk_kernel(const ChunkArgs a) {
    constexpr int LD = D + 4, STAGE = d_rows<D>() + D_SIDE, KS = D / 4, CPT = D / 64;
    extern __shared__ __align__(16) float sh[];
    float* const st = sh + 2 * STAGE;                   // [D][DV] state
    float* const part = st + D * DV;                    // [4][2 DC][DV] partial K M0, Q M0
    float* const w = part + 4 * 2 * DC * DV;            // [DC][DV] V - C o (K M0)
    float* const u = w + DC * DV;                       // [DC][DV]
    float* const ue = u + DC * DV;                      // [DC][DV] U times C_last / C_t
    const int col0 = blockIdx.x * DV, h = blockIdx.y, b = blockIdx.z, g = h / (a.heads / a.kv_heads);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int first = first_token(a, b), n = (a.S - first + DC - 1) / DC;
    const int ld = 2 * a.kv_heads * a.dim + a.heads * a.vdim, off_v = 2 * a.kv_heads * a.dim + h * a.vdim + col0;
    float* const ob = a.o + (((long)b * a.S) * a.heads + h) * a.vdim + col0;
    const long o_ld = (long)a.heads * a.vdim;
    const int cols = min(DV, a.vdim - col0);
    for (int i = tid; i < first * DV; i += DT) if (i % DV < cols) ob[(i / DV) * o_ld + i % DV] = 0.0f;

    // the thread's part of the state: rows 4 sr .. 4 sr + 3, columns sc .. sc + CPT - 1
    const int sr = tid / (DV / CPT), sc = tid % (DV / CPT) * CPT;
    float* const stg = a.state + ((long)b * a.heads + h) * a.dim * a.vdim + col0;
    float m[4][CPT];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int e = 0; e < CPT; ++e) {
            m[r][e] = 4 * sr + r < a.dim && sc + e < cols ? stg[(long)(4 * sr + r) * a.vdim + sc + e] : 0.0f;
            st[(4 * sr + r) * DV + sc + e] = m[r][e];
        }
    const float* const rows = a.rows + ((long)b * a.kv_heads + g) * a.n_chunks * d_rows<D>();
    const float* const side = a.side + ((long)b * a.heads + h) * a.n_chunks * D_SIDE;
    auto stage = [&](int c) {
        if (c < n) {
            float* const dst = sh + (c & 1) * STAGE;
            for (int i = tid; i < d_rows<D>() / 4; i += DT) cp16(dst + 4 * i, rows + (long)c * d_rows<D>() + 4 * i);
            for (int i = tid; i < D_SIDE / 4; i += DT) cp16(dst + d_rows<D>() + 4 * i, side + (long)c * D_SIDE + 4 * i);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // rows 0-31 of K M0 belong to threads 0-127 (row tid / 4, four columns), whose values they also fetch; rows of Q M0 to the others
    const int pr = tid >> 2, pc = 4 * (tid & 3);
    auto values = [&](int c, float (&v)[4]) {
        const int t = first + c * DC + pr;
#pragma unroll
        for (int e = 0; e < 4; ++e)
            v[e] = pr < DC && c < n && t < a.S && pc + e < cols ? to_f(((const T*)a.conv)[((long)b * a.S + t) * ld + off_v + pc + e]) : 0.0f;
    };
    float v[4];
    stage(0);
    values(0, v);
    for (int c = 0; c < n; ++c) {
        stage(c + 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();                                // chunk c is staged, the state of chunk c - 1 is in place
        const float* const kq = sh + (c & 1) * STAGE;   // keys, then queries
        const float* const tm = kq + d_rows<D>();
        const float* const am = tm + DC * DC;
        const float* const cd = am + DC * DC;           // C_t, then C_last / C_t
        // ---- K M0 and Q M0: a quarter of the rows of M0 per pair of warps, 4 x 4 outputs a thread
        {
            const int rg = (lane >> 2) + 8 * (warp & 1), cg = 4 * (lane & 3), k0 = (warp >> 1) * KS;
            float acc[4][4] = {};
#pragma unroll 2
            for (int k = k0; k < k0 + KS; k += 4) {
                float4 x[4], y[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) { x[i] = *reinterpret_cast<const float4*>(kq + (rg + 16 * i) * LD + k); y[i] = *reinterpret_cast<const float4*>(st + (k + i) * DV + cg); }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    acc[i][0] += x[i].x * y[0].x + x[i].y * y[1].x + x[i].z * y[2].x + x[i].w * y[3].x;
                    acc[i][1] += x[i].x * y[0].y + x[i].y * y[1].y + x[i].z * y[2].y + x[i].w * y[3].y;
                    acc[i][2] += x[i].x * y[0].z + x[i].y * y[1].z + x[i].z * y[2].z + x[i].w * y[3].z;
                    acc[i][3] += x[i].x * y[0].w + x[i].y * y[1].w + x[i].z * y[2].w + x[i].w * y[3].w;
                }
            }
            float* const p = part + (warp >> 1) * (2 * DC * DV);
#pragma unroll
            for (int i = 0; i < 4; ++i) *reinterpret_cast<float4*>(p + (rg + 16 * i) * DV + cg) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        }
        __syncthreads();
        float read[4];                                  // this thread's four sums, times C_t
        {
            const float4 p0 = *reinterpret_cast<const float4*>(part + pr * DV + pc), p1 = *reinterpret_cast<const float4*>(part + (2 * DC + pr) * DV + pc),
                         p2 = *reinterpret_cast<const float4*>(part + (4 * DC + pr) * DV + pc), p3 = *reinterpret_cast<const float4*>(part + (6 * DC + pr) * DV + pc);
            const float ct = cd[pr & (DC - 1)];
            read[0] = ct * ((p0.x + p1.x) + (p2.x + p3.x)); read[1] = ct * ((p0.y + p1.y) + (p2.y + p3.y));
            read[2] = ct * ((p0.z + p1.z) + (p2.z + p3.z)); read[3] = ct * ((p0.w + p1.w) + (p2.w + p3.w));
            if (pr < DC) *reinterpret_cast<float4*>(w + pr * DV + pc) = make_float4(v[0] - read[0], v[1] - read[1], v[2] - read[2], v[3] - read[3]);
        }
        values(c + 1, v);
        __syncthreads();
        // ---- U = T W: one row, two columns a thread
        {
            const int t = tid >> 3, cc = 2 * (tid & 7);
            float a0 = 0.0f, a1 = 0.0f, b0 = 0.0f, b1 = 0.0f;
#pragma unroll
            for (int j = 0; j < DC; j += 4) {
                const float4 x = *reinterpret_cast<const float4*>(tm + t * DC + j);
                const float2 y0 = *reinterpret_cast<const float2*>(w + j * DV + cc), y1 = *reinterpret_cast<const float2*>(w + (j + 1) * DV + cc),
                             y2 = *reinterpret_cast<const float2*>(w + (j + 2) * DV + cc), y3 = *reinterpret_cast<const float2*>(w + (j + 3) * DV + cc);
                a0 += x.x * y0.x + x.z * y2.x; a1 += x.x * y0.y + x.z * y2.y;
                b0 += x.y * y1.x + x.w * y3.x; b1 += x.y * y1.y + x.w * y3.y;
            }
            const float u0 = a0 + b0, u1 = a1 + b1, e = cd[DC + t];
            *reinterpret_cast<float2*>(u + t * DV + cc) = make_float2(u0, u1);
            *reinterpret_cast<float2*>(ue + t * DV + cc) = make_float2(e * u0, e * u1);
        }
        __syncthreads();
        // ---- the state: C_last M0 + K^T (U C_last / C_t)
        {
            const float decay = cd[DC - 1];
            float add[4][CPT] = {};
#pragma unroll 4
            for (int t = 0; t < DC; ++t) {
                const float4 x = *reinterpret_cast<const float4*>(kq + t * LD + 4 * sr);
                const float xr[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                for (int e = 0; e < CPT; ++e) {
                    const float y = ue[t * DV + sc + e];
#pragma unroll
                    for (int r = 0; r < 4; ++r) add[r][e] += xr[r] * y;
                }
            }
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int e = 0; e < CPT; ++e) { m[r][e] = decay * m[r][e] + add[r][e]; st[(4 * sr + r) * DV + sc + e] = m[r][e]; }
        }
        // ---- outputs: C_t Q M0 + A U
        if (pr >= DC) {
            const int t = pr - DC, slot = first + c * DC + t;
            float4 s = make_float4(read[0], read[1], read[2], read[3]);
#pragma unroll 8
            for (int j = 0; j < DC; ++j) {
                const float x = am[t * DC + j];
                const float4 y = *reinterpret_cast<const float4*>(u + j * DV + pc);
                s.x += x * y.x; s.y += x * y.y; s.z += x * y.z; s.w += x * y.w;
            }
            if (slot < a.S) {
                float* const p = ob + slot * o_ld + pc;
                const float r[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) if (pc + e < cols) p[e] = r[e];
            }
        }
        __syncthreads();                                // this chunk's stage may be overwritten
    }
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int e = 0; e < CPT; ++e)
            if (4 * sr + r < a.dim && sc + e < cols) stg[(long)(4 * sr + r) * a.vdim + sc + e] = m[r][e];
}

template <typename T, int D> int launch_chunks(const ChunkArgs& a, cudaStream_t st) {
    constexpr int gram = (2 * DC * (D + 4) + 2 * DC * DC + (DT / 32) * DC * DC) * 4;
    constexpr int walk = (2 * (d_rows<D>() + D_SIDE) + D * DV + 4 * 2 * DC * DV + 3 * DC * DV) * 4;
    static bool configured_dev[64] = {};                // the attributes are per device context
    int dev = 0;
    cudaGetDevice(&dev);
    if (!configured_dev[dev & 63]) {
        cudaFuncSetAttribute(delta_gram_kernel<T, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, gram);
        cudaFuncSetAttribute(delta_walk_kernel<T, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, walk);
        configured_dev[dev & 63] = true;
    }
    delta_gram_kernel<T, D><<<dim3(a.n_chunks, a.kv_heads, a.B), DT, gram, st>>>(a);
    delta_walk_kernel<T, D><<<dim3((a.vdim + DV - 1) / DV, a.heads, a.B), DT, walk, st>>>(a);
    return mixers_status();
}

}  // namespace

extern "C" long mixers_gated_delta_chunks_workspace(int B, int S, int kv_heads, int heads, int dim) {
    if (B <= 0 || S <= 0 || dim <= 0 || dim > 128 || kv_heads <= 0 || kv_heads > 65535 || heads > 65535 || B > 65535) return -1;
    const long n = (S + DC - 1) / DC, rows = dim <= 64 ? d_rows<64>() : d_rows<128>();
    return 4 * n * B * (kv_heads * rows + (long)heads * D_SIDE);
}

extern "C" int mixers_gated_delta_chunks(int dtype, const void* conv, int B, int S, int kv_heads, int heads, int dim, int vdim, const void* proj, int ld,
                                         int off_b, int off_a, const void* A_log, const void* dt_bias, float* state, int slot0, const int32_t* pad, float* o,
                                         float* workspace, mixers_stream_t stream) {
    if (B <= 0 || S <= 0) return 0;
    if (kv_heads <= 0 || heads % kv_heads != 0 || mixers_gated_delta_chunks_workspace(B, S, kv_heads, heads, dim) < 0 || !workspace || ((uintptr_t)workspace & 15)) return (int)cudaErrorInvalidValue;
    ChunkArgs a = {};
    a.conv = conv; a.proj = proj; a.A_log = A_log; a.dt_bias = dt_bias;
    a.B = B; a.S = S; a.kv_heads = kv_heads; a.heads = heads; a.dim = dim; a.vdim = vdim; a.ld_proj = ld; a.off_b = off_b; a.off_a = off_a;
    a.slot0 = slot0; a.n_chunks = (S + DC - 1) / DC; a.pad = pad; a.state = state; a.o = o;
    a.rows = workspace;
    a.side = workspace + (long)B * kv_heads * a.n_chunks * (dim <= 64 ? d_rows<64>() : d_rows<128>());
    MIXERS_DISPATCH(dtype, return (dim <= 64 ? launch_chunks<T, 64>(a, (cudaStream_t)stream) : launch_chunks<T, 128>(a, (cudaStream_t)stream)));
    return 0;
}
