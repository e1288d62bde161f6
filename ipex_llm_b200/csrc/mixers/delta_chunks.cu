// Gated delta rule over a prompt, 32 tokens at a time.
//
//   M <- g M;  u = beta (v - M^T k);  M <- M + k u^T;  o = M^T q          (M [dim, vdim]; see recurrence.cu)
//
// With C_t = the product of the decays of the chunk's tokens up to t and M0 the state in front of the chunk, the chunk's updates solve a
// unit lower triangular system:
//   u_t + beta_t sum_{j < t} (C_t / C_j) (k_j . k_t) u_j = beta_t (v_t - C_t M0^T k_t)          (I + L) U = diag(beta) (V - C o (K M0))
//   o_t = C_t M0^T q_t + sum_{j <= t} (C_t / C_j) (k_j . q_t) u_j                                O = C o (Q M0) + A U
//   M   = C_last M0 + sum_j (C_last / C_j) k_j u_j^T
// The right side is linear in M0, so the system is solved before M0 is known: U = U0 - W M0 with T = (I + L)^-1 diag(beta), U0 = T V and
// W = T (C o K).  delta_gram_kernel does that for all chunks at once; what stays serial is two products per chunk and block of 16 value
// columns, W M0 and the state's update, with the outputs beside them (delta_walk_kernel).
// Everything is 32-bit, L, its inverse and T among it, but the gates, the norms, the quotients C_t / C_j and the scalar factors: they come from
// sums of logarithms held, and raised, in double precision (a quotient of 32-bit products would carry the rounding of both) and are rounded
// once, as they are handed over.  Keys and queries stay as they were given, times a power of two near 1 / norm: a 16-bit input is then one (bf16) or two
// (fp16) exact bf16 planes where a unit vector would need three; the rest of 1 / norm goes into the factors of a token.
#include "mixers_common.cuh"
#include <limits.h>
#include <math.h>
#include <stdlib.h>
#include <string.h>
#include <atomic>
#include <mutex>
#include <type_traits>

namespace {

constexpr int DC = 32;                                  // tokens per chunk
constexpr int DV = 16;                                  // value columns per block of the walk
constexpr int DT = 256;                                 // threads of the first kernel
constexpr int DH = 4;                                   // heads that it holds at a time
constexpr int DW = 4;                                   // warps of the walk that own a slice of D / DW rows of the state; as many finish the outputs
constexpr int D_U0 = DV + 4;                            // padded row of U0 in shared memory: a warp's eight columns by four token pairs lie in 32 banks
// the first kernel's padded rows: of the Gram matrices, of L by columns, of its inverse
constexpr int D_G = DC + 8, D_L = DC + 4, D_X = DC + 8, D_TP = DH * 2 * 3 * 3 * 32 * 4;
static_assert(D_TP >= DC * (128 + 8) && D_TP >= DH * DC * D_L, "T takes the place of the queries and of L");
// Operands of the walk's products lie as the lanes of mma.sync take them (gq = lane / 4, tq = lane % 4), so that every word is read once, by
// its lane.  A tile [8 n x 16 k] of one bf16 plane is two words of a lane, n = gq, k = 2 tq, + 1 and 2 tq + 8, + 9; two tiles share 16 bytes:
//   rows of a (group, chunk): K [8 dims][plane][lane][16 tokens: 2]: n = dim, k = token; Q [16 dims][16 tokens][plane][lane][8 tokens: 2]:
//   n = token, k = dim
//   side of a (head, chunk): W as Q, three planes; A [tile][plane][lane], n = t, k = j: four tiles of j < 16, then t >= 16, j >= 16;
//   C_t / norm of q_t; C_last / C_t / norm of k_t; C_t
template <typename T> __host__ __device__ constexpr int d_planes() { return sizeof(T) == 4 ? 3 : 1; }
template <> __host__ __device__ constexpr int d_planes<__half>() { return 2; }
template <int D, int NP> __host__ __device__ constexpr int d_rows() { return NP * DC * D; }            // 32-bit words
template <int D> __host__ __device__ constexpr int d_side() { return 3 * DC * D / 2 + 6 * 3 * 64 + 3 * DC; }
template <int D, int NP> __host__ __device__ constexpr int d_stage() { return d_rows<D, NP>() + d_side<D>() + DC * D_U0; }
// chunks in shared memory: two where three would not fit
template <int D, int NP> __host__ __device__ constexpr int d_stages() { return D > 64 && NP > 1 ? 2 : 3; }

struct ChunkArgs {
    const void* conv; const void* proj; const void* A_log; const void* dt_bias;
    int B, S, kv_heads, heads, dim, vdim, ld_proj, off_b, off_a, slot0, n_chunks;
    int seq;                                            // tokens from one sequence to the next: S, or more when S is a portion of them
    int parts;                                          // blocks of the first kernel that share a group's heads
    double q_scale;                                     // dim^-1/2
    const int32_t* pad;
    uint32_t* rows;                                     // [B][kv_heads][n_chunks][d_rows]
    uint32_t* side;                                     // [B][heads][n_chunks][d_side]
    unsigned int* late;                                 // in host memory: a wait ran out
    long long limit; int most;                          // of a wait, in SM clocks; the chunks that come (tests: fewer than there are)
    float* state; float* o;                             // o holds U0 until the walk has read it
};

__device__ __forceinline__ int first_token(const ChunkArgs& a, int b) {
    const int f = a.pad ? a.pad[b] - a.slot0 : 0;
    return f < 0 ? 0 : f > a.S ? a.S : f;
}

// the first NP bf16 planes of two values (hi + mid + lo = the value); the differences are exact
template <int NP> __device__ __forceinline__ void split(float a, float b, uint32_t (&out)[NP]) {
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(out[p]) : "f"(b), "f"(a));
        if (p + 1 < NP)
            asm("{ .reg .b64 x, y; mov.b64 x, {%0, %1}; mov.b64 y, {%2, %3}; add.rn.f32x2 x, x, y; mov.b64 {%0, %1}, x; }"
                : "+f"(a), "+f"(b) : "r"(out[p] * 65536u + 0x80000000u), "r"((out[p] & 0xffff0000u) ^ 0x80000000u));
    }
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_bf16_new(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
                 : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.0f));
}
// two sums, and two products added to them, per instruction
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    asm("{ .reg .b64 x, y; mov.b64 x, {%0, %1}; mov.b64 y, {%2, %3}; add.rn.f32x2 x, x, y; mov.b64 {%0, %1}, x; }" : "+f"(a.x), "+f"(a.y) : "f"(b.x), "f"(b.y));
    return a;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    asm("{ .reg .b64 x, y, z; mov.b64 x, {%2, %3}; mov.b64 y, {%4, %5}; mov.b64 z, {%0, %1}; fma.rn.f32x2 z, x, y, z; mov.b64 {%0, %1}, z; }"
        : "+f"(c.x), "+f"(c.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return c;
}
// the products of an NA-plane and an NB-plane number above 2^-25 of the largest, smallest first
template <int NA, int NB> struct Products {
    int n = 0, a[9] = {}, b[9] = {};
    constexpr Products() {
        for (int s = 2; s >= 0; --s)
            for (int i = s; i >= 0; --i)
                if (i < NA && s - i < NB) { a[n] = i; b[n] = s - i; ++n; }
    }
};

// a value as it is loaded: the compiler may not put the load off until it is used, or skip it
template <typename T> __device__ __forceinline__ T load_now(const T* p, bool there) {
    if constexpr (sizeof(T) == 4) {
        uint32_t v = 0;
        asm volatile("{ .reg .pred q; setp.ne.b32 q, %2, 0; @q ld.global.b32 %0, [%1]; }" : "+r"(v) : "l"(p), "r"((int)there));
        return *reinterpret_cast<const T*>(&v);
    } else {
        unsigned short v = 0;
        asm volatile("{ .reg .pred q; setp.ne.b32 q, %2, 0; @q ld.global.b16 %0, [%1]; }" : "+h"(v) : "l"(p), "r"((int)there));
        return *reinterpret_cast<const T*>(&v);
    }
}
__device__ __forceinline__ bool finite(float v) { return fabsf(v) < INFINITY; }
// enters the products of planes: no infinity, no NaN, and no value whose first plane rounds to infinity (from 3.3962e38 on)
__device__ __forceinline__ bool splits(float v) { return fabsf(v) <= 1e38f; }
// one copy of the code (the kernel is run through once per block, and its length is time), two at a time
__device__ __noinline__ double2 exp_64(double x, double y) { return make_double2(exp(x), exp(y)); }
// the gates of one token, lane = token; in double: a decay's error counts as often as there are tokens behind it.
// to [4][DC]: C_t, 1 / C_t, log C_t, beta_t
__device__ __noinline__ void gate_64(float a, float bias, float a_log, float b, bool there, double* to) {
    const int lane = threadIdx.x & 31;
    const double z = (double)a + (double)bias;
    const double2 f = exp_64((double)a_log, z);
    double lg = -f.x * (z > 20.0 ? z : log1p(f.y));
    lg = lg < -200.0 ? -200.0 : lg;                     // e^-200 is zero in 32 bits; an infinite logarithm would not cancel in a quotient
    double cum = there ? lg : 0.0;
#pragma unroll
    for (int m = 1; m < 32; m <<= 1) { const double v = __shfl_up_sync(0xffffffffu, cum, m); if (lane >= m) cum += v; }
    to[2 * DC + lane] = cum;
    const double2 c = exp_64(cum, -cum), g = exp_64(-(double)b, 0.0);
    to[lane] = c.x; to[DC + lane] = c.y;
    to[3 * DC + lane] = there ? 1.0 / (1.0 + g.x) : 0.0;
}
// rows and columns of an 8 x 8 tile of 16-bit values changed over
__device__ __forceinline__ uint32_t turned(uint32_t v) {
    uint32_t r;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
    return r;
}

// grid (chunks, key/value heads x parts, batch).  Everything of a chunk that needs no state: unit vectors, Gram matrices, gates, L, A,
// (I + L)^-1 per head, and its products with keys and values.  A block is a chain of short phases (gates in double 3400 clocks, the inverse
// 3500, the products 10000 for four heads), two blocks a SM: bound by their latencies; at the 128 registers that this leaves 16 bytes (bf16, 64
// dims) to 156 (fp32, 128) are spilled.  2048 tokens, 4 / 16 heads of 128, bf16: 27 us for
// 45 MB written (19 us without the solved right sides, which the walk multiplied out itself).  The products by mma.sync: as scalar fmas
// (a column per thread) the matrix's broadcast loads fill the shared-memory pipe, 84 us
template <typename T, int D>
__global__ void __launch_bounds__(DT, 2) delta_gram_kernel(const ChunkArgs a) {
    constexpr int LD = D + 8, NP = d_planes<T>(), TOK = DC / (DT / 32);
    extern __shared__ __align__(16) float sh[];
    float* const ks = sh;                               // [DC][LD]
    float* const kk = ks + DC * LD;                     // [DC][D_G] k_i . k_j
    float* const qk = kk + DC * D_G;                    // [DC][D_G] q_i . k_j
    double* const norms = reinterpret_cast<double*>(qk + DC * D_G);                      // [2][DC] what 1 / norm of keys and queries has beside the power of two
    double* const gates = norms + 2 * DC;               // [DH][4][DC] C_t, 1 / C_t, log C_t, beta_t
    float* const scale = reinterpret_cast<float*>(gates + DH * 4 * DC);                  // [2][DC] the powers of two
    int* const whole = reinterpret_cast<int*>(scale + 2 * DC);                           // [DC] the key has no infinity and no NaN
    float* const diag = scale + 3 * DC;                 // [DH][2][DC] T's diagonals
    float* const inv = diag + 2 * DH * DC;              // [DH][DC][D_X] (I + L)^-1
    // one after the other: queries [DC][LD]; L by columns [DH][DC][D_L]; T [DH][values, keys][3 tiles][plane][lane]
    float* const qs = inv + DH * DC * D_X;
    float* const lower = qs;
    uint4* const tp = reinterpret_cast<uint4*>(qs);
    const int c = blockIdx.x, g = blockIdx.y / a.parts, part = blockIdx.y % a.parts, b = blockIdx.z;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, gq = lane >> 2, tq = lane & 3;
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int t0 = first_token(a, b) + c * DC, nt = min(DC, a.S - t0);
    if (nt <= 0) return;
    const int ld = 2 * a.kv_heads * a.dim + a.heads * a.vdim;
    const int n_rep = a.heads / a.kv_heads, h_end = g * n_rep + (int)((long)n_rep * (part + 1) / a.parts);
    int h0 = g * n_rep + (int)((long)n_rep * part / a.parts);
    auto gate = [&](int hi) {                           // of up to DH heads from h0: a warp per head
        const int h = h0 + hi;
        const T* pr = (const T*)a.proj + ((long)b * a.seq + t0 + (lane < nt ? lane : 0)) * a.ld_proj + h;
        gate_64(to_f(pr[a.off_a]), to_f(((const T*)a.dt_bias)[h]), to_f(((const T*)a.A_log)[h]), to_f(pr[a.off_b]), lane < nt, gates + hi * 4 * DC);
    };
    {
        T kv[TOK][D / 32], qv[TOK][D / 32];
#pragma unroll
        for (int s = 0; s < TOK; ++s) {                 // token warp + 8 s
            const int t = warp + s * (DT / 32);
            const T* row = (const T*)a.conv + ((long)b * a.seq + t0 + (t < nt ? t : 0)) * ld + g * a.dim + lane;
#pragma unroll
            for (int e = 0; e < D / 32; ++e) {
                const bool ok = t < nt && lane + 32 * e < a.dim;
                qv[s][e] = load_now(row + 32 * e, ok);
                kv[s][e] = load_now(row + a.kv_heads * a.dim + 32 * e, ok);
            }
        }
        if (warp >= DT / 32 - DH && warp - (DT / 32 - DH) < h_end - h0) gate(warp - (DT / 32 - DH));
#pragma unroll
        for (int s = 0; s < TOK; ++s) {
            float sk = 0.0f, sq = 0.0f;
#pragma unroll
            for (int e = 0; e < D / 32; ++e) { const float k = to_f(kv[s][e]), q = to_f(qv[s][e]); sq += q * q; sk += k * k; }
            sq = warp_sum(sq); sk = warp_sum(sk);
            if (lane == 0) { norms[warp + s * (DT / 32)] = sk; norms[DC + warp + s * (DT / 32)] = sq; }
        }
        __syncthreads();
        if (warp < 2) {                                 // keys, then queries
            const double r = (warp ? a.q_scale : 1.0) * rsqrt(norms[tid] + 1e-6);
            const bool plain = r > 0.0;                 // no infinity, no NaN among the sums; then it lies between 2^-65 and 2^10
            const int hi = __double2hiint(r);
            // a key's rest lies in [1/4, 1/2): U C_last / C_t times it splits into planes whenever U is finite; a query's in [1, 2): Q M0 before it
            // is no larger than the output
            scale[tid] = plain ? __int_as_float(((hi >> 20) - 1023 + (warp ? 0 : 2) + 127) << 23) : (float)r;
            norms[tid] = plain ? __hiloint2double((hi & 0xfffff) | (warp ? 0x3ff00000 : 0x3fd00000), __double2loint(r)) : 1.0;
        }
        __syncthreads();
#pragma unroll
        for (int s = 0; s < TOK; ++s) {
            const int t = warp + s * (DT / 32);
            const float xk = scale[t], xq = scale[DC + t];
            bool ok = true;
#pragma unroll
            for (int e = 0; e < D / 32; ++e) {
                const float k = to_f(kv[s][e]) * xk;
                ks[t * LD + lane + 32 * e] = k; qs[t * LD + lane + 32 * e] = to_f(qv[s][e]) * xq;
                ok = ok && finite(k);
            }
            ok = __all_sync(0xffffffffu, ok);
            if (lane == 0) whole[t] = ok;
        }
    }
    __syncthreads();
    if (part == 0) {
        uint4* const rows = reinterpret_cast<uint4*>(a.rows + (((long)b * a.kv_heads + g) * a.n_chunks + c) * d_rows<D, NP>());
#pragma unroll 2
        for (int i = warp; i < D / 8; i += DT / 32) {   // K: eight dims; Q: 16 dims by 16 tokens
            uint32_t k[4][NP], q[4][NP];
            const float* kp = ks + 2 * tq * LD + 8 * i + gq;
            const float* qp = qs + (16 * (i & 1) + gq) * LD + 16 * (i >> 1) + 2 * tq;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                split<NP>(kp[8 * e * LD], kp[(8 * e + 1) * LD], k[e]);
                const float2 v = *reinterpret_cast<const float2*>(qp + 8 * (e >> 1) * LD + 8 * (e & 1));
                split<NP>(v.x, v.y, q[e]);
            }
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                rows[(i * NP + p) * 32 + lane] = make_uint4(k[0][p], k[1][p], k[2][p], k[3][p]);
                rows[(D / 8 * NP + i * NP + p) * 32 + lane] = make_uint4(q[0][p], q[1][p], q[2][p], q[3][p]);
            }
        }
    }
    // the two Gram matrices.  What the sums' rounding leaves sets the error of a chunk's outputs
    if constexpr (NP == 1) {                            // exact products, in sums of 32 dims each: a tile of 16 x 8 of each matrix per warp
        const int i0 = 16 * (warp >> 2) + gq, j0 = 8 * (warp & 3);
        float sx[4] = {}, sy[4] = {};
#pragma unroll 1
        for (int d0 = 0; d0 < D; d0 += 32) {
            float x[4] = {}, y[4] = {};
#pragma unroll
            for (int d = d0; d < d0 + 32; d += 16) {
                uint32_t ka[4], qa[4], kb[2];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int at = (i0 + 8 * (e & 1)) * LD + d + 8 * (e >> 1) + 2 * tq;
                    const float2 kf = *reinterpret_cast<const float2*>(ks + at), qf = *reinterpret_cast<const float2*>(qs + at);
                    uint32_t pk[1], pq[1];
                    split<1>(kf.x, kf.y, pk); split<1>(qf.x, qf.y, pq);
                    ka[e] = pk[0]; qa[e] = pq[0];
                }
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const float2 kf = *reinterpret_cast<const float2*>(ks + (j0 + gq) * LD + d + 8 * e + 2 * tq);
                    uint32_t pk[1];
                    split<1>(kf.x, kf.y, pk);
                    kb[e] = pk[0];
                }
                mma_bf16(x, ka, kb[0], kb[1]);
                mma_bf16(y, qa, kb[0], kb[1]);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) { sx[e] += x[e]; sy[e] += y[e]; }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int at = (i0 + 8 * (e >> 1)) * D_G + j0 + 2 * tq + (e & 1);
            kk[at] = sx[e]; qk[at] = sy[e];
        }
    } else {                                            // 2 x 2 of each per thread, eight sums per dot product
        const int i0 = tid >> 4, j0 = tid & 15;
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
            for (int s = 0; s < 2; ++s) {
                const int at = (i0 + 16 * r) * D_G + j0 + 16 * s;
                kk[at] = sum8(x[r][s]); qk[at] = sum8(y[r][s]);
            }
    }
    for (bool more = false; h0 < h_end; h0 += DH, more = true) {
        const int nh = min(DH, h_end - h0);
        __syncthreads();                                // the Gram matrices; the heads before these have been left
        if (more) {
            if (warp < nh) gate(warp);
            __syncthreads();
        }
        // L and A, a tile of A (and the same elements of L) per warp
        auto tile_of = [&](int i, bool plain) {
            const int hi = i / 6, tile = i % 6, th = tile >> 2, t = 8 * (th ? tile - 2 : tile) + gq;
            const double* const gt = gates + hi * 4 * DC;
            float* const L = lower + hi * DC * D_L;
            uint32_t* const side = a.side + (((long)b * a.heads + h0 + hi) * a.n_chunks + c) * d_side<D>();
            const double ct = plain ? gt[t] : 1.0, lt = ct * gt[3 * DC + t] * norms[t], at = ct * norms[DC + t];
            float out[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int j = 16 * th + 2 * tq + (e & 1) + 8 * (e >> 1);
                const double r = (plain ? gt[DC + j] : exp_64(gt[2 * DC + t] - gt[2 * DC + j], 0.0).x) * norms[j];
                out[e] = j <= t ? (float)(at * r) * qk[t * D_G + j] : 0.0f;
                L[j * D_L + t] = j < t ? (float)(lt * r) * kk[t * D_G + j] : 0.0f;
            }
            uint32_t lo[3], hi2[3];
            split<3>(out[0], out[1], lo);
            split<3>(out[2], out[3], hi2);
            uint2* const to = reinterpret_cast<uint2*>(side + 3 * DC * D / 2) + tile * 96 + lane;
#pragma unroll
            for (int p = 0; p < 3; ++p) to[32 * p] = make_uint2(lo[p], hi2[p]);
        };
        bool plain = true;                              // no factor of a quotient C_t / C_j leaves the range of a double
        for (int hi = 0; hi < nh; ++hi) plain = plain && gates[hi * 4 * DC + 2 * DC + 31] > -600.0;
        if (plain) {
#pragma unroll 3
            for (int i = warp; i < 6 * nh; i += DT / 32) tile_of(i, true);
        } else {
#pragma unroll 1
            for (int i = warp; i < 6 * nh; i += DT / 32) tile_of(i, false);
        }
        __syncthreads();
        if (warp < nh) {                                // X = (I + L)^-1, lane = column, eight rows at a time
            const float* const L = lower + warp * DC * D_L;
            float* const X = inv + warp * DC * D_X + lane;
#pragma unroll 1
            for (int i0 = 0; i0 < DC; i0 += 8) {
                float x[8];
#pragma unroll
                for (int r = 0; r < 8; ++r) x[r] = i0 + r == lane ? 1.0f : 0.0f;
                auto take = [&](const float* l, float xm, int from) {
#pragma unroll
                    for (int r = 0; r < 8; r += 4)
                        if (r + 3 >= from) {
                            const float4 f = *reinterpret_cast<const float4*>(l + r);
                            if (r >= from) x[r] = fmaf(-f.x, xm, x[r]);
                            if (r + 1 >= from) x[r + 1] = fmaf(-f.y, xm, x[r + 1]);
                            if (r + 2 >= from) x[r + 2] = fmaf(-f.z, xm, x[r + 2]);
                            x[r + 3] = fmaf(-f.w, xm, x[r + 3]);
                        }
                };
#pragma unroll 8
                for (int m = 0; m < i0; ++m) take(L + m * D_L + i0, X[m * D_X], 0);
#pragma unroll
                for (int r = 0; r < 7; ++r) take(L + (i0 + r) * D_L + i0, x[r], r + 1);
#pragma unroll
                for (int r = 0; r < 8; ++r) X[(i0 + r) * D_X] = x[r];            // the lane's own column
            }
            // T's diagonals apart: a token's own term is added last, as it is
            const double bt = gates[warp * 4 * DC + 3 * DC + lane];
            diag[warp * 2 * DC + lane] = (float)bt; diag[warp * 2 * DC + DC + lane] = (float)(bt * gates[warp * 4 * DC + lane] * norms[lane]);
            float* const cd = reinterpret_cast<float*>(a.side + (((long)b * a.heads + h0 + warp) * a.n_chunks + c) * d_side<D>() + 3 * DC * D / 2 + 6 * 3 * 64) + lane;
            const double* const gt = gates + warp * 4 * DC;
            cd[0] = (float)(gt[lane] * norms[DC + lane]);
            cd[DC] = (float)((plain ? gt[31] * gt[DC + lane] : exp_64(gt[2 * DC + 31] - gt[2 * DC + lane], 0.0).x) * norms[lane]);
            cd[2 * DC] = (float)gt[lane];
        }
        __syncthreads();
        // T = X times beta, for the values, and times beta C / norm, for the keys, without its diagonals, as planes: a tile [16 x 16] per warp
        for (int i = warp; i < 6 * nh; i += DT / 32) {
            const int hi = i / 6, of_w = i / 3 & 1, tile = i % 3, mt = tile > 0, th = tile > 1;
            const float* const X = inv + hi * DC * D_X, *const td = diag + (2 * hi + of_w) * DC;
            uint32_t pl[4][3];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int t = 16 * mt + 8 * (e & 1) + gq, j = 16 * th + 8 * (e >> 1) + 2 * tq;
                const float2 f = *reinterpret_cast<const float2*>(X + t * D_X + j), d = *reinterpret_cast<const float2*>(td + j);
                split<3>(j < t ? f.x * d.x : 0.0f, j + 1 < t ? f.y * d.y : 0.0f, pl[e]);
            }
            uint4* const to = tp + (i * 3) * 32 + lane;
#pragma unroll
            for (int p = 0; p < 3; ++p) to[32 * p] = make_uint4(pl[0][p], pl[1][p], pl[2][p], pl[3][p]);
        }
        __syncthreads();
        // W = T K and U0 = T V, 32 columns per warp at a time.  Values that do not split leave the products (whose zeros would turn them into NaN
        // for earlier tokens) and are added one by one
        const int n_w = D / 32, n_v = (a.vdim + 31) / 32;
        const bool pairs = (a.vdim & 1) == 0 && ((uintptr_t)a.o & 7) == 0;               // the outputs' rows start on 8 bytes
        uint32_t y[4][2][2][NP];                        // [8 columns][16 tokens][half][plane]
        float own[4][4][2];                             // [8 columns][8 tokens]: token gq, columns 2 tq, + 1
        int keys = -1;                                  // the columns of the keys that y and own hold
#pragma unroll 1
        for (int i = warp; i < nh * (n_w + n_v); i += DT / 32) {
            const int hi = i / (n_w + n_v), part_of = i % (n_w + n_v), h = h0 + hi;
            const bool of_w = part_of < n_w;
            const int c0 = 32 * (of_w ? part_of : part_of - n_w);
            const uint4* const tm = tp + (2 * hi + of_w) * 9 * 32 + lane;
            const T* const vp = (const T*)a.conv + ((long)b * a.seq + t0) * ld + 2 * a.kv_heads * a.dim + h * a.vdim + c0 + gq;
            bool odd = false;
            if (of_w) {
                if (keys != c0)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int j = 8 * e + 2 * tq;
                        const bool w0 = whole[j], w1 = whole[j + 1];
#pragma unroll
                        for (int n = 0; n < 4; ++n) {
                            const float* const kp = ks + j * LD + c0 + 8 * n + gq;
                            split<NP>(w0 ? kp[0] : 0.0f, w1 ? kp[LD] : 0.0f, y[n][e >> 1][e & 1]);
                            const float2 f = *reinterpret_cast<const float2*>(ks + (8 * e + gq) * LD + c0 + 8 * n + 2 * tq);
                            own[n][e][0] = f.x; own[n][e][1] = f.y;
                        }
                    }
                keys = c0;
            } else {
                keys = -1;
                T v[4][4][2];
#pragma unroll
                for (int n = 0; n < 4; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e)
#pragma unroll
                        for (int s = 0; s < 2; ++s) {
                            const int j = 8 * e + 2 * tq + s;
                            v[n][e][s] = load_now(vp + (long)j * ld + 8 * n, j < nt && c0 + 8 * n + gq < a.vdim);
                        }
#pragma unroll
                for (int n = 0; n < 4; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        if constexpr (sizeof(T) == 2) {
                            const uint32_t w = turned((uint32_t)*reinterpret_cast<const unsigned short*>(&v[n][e][0]) |
                                                      (uint32_t)*reinterpret_cast<const unsigned short*>(&v[n][e][1]) << 16);
                            const unsigned short h[2] = {(unsigned short)w, (unsigned short)(w >> 16)};
                            own[n][e][0] = to_f(*reinterpret_cast<const T*>(&h[0])); own[n][e][1] = to_f(*reinterpret_cast<const T*>(&h[1]));
                        } else {
                            const uint32_t w0 = __float_as_uint(to_f(v[n][e][0])), w1 = __float_as_uint(to_f(v[n][e][1]));
                            const uint32_t lo = turned(__byte_perm(w0, w1, 0x5410)), hi = turned(__byte_perm(w0, w1, 0x7632));
                            own[n][e][0] = __uint_as_float(__byte_perm(lo, hi, 0x5410)); own[n][e][1] = __uint_as_float(__byte_perm(lo, hi, 0x7632));
                        }
                        float f0 = to_f(v[n][e][0]), f1 = to_f(v[n][e][1]);
                        if (!splits(f0)) { f0 = 0.0f; odd = true; }
                        if (!splits(f1)) { f1 = 0.0f; odd = true; }
                        split<NP>(f0, f1, y[n][e >> 1][e & 1]);
                    }
            }
            constexpr Products<3, NP> pr;
            float x[2][4][4] = {}, xs[2][4][4] = {};    // [16 tokens][8 columns]; the largest products, the others
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int th = 0; th <= mt; ++th) {
                    uint32_t ta[3][4];
#pragma unroll
                    for (int p = 0; p < 3; ++p) {
                        const uint4 v = tm[((mt + th) * 3 + p) * 32];
                        ta[p][0] = v.x; ta[p][1] = v.y; ta[p][2] = v.z; ta[p][3] = v.w;
                    }
#pragma unroll
                    for (int q = 0; q < pr.n; ++q)
#pragma unroll
                        for (int n = 0; n < 4; ++n)
                            mma_bf16(q + 1 < pr.n ? xs[mt][n] : x[mt][n], ta[pr.a[q]], y[n][th][0][pr.b[q]], y[n][th][1][pr.b[q]]);
                }
            const float* const td = diag + (2 * hi + of_w) * DC + gq;
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int n = 0; n < 4; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        x[mt][n][e] = fmaf(td[16 * mt + 8 * (e >> 1)], own[n][2 * mt + (e >> 1)][e & 1], x[mt][n][e] + xs[mt][n][e]);
            if (of_w) {
                uint4* const side = reinterpret_cast<uint4*>(a.side + (((long)b * a.heads + h) * a.n_chunks + c) * d_side<D>()) + lane;
#pragma unroll
                for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                    for (int np = 0; np < 2; ++np) {
                        uint32_t w[4][3];
#pragma unroll
                        for (int e = 0; e < 4; ++e) split<3>(x[mt][2 * np + (e & 1)][2 * (e >> 1)], x[mt][2 * np + (e & 1)][2 * (e >> 1) + 1], w[e]);
#pragma unroll
                        for (int p = 0; p < 3; ++p) side[(((c0 / 16 + np) * 2 + mt) * 3 + p) * 32] = make_uint4(w[0][p], w[1][p], w[2][p], w[3][p]);
                    }
            } else {
                float* const ob = a.o + (((long)b * a.seq + t0) * a.heads + h) * a.vdim + c0;
                const long o_ld = (long)a.heads * a.vdim;
#pragma unroll
                for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                    for (int n = 0; n < 4; ++n)
#pragma unroll
                        for (int e = 0; e < 4; e += 2) {
                            const int t = 16 * mt + 4 * e + gq, col = 8 * n + 2 * tq;
                            if (t < nt && c0 + col < a.vdim) {
                                float* const to = ob + t * o_ld + col;
                                if (pairs) *reinterpret_cast<float2*>(to) = make_float2(x[mt][n][e], x[mt][n][e + 1]);
                                else {
                                    to[0] = x[mt][n][e];
                                    if (c0 + col + 1 < a.vdim) to[1] = x[mt][n][e + 1];
                                }
                            }
                        }
                if (__any_sync(0xffffffffu, odd)) {     // one by one, a lane per column
                    __syncwarp();
                    __threadfence_block();
                    if (c0 + lane < a.vdim)
                        for (int j = 0; j < nt; ++j) {
                            const float v = to_f(vp[(long)j * ld + lane - gq]);
                            if (!splits(v))
                                for (int t = j + 1; t < nt; ++t) ob[t * o_ld + lane] += inv[(hi * DC + t) * D_X + j] * diag[2 * hi * DC + j] * v;
                        }
                }
            }
        }
    }
}

template <int BYTES> __device__ __forceinline__ void cp_async(float* dst, const float* src, bool there) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "n"(BYTES), "r"(there ? BYTES : 0) : "memory");
}
__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
// A wait that runs out raises the device's word in host memory and the block's in shared memory.  The block's waits end at once from then on, its
// results are undefined, and the warp that brings the chunks in brings no more and stays until its copies have landed
constexpr long long kWait = 4000000000ll;               // about two seconds
__device__ __forceinline__ bool arrived(uint32_t bar, uint32_t parity) {
    uint32_t there;
    asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }" : "=r"(there) : "r"(bar), "r"(parity) : "memory");
    return there != 0;
}
__device__ __forceinline__ bool wait_on(uint32_t bar, uint32_t parity, unsigned int* late, long long limit, volatile int* failed) {
    const long long t0 = clock64();
    while (!arrived(bar, parity))
        if (clock64() - t0 > limit || (failed && *failed)) {
            if (failed) *failed = 1;
            *(volatile unsigned int*)late = 1u;
            __threadfence_system();
            return false;
        }
    return true;
}
__device__ __forceinline__ void wait_for(uint32_t bar, uint32_t parity, const ChunkArgs& a, volatile int* failed) {
    if (!arrived(bar, parity)) wait_on(bar, parity, a.late, a.limit, failed);
}
// whole warp, the same answer in every lane
__device__ __forceinline__ bool wait_warp(uint32_t bar, uint32_t parity, const ChunkArgs& a, volatile int* failed) {
    return __all_sync(0xffffffffu, arrived(bar, parity)) || __all_sync(0xffffffffu, wait_on(bar, parity, a.late, a.limit, failed));
}
// two accumulator tiles side by side, [16 x 8] each, as planes of one [16 x 16] operand
__device__ __forceinline__ void split_pair(const float (&l)[4], const float (&r)[4], uint32_t (&a)[3][4]) {
    uint32_t t[4][3];
    split<3>(l[0], l[1], t[0]); split<3>(l[2], l[3], t[1]); split<3>(r[0], r[1], t[2]); split<3>(r[2], r[3], t[3]);
#pragma unroll
    for (int p = 0; p < 3; ++p)
#pragma unroll
        for (int e = 0; e < 4; ++e) a[p][e] = t[e][p];
}

// grid (blocks of DV value columns, heads, batch); warps 0 to DW - 1 walk, DW to 2 DW - 1 finish the outputs and bring the chunks in.
// All products by mma.sync on bf16 planes (each product exact, sums in 32 bits; see Products): scalar fmas would cost every operand its 4
// bytes of the 128 that shared memory yields per clock.  The state stays in registers, transposed: a warp owns D / DW of its rows as the
// accumulators of tiles [16 columns x 8 rows], and those are, split into planes, operands of the next chunk's products.  A chunk costs its
// chain two exchanges between the four warps: the slices' sums of W M0, then U as planes, each summed and split by one warp.  Q M0 fills
// the tensor pipe while they wait; A U and the stores belong to the other four warps and may lag a chunk behind.
// Measured, 2048 tokens, 16 heads, 128 x 128, bf16: 70 us, 1940 clocks a chunk, of which 960 in the tensor pipe (120 instructions a SM
// quarter, 8 clocks each); the rest is the chain's latency (the splits, the exchanges).  68 us since the copying warp asks for its phases as
// a whole warp.  When T (V - C o (K M0)) was formed inside the
// walk, with eight partial sums and three barriers, and keys took three planes: 141 us, 4100 clocks.  Error of the outputs against 64 bits,
// relative to their norm: 1.00e-7 (1.05e-7 then).
template <typename T, int D>
__global__ void __launch_bounds__(64 * DW, 1) delta_walk_kernel(const ChunkArgs a) {
    constexpr int NP = d_planes<T>(), KT = D / DW / 16, DTL = 2 * KT;                    // planes of K and Q; blocks of 16 and of 8 rows of the state per warp
    constexpr int STAGE = d_stage<D, NP>(), STAGES = d_stages<D, NP>(), AT = d_rows<D, NP>() + 3 * DC * D / 2, CD = AT + 6 * 3 * 64, U0 = CD + 3 * DC;
    extern __shared__ __align__(16) float sh[];
    float4* const wsum = reinterpret_cast<float4*>(sh + STAGES * STAGE);                 // [2 chunks][4 tiles][DW slices][32] partial (W M0)^T
    float4* const osum = wsum + 2 * DW * 4 * 32;                                         // [STAGES chunks][4 tiles][DW slices][32] partial (Q M0)^T
    float4* const us = osum + STAGES * DW * 4 * 32;                                      // [STAGES chunks][4 tiles][32] U^T
    uint2* const up_sh = reinterpret_cast<uint2*>(us + STAGES * 4 * 32);                 // [2 chunks][16 tokens][plane][lane][8 tokens] (U C_last / C_t)^T
    // per slot: the chunk has come; its U and the slices' sums are there; state and outputs have left it
    const uint32_t full = (uint32_t)__cvta_generic_to_shared(up_sh + 2 * 2 * 3 * 64), ready = full + 8 * STAGES, empty = ready + 8 * STAGES;
    const int col0 = blockIdx.x * DV, h = blockIdx.y, b = blockIdx.z, g = h / (a.heads / a.kv_heads);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, gq = lane >> 2, tq = lane & 3;
    volatile int* const failed = reinterpret_cast<volatile int*>(up_sh + 2 * 2 * 3 * 64 + 3 * STAGES);
    if (threadIdx.x == 0) {
        *failed = 0;
#pragma unroll
        for (int i = 0; i < STAGES; ++i) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 33;" ::"r"(full + 8 * i) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(ready + 8 * i), "n"(DW) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(empty + 8 * i), "n"(2 * DW) : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int first = first_token(a, b), n = (a.S - first + DC - 1) / DC;
    const int cols = min(DV, a.vdim - col0);
    const long o_ld = (long)a.heads * a.vdim;
    float* const ob = a.o + (((long)b * a.seq) * a.heads + h) * a.vdim + col0;
    __syncthreads();

    if (warp >= DW) {                                   // outputs: C_t Q M0 + A U, eight tokens per warp
        const int w = warp - DW;
        // the first of these warps brings the chunks in
        const uint32_t* const rows = a.rows + ((long)b * a.kv_heads + g) * a.n_chunks * d_rows<D, NP>();
        const uint32_t* const side = a.side + ((long)b * a.heads + h) * a.n_chunks * d_side<D>();
        const uint32_t at0 = (uint32_t)__cvta_generic_to_shared(sh);
        const bool wide = (a.vdim & 3) == 0 && ((uintptr_t)a.o & 15) == 0;
        const int come = min(n, a.most);
        auto bring = [&](int c) {
            const int slot = c % STAGES;
            const uint32_t at = at0 + slot * STAGE * 4, bar = full + 8 * slot;
            if (c >= STAGES && !wait_warp(empty + 8 * slot, (c / STAGES - 1) & 1, a, failed)) return false;
            if (lane == 0) {
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "n"(4 * (d_rows<D, NP>() + d_side<D>())) : "memory");
                bulk_copy(at + 4 * d_rows<D, NP>(), side + (long)c * d_side<D>(), 4 * d_side<D>(), bar);
                bulk_copy(at, rows + (long)c * d_rows<D, NP>(), 4 * d_rows<D, NP>(), bar);
            }
            float* const u0 = sh + slot * STAGE + U0;
            const int t0 = first + c * DC;
            if (wide) {
#pragma unroll
                for (int i = lane; i < DC * DV / 4; i += 32) {
                    const int t = i / (DV / 4), e = 4 * (i % (DV / 4));
                    const bool there = t0 + t < a.S && e < cols;
                    cp_async<16>(u0 + t * D_U0 + e, there ? ob + (t0 + t) * o_ld + e : ob, there);
                }
            } else {
#pragma unroll 1
                for (int i = lane; i < DC * DV; i += 32) {
                    const int t = i / DV, e = i % DV;
                    const bool there = t0 + t < a.S && e < cols;
                    cp_async<4>(u0 + t * D_U0 + e, there ? ob + (t0 + t) * o_ld + e : ob, there);
                }
            }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
            return true;
        };
        if (w == 0)
#pragma unroll 1
            for (int c = 0; c < STAGES && c < come; ++c) bring(c);
        for (int i = threadIdx.x - 32 * DW; i < first * DV; i += 32 * DW) if (i % DV < cols) ob[(i / DV) * o_ld + i % DV] = 0.0f;
        int c = 0;
#pragma unroll 1
        for (; c < n; ++c) {
            const float* const stage = sh + (c % STAGES) * STAGE;
            constexpr Products<3, 3> pr;
            const int slot = c % STAGES;
            wait_for(ready + 8 * slot, (c / STAGES) & 1, a, failed);
            if (!wait_warp(full + 8 * slot, (c / STAGES) & 1, a, failed)) break;     // (long over; A and the factors were written by copies)
            const float4* const at = osum + (slot * 4 + w) * DW * 32 + lane;
            const float4 p0 = at[0], p1 = at[32], p2 = at[64], p3 = at[96];
            const float ct0 = stage[CD + 8 * w + 2 * tq], ct1 = stage[CD + 8 * w + 2 * tq + 1];
            uint2 ap[2][3];
#pragma unroll
            for (int th = 0; th < 2; ++th)
                if (th == 0 || w >= 2)
#pragma unroll
                    for (int p = 0; p < 3; ++p) ap[th][p] = reinterpret_cast<const uint2*>(stage + AT)[((th ? 2 + w : w) * 3 + p) * 32 + lane];
            float u[4][4];
#pragma unroll
            for (int tt = 0; tt < 4; ++tt) {
                const float4 v = us[(slot * 4 + tt) * 32 + lane];
                u[tt][0] = v.x; u[tt][1] = v.y; u[tt][2] = v.z; u[tt][3] = v.w;
            }
            float r[4] = {ct0 * ((p0.x + p1.x) + (p2.x + p3.x)), ct1 * ((p0.y + p1.y) + (p2.y + p3.y)),
                          ct0 * ((p0.z + p1.z) + (p2.z + p3.z)), ct1 * ((p0.w + p1.w) + (p2.w + p3.w))};
            // A token's sum must not meet what later tokens of the chunk hold if that does not split: such values leave the products (whose
            // zeros would turn them into NaN) and enter one by one
            bool odd = false;
#pragma unroll
            for (int tt = 0; tt < 4; ++tt)
#pragma unroll
                for (int e = 0; e < 4; ++e) odd |= !splits(u[tt][e]);
            odd = __any_sync(0xffffffffu, odd);
            float f[4][4];
#pragma unroll
            for (int tt = 0; tt < 4; ++tt)
#pragma unroll
                for (int e = 0; e < 4; ++e) f[tt][e] = splits(u[tt][e]) ? u[tt][e] : 0.0f;
            float x[3][4] = {};
#pragma unroll
            for (int th = 0; th < 2; ++th)
                if (th == 0 || w >= 2) {
                    uint32_t up[3][4];
                    split_pair(f[2 * th], f[2 * th + 1], up);
#pragma unroll
                    for (int q = 0; q < pr.n; ++q) mma_bf16(x[q % 3], up[pr.a[q]], ap[th][pr.b[q]].x, ap[th][pr.b[q]].y);
                }
#pragma unroll
            for (int e = 0; e < 4; ++e) r[e] += (x[0][e] + x[1][e]) + x[2][e];
            if (!odd) {                                 // all that was read has been used (an arrival behind loads under way may be overtaken)
                __syncwarp();
                if (lane == 0) arrive(empty + 8 * slot);
            }
            if (odd)
#pragma unroll 1
                for (int j = 0; j < 8 * w + 8; ++j) {
                    const float* const uj = reinterpret_cast<const float*>(us + (slot * 4 + (j >> 3)) * 32 + (lane & ~3) + ((j & 7) >> 1)) + (j & 1);
#pragma unroll
                    for (int hf = 0; hf < 2; ++hf)
                        if (const float v = uj[2 * hf]; !splits(v))
#pragma unroll
                            for (int s = 0; s < 2; ++s) {
                                const int tl = 2 * tq + s;           // A [8 w + tl][j], of its planes
                                if (j > 8 * w + tl) continue;
                                const uint2* const aj = reinterpret_cast<const uint2*>(stage + AT) + ((j >> 4) ? 2 + w : w) * 96 + tl * 4 + ((j & 7) >> 1);
                                float av = 0.0f;
#pragma unroll
                                for (int p = 2; p >= 0; --p) {
                                    const uint32_t pair = (j >> 3) & 1 ? aj[32 * p].y : aj[32 * p].x;
                                    av += __uint_as_float(j & 1 ? pair & 0xffff0000u : pair << 16);
                                }
                                r[2 * hf + s] += av * v;
                            }
                }
            if (odd) {
                __syncwarp();
                if (lane == 0) arrive(empty + 8 * slot);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int t = first + c * DC + 8 * w + 2 * tq + (e & 1), col = gq + 8 * (e >> 1);
                if (t < a.S && col < cols) ob[t * o_ld + col] = r[e];
            }
            if (w == 0 && c + STAGES < come && !bring(c + STAGES)) break;            // (every chunk's copies are waited for before it is read)
        }
        if (w == 0 && c < n)                            // a wait ran out: the copies under way
            for (const int end = min(come, c + STAGES); c < end; ++c) wait_on(full + 8 * (c % STAGES), (c / STAGES) & 1, a.late, kWait, nullptr);
        return;
    }

    const int k0 = warp * (D / DW);
    float* const stg = a.state + ((long)b * a.heads + h) * a.dim * a.vdim + col0;
    float m[DTL][4];                                    // the state, transposed: columns gq, gq + 8 by rows k0 + 8 dt + 2 tq, + 1
#pragma unroll
    for (int dt = 0; dt < DTL; ++dt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int i = k0 + 8 * dt + 2 * tq + (e & 1), col = gq + 8 * (e >> 1);
            m[dt][e] = i < a.dim && col < cols ? stg[(long)i * a.vdim + col] : 0.0f;
        }
    uint4 w[KT][2][3];                                  // W of the next chunk, the slice's rows
    auto load_w = [&](int c) {
        const uint4* const at = reinterpret_cast<const uint4*>(sh + (c % STAGES) * STAGE + d_rows<D, NP>()) + warp * KT * 2 * 96 + lane;
#pragma unroll
        for (int kt = 0; kt < KT; ++kt)
#pragma unroll
            for (int tp = 0; tp < 2; ++tp)
#pragma unroll
                for (int p = 0; p < 3; ++p) w[kt][tp][p] = at[((kt * 2 + tp) * 3 + p) * 32];
    };
    uint32_t mp[KT][3][4];                              // the state's planes
#pragma unroll
    for (int kt = 0; kt < KT; ++kt) split_pair(m[2 * kt], m[2 * kt + 1], mp[kt]);
    if (n > 0) { wait_for(full, 0, a, failed); load_w(0); }
#pragma unroll 1
    for (int c = 0; c < n; ++c) {
        const int slot = c % STAGES;
        const float* const stage = sh + slot * STAGE;
        float4* const wp = wsum + (c & 1) * DW * 4 * 32;
        constexpr Products<3, 3> p33;
        constexpr Products<3, NP> p3n;
        // ---- (W M0)^T over the slice's rows of M0: tiles of 8 tokens.  What the rest of the chunk takes from shared memory, and the next chunk's W,
        // is read beside these products
        float acc[KT][4][4];
        auto w_half = [&](int kt) {
#pragma unroll
            for (int q = 0; q < p33.n; ++q)
#pragma unroll
                for (int tt = 0; tt < 4; ++tt) {
                    const uint4& t = w[kt][tt >> 1][p33.b[q]];
                    if (q == 0) mma_bf16_new(acc[kt][tt], mp[kt][p33.a[q]], tt & 1 ? t.z : t.x, tt & 1 ? t.w : t.y);
                    else mma_bf16(acc[kt][tt], mp[kt][p33.a[q]], tt & 1 ? t.z : t.x, tt & 1 ? t.w : t.y);
                }
        };
        w_half(0);
        uint4 qf[KT][2][NP], kf[DTL][NP];
        const uint4* const qat = reinterpret_cast<const uint4*>(stage + d_rows<D, NP>() / 2) + warp * KT * 2 * NP * 32 + lane;
        const uint4* const kat = reinterpret_cast<const uint4*>(stage) + warp * DTL * NP * 32 + lane;
#pragma unroll
        for (int kt = 0; kt < KT; ++kt)
#pragma unroll
            for (int tp = 0; tp < 2; ++tp)
#pragma unroll
                for (int p = 0; p < NP; ++p) qf[kt][tp][p] = qat[((kt * 2 + tp) * NP + p) * 32];
        // the warp's own tile of U0, and what the update needs beside U
        const float* const ur = stage + U0 + gq + (8 * warp + 2 * tq) * D_U0;
        const float2 u0a = make_float2(ur[0], ur[D_U0]), u0b = make_float2(ur[8], ur[D_U0 + 8]);
        const float2 e = *reinterpret_cast<const float2*>(stage + CD + DC + 8 * warp + 2 * tq);
        const float decay = stage[CD + 3 * DC - 1];
        if constexpr (KT == 2) w_half(1);
#pragma unroll
        for (int dt = 0; dt < DTL; ++dt)
#pragma unroll
            for (int p = 0; p < NP; ++p) kf[dt][p] = kat[(dt * NP + p) * 32];
        auto next_w = [&] {
            if (c + 1 < n) { wait_for(full + 8 * ((c + 1) % STAGES), ((c + 1) / STAGES) & 1, a, failed); load_w(c + 1); }
        };
        if constexpr (STAGES > 2) next_w();             // (of two chunks the second comes while the first is used)
#pragma unroll
        for (int tt = 0; tt < 4; ++tt) {
            float2 x = make_float2(acc[0][tt][0], acc[0][tt][1]), y = make_float2(acc[0][tt][2], acc[0][tt][3]);
            if constexpr (KT == 2) { x = add2(x, make_float2(acc[1][tt][0], acc[1][tt][1])); y = add2(y, make_float2(acc[1][tt][2], acc[1][tt][3])); }
            wp[(tt * DW + warp) * 32 + lane] = make_float4(x.x, x.y, y.x, y.y);
        }
        asm volatile("barrier.cta.sync 1, %0;" ::"n"(32 * DW) : "memory");
        const float4 p0 = wp[warp * DW * 32 + lane], p1 = wp[(warp * DW + 1) * 32 + lane], p2 = wp[(warp * DW + 2) * 32 + lane], p3 = wp[(warp * DW + 3) * 32 + lane];
        // ---- (Q M0)^T likewise, beside the exchange of U: one half before, one behind
        float oa[4][4];
        auto q_half = [&](int q0, int q1) {
#pragma unroll
            for (int i = q0; i < q1; ++i) {
                const int q = i / KT, kt = i % KT;
#pragma unroll
                for (int tt = 0; tt < 4; ++tt) {
                    const uint4& t = qf[kt][tt >> 1][p3n.b[q]];
                    if (i == 0) mma_bf16_new(oa[tt], mp[kt][p3n.a[q]], tt & 1 ? t.z : t.x, tt & 1 ? t.w : t.y);
                    else mma_bf16(oa[tt], mp[kt][p3n.a[q]], tt & 1 ? t.z : t.x, tt & 1 ? t.w : t.y);
                }
            }
        };
        q_half(0, p3n.n * KT / 2);
        {                                               // U = U0 - W M0, a tile per warp
            const float2 sa = add2(add2(make_float2(p0.x, p0.y), make_float2(p1.x, p1.y)), add2(make_float2(p2.x, p2.y), make_float2(p3.x, p3.y)));
            const float2 sb = add2(add2(make_float2(p0.z, p0.w), make_float2(p1.z, p1.w)), add2(make_float2(p2.z, p2.w), make_float2(p3.z, p3.w)));
            const float2 ua = make_float2(u0a.x - sa.x, u0a.y - sa.y), ub = make_float2(u0b.x - sb.x, u0b.y - sb.y);
            uint32_t xa[3], xb[3];
            split<3>(ua.x * e.x, ua.y * e.y, xa);
            split<3>(ub.x * e.x, ub.y * e.y, xb);
#pragma unroll
            for (int p = 0; p < 3; ++p) up_sh[(((c & 1) * 2 + (warp >> 1)) * 3 + p) * 64 + 2 * lane + (warp & 1)] = make_uint2(xa[p], xb[p]);
            us[(slot * 4 + warp) * 32 + lane] = make_float4(ua.x, ua.y, ub.x, ub.y);
        }
        q_half(p3n.n * KT / 2, p3n.n * KT);
        asm volatile("barrier.cta.sync 2, %0;" ::"n"(32 * DW) : "memory");
        // ---- the state: C_last M0 + K^T (U C_last / C_t)
        float add[2][DTL][4];
        uint32_t up[2][3][4];
#pragma unroll
        for (int th = 0; th < 2; ++th)
#pragma unroll
            for (int p = 0; p < 3; ++p) {
                const uint4 v = reinterpret_cast<const uint4*>(up_sh)[(((c & 1) * 2 + th) * 3 + p) * 32 + lane];
                up[th][p][0] = v.x; up[th][p][1] = v.y; up[th][p][2] = v.z; up[th][p][3] = v.w;
            }
#pragma unroll
        for (int th = 0; th < 2; ++th)
#pragma unroll
            for (int d0 = 0; d0 < DTL; d0 += th ? 2 : DTL)           // at last by pairs: the first is split while the second is multiplied
#pragma unroll
                for (int q = 0; q < p3n.n; ++q)
#pragma unroll
                    for (int dt = d0; dt < d0 + (th ? 2 : DTL); ++dt) {
                        const uint4& t = kf[dt][p3n.b[q]];
                        if (q == 0) mma_bf16_new(add[th][dt], up[th][p3n.a[q]], th ? t.z : t.x, th ? t.w : t.y);
                        else mma_bf16(add[th][dt], up[th][p3n.a[q]], th ? t.z : t.x, th ? t.w : t.y);
                    }
        float4* const op = osum + slot * 4 * DW * 32;
#pragma unroll
        for (int tt = 0; tt < 4; ++tt) op[(tt * DW + warp) * 32 + lane] = make_float4(oa[tt][0], oa[tt][1], oa[tt][2], oa[tt][3]);
        __syncwarp();
        if (lane == 0) arrive(ready + 8 * slot);
        if constexpr (STAGES == 2) next_w();
        const float2 dd = make_float2(decay, decay);
#pragma unroll
        for (int kt = 0; kt < KT; ++kt) {
#pragma unroll
            for (int dt = 2 * kt; dt < 2 * kt + 2; ++dt)
#pragma unroll
                for (int i = 0; i < 4; i += 2) {
                    const float2 v = fma2(dd, make_float2(m[dt][i], m[dt][i + 1]),
                                          add2(make_float2(add[0][dt][i], add[0][dt][i + 1]), make_float2(add[1][dt][i], add[1][dt][i + 1])));
                    m[dt][i] = v.x; m[dt][i + 1] = v.y;
                }
            split_pair(m[2 * kt], m[2 * kt + 1], mp[kt]);
        }
        __syncwarp();
        if (lane == 0) arrive(empty + 8 * slot);        // all that was read has been used
    }
#pragma unroll
    for (int dt = 0; dt < DTL; ++dt)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = k0 + 8 * dt + 2 * tq + (i & 1), col = gq + 8 * (i >> 1);
            if (r < a.dim && col < cols) stg[(long)r * a.vdim + col] = m[dt][i];
        }
}

template <typename T, int D> int launch_chunks(ChunkArgs a, cudaStream_t st) {
    constexpr int NP = d_planes<T>();
    constexpr int gram = (DC * (D + 8) + 2 * DC * D_G + 3 * DC + 2 * DH * DC + DH * DC * D_X + D_TP) * 4 + (2 + DH * 4) * DC * 8;
    constexpr int walk = (d_stages<D, NP>() * d_stage<D, NP>() + (2 * DW + d_stages<D, NP>() * (DW + 1)) * 4 * 32 * 4 + 2 * 2 * 3 * 64 * 2) * 4 + 24 * d_stages<D, NP>() + 8;
    static_assert(walk <= 232448, "shared memory");
    static bool configured_dev[64] = {};                // the attributes are per device context
    static int sms_dev[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (!configured_dev[dev & 63]) {
        cudaFuncSetAttribute(delta_gram_kernel<T, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, gram);
        cudaFuncSetAttribute(delta_walk_kernel<T, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, walk);
        if (cudaDeviceGetAttribute(&sms_dev[dev & 63], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) { cudaGetLastError(); sms_dev[dev & 63] = 148; }
        configured_dev[dev & 63] = true;
    }
    a.parts = 1;                                        // until every SM has a block (a part forms the Gram matrices again, a fifth of a head's work)
    while (a.parts * 2 <= a.heads / a.kv_heads && (long)a.n_chunks * a.kv_heads * a.B * a.parts < sms_dev[dev & 63] && a.kv_heads * a.parts * 2 <= 65535) a.parts *= 2;
    // Both start while the kernel in front drains and wait for its end before they touch memory; in a captured stream the graph's edges stay plain
    cudaStreamCaptureStatus state = cudaStreamCaptureStatusNone;
    const bool overlap = cudaStreamIsCapturing(st, &state) == cudaSuccess && state == cudaStreamCaptureStatusNone;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.stream = st; cfg.attrs = at; cfg.numAttrs = overlap ? 1 : 0;
    cfg.gridDim = dim3(a.n_chunks, a.kv_heads * a.parts, a.B); cfg.blockDim = dim3(DT); cfg.dynamicSmemBytes = gram;
    cudaLaunchKernelEx(&cfg, delta_gram_kernel<T, D>, (const ChunkArgs)a);
    cfg.gridDim = dim3((a.vdim + DV - 1) / DV, a.heads, a.B); cfg.blockDim = dim3(64 * DW); cfg.dynamicSmemBytes = walk;
    cudaLaunchKernelEx(&cfg, delta_walk_kernel<T, D>, (const ChunkArgs)a);
    return mixers_status();
}

}  // namespace

// Scratch of a call at most (or one chunk's, where that is more): 21 KB a token at 4 / 16 heads of 128, 42 KB at 8 / 32.  Longer prompts
// run in portions of whole chunks, the state carried through memory as between two calls
namespace {
constexpr long kDeltaScratch = 512l << 20;
// rows as three planes, whatever the inputs' type
long rows_words(int dim) { return dim <= 64 ? d_rows<64, 3>() : d_rows<128, 3>(); }
long chunk_bytes(int B, int kv_heads, int heads, int dim) { return 4l * B * (kv_heads * rows_words(dim) + (long)heads * (dim <= 64 ? d_side<64>() : d_side<128>())); }
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

// a word per device, each in a cache line of its own, in host memory that every device writes; never freed (recorded graphs hold it)
static unsigned int* late_word() {
    static std::atomic<unsigned int*> words{nullptr};
    if (!words.load(std::memory_order_acquire)) {
        static std::mutex mu;
        std::lock_guard<std::mutex> lock(mu);
        if (!words.load(std::memory_order_relaxed)) {
            cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;                   // page-locking is no part of a capture
            cudaThreadExchangeStreamCaptureMode(&mode);
            void* p = nullptr;
            const cudaError_t e = cudaHostAlloc(&p, 64 * 128, cudaHostAllocPortable | cudaHostAllocMapped);
            cudaThreadExchangeStreamCaptureMode(&mode);
            if (e != cudaSuccess) return nullptr;
            memset(p, 0, 64 * 128);
            words.store((unsigned int*)p, std::memory_order_release);
        }
    }
    int dev = 0;
    return cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64 ? words.load(std::memory_order_acquire) + 32 * dev : nullptr;
}

// the limit of the waits in this thread's launches, 0: the usual one
static thread_local long long t_wait_limit = 0;

template <typename T> static int run_portions(ChunkArgs a, cudaStream_t st) {
    const int S = a.S, slot0 = a.slot0, step = DC * (int)portion_chunks(a.B, S, a.kv_heads, a.heads, a.dim);
    const long ld = 2 * a.kv_heads * a.dim + a.heads * a.vdim;
    const T *const conv = (const T*)a.conv, *const proj = (const T*)a.proj;
    float* const o = a.o;
    a.seq = S;
    a.side = a.rows + (long)a.B * a.kv_heads * (step / DC) * rows_words(a.dim);
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
    a.q_scale = 1.0 / sqrt((double)dim);
    a.slot0 = slot0; a.pad = pad; a.state = state; a.o = o; a.rows = reinterpret_cast<uint32_t*>(workspace);
    a.late = late_word(); a.limit = t_wait_limit ? llabs(t_wait_limit) : kWait; a.most = t_wait_limit < 0 ? 1 : INT_MAX;
    if (!a.late) return (int)cudaErrorMemoryAllocation;
    if (*(volatile unsigned int*)a.late) {              // a wait inside an earlier call ran out: its results are undefined
        *(volatile unsigned int*)a.late = 0;
        return (int)cudaErrorLaunchTimeout;
    }
    MIXERS_DISPATCH(dtype, return run_portions<T>(a, (cudaStream_t)stream));
    return 0;
}

extern "C" int mixers_wait_expired(void) {
    if (cudaDeviceSynchronize() != cudaSuccess) { cudaGetLastError(); return -1; }
    const unsigned int* const late = late_word();
    return late ? *(const volatile unsigned int*)late != 0 : -1;
}

// development aid, not in the public header: the limit, in SM clocks, of the waits in this thread's launches (0: the usual one; below zero: a
// block's first chunk alone comes, and the waits for the others run out after that many clocks)
extern "C" void mixers_debug_set_wait_limit(long long clocks) { t_wait_limit = clocks; }
