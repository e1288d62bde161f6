// tc_common.cuh -- what the tcgen05 dequant-GEMM kernels share (gemm_pair.cu: prompts; gemm_tc.cu: small batches): mbarrier, TMA and
// tcgen05 wrappers, and the codecs that expand one 16x64 tile of packed weights to fp16.
#pragma once
#include <cuda.h>
#include <cuda_fp8.h>
#include <mutex>
#include "lowbit_common.cuh"
#include "lowbit_internal.h"
#include "gemv_args.h"       // apply_act

namespace lowbit {
namespace gemmtc {

constexpr int kTileN = 128;          // features per CTA (two 64-row groups)
constexpr int kTileBytesAB = 128 * 128;   // one 128-row x 64-element 2-byte operand tile

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_wait(uint32_t bar, uint32_t parity) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "WAIT_%=:\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%0], %1;\n\t"
        "@p bra DONE_%=;\n\t"
        "bra WAIT_%=;\n\t"
        "DONE_%=:\n\t}" ::"r"(bar), "r"(parity) : "memory");
}
// K-major, 128B-swizzled operand tile whose rows are 128 bytes: LBO = 1 (unused), SBO = 1024 B
// (eight rows), descriptor version 1 (sm_100), layout type 2 = SWIZZLE_128B
__device__ __forceinline__ uint64_t make_desc(uint32_t smem_addr) {
    return (uint64_t)((smem_addr >> 4) & 0x3fff) | ((uint64_t)1 << 16) | ((uint64_t)64 << 32) | ((uint64_t)1 << 46) |
           ((uint64_t)2 << 61);
}
// Issued by a whole warp in warp-uniform control flow: `leader` is true in one elected lane.  With every operand
// computed identically by all lanes the compiler keeps descriptors and addresses in uniform registers; a single-lane
// branch made it move every operand into a uniform register per instruction (~23 instructions and 45 ns per MMA).
__device__ __forceinline__ void umma_f16_w(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate, uint32_t leader) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(leader) : "memory");
}
__device__ __forceinline__ void umma_commit_w(uint32_t bar, uint32_t leader) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "setp.ne.b32 q, %1, 0;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar), "r"(leader) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx_w(uint32_t bar, uint32_t bytes, uint32_t leader) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t@q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t}"
                 ::"r"(bar), "r"(bytes), "r"(leader) : "memory");
}
__device__ __forceinline__ void bulk_g2s_w(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar, uint32_t leader) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %4, 0;\n\t"
                 "@q cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n\t}"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar), "r"(leader) : "memory");
}
__device__ __forceinline__ void tma_load_2d_w(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar, uint32_t leader) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %5, 0;\n\t"
                 "@q cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n\t}"
                 ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(bar), "r"(leader) : "memory");
}
// ---- bounded waits: one that runs out raises the device's word in host memory (lowbit_internal.h), and the kernel winds down: every
// role leaves its loop, waits for the copies and MMAs of its own that are still under way, and the block frees its TMEM
constexpr long long kWaitCycles = 4000000000ll;           // about two seconds
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// whole warp.  A limit below zero (tests): copies of the kernel stop half-way, and the waits for them run out after that many clocks
__device__ __forceinline__ bool wait_over(long long t0, const Waits& W) {
    if (!__any_sync(0xffffffffu, clock64() - t0 > (W.limit < 0 ? -W.limit : W.limit))) return false;
    if ((threadIdx.x & 31) == 0) { *(volatile unsigned int*)W.word = 1u; __threadfence_system(); }
    return true;
}
// whole warp; the same answer in every lane.  false: the limit ran out
__device__ __forceinline__ bool mbar_wait_lim(uint32_t bar, uint32_t parity, const Waits& W) {
    if (__all_sync(0xffffffffu, mbar_test(bar, parity))) return true;
    const long long t0 = clock64();
    while (!__all_sync(0xffffffffu, mbar_test(bar, parity)))
        if (wait_over(t0, W)) return false;
    return true;
}
// three barriers at once: a test takes about 100 clocks to answer, and these overlap.  Tests that do not suspend the warp: the answer
// may be wanted early, for a phase that is far off
__device__ __forceinline__ bool mbar_test3(uint32_t b0, uint32_t p0, uint32_t b1, uint32_t p1, uint32_t b2, uint32_t p2) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p, q, r;\n\t"
                 "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "mbarrier.test_wait.parity.shared::cta.b64 q, [%3], %4;\n\t"
                 "mbarrier.test_wait.parity.shared::cta.b64 r, [%5], %6;\n\t"
                 "and.pred p, p, q;\n\tand.pred p, p, r;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(b0), "r"(p0), "r"(b1), "r"(p1), "r"(b2), "r"(p2) : "memory");
    return ok != 0;
}
// `ready`: what mbar_test3 said earlier
__device__ __forceinline__ bool mbar_wait3_lim(bool ready, uint32_t b0, uint32_t p0, uint32_t b1, uint32_t p1, uint32_t b2, uint32_t p2, const Waits& W) {
    if (__all_sync(0xffffffffu, ready)) return true;
    const long long t0 = clock64();
    while (!__all_sync(0xffffffffu, mbar_test3(b0, p0, b1, p1, b2, p2)))
        if (wait_over(t0, W)) return false;
    return true;
}
// the same for four
__device__ __forceinline__ bool mbar_test4(uint32_t b0, uint32_t p0, uint32_t b1, uint32_t p1, uint32_t b2, uint32_t p2, uint32_t b3, uint32_t p3) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p, q, r, s;\n\t"
                 "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "mbarrier.test_wait.parity.shared::cta.b64 q, [%3], %4;\n\t"
                 "mbarrier.test_wait.parity.shared::cta.b64 r, [%5], %6;\n\t"
                 "mbarrier.test_wait.parity.shared::cta.b64 s, [%7], %8;\n\t"
                 "and.pred p, p, q;\n\tand.pred r, r, s;\n\tand.pred p, p, r;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(b0), "r"(p0), "r"(b1), "r"(p1), "r"(b2), "r"(p2), "r"(b3), "r"(p3) : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_wait4_lim(bool ready, uint32_t b0, uint32_t p0, uint32_t b1, uint32_t p1, uint32_t b2, uint32_t p2, uint32_t b3, uint32_t p3,
                                               const Waits& W) {
    if (__all_sync(0xffffffffu, ready)) return true;
    const long long t0 = clock64();
    while (!__all_sync(0xffffffffu, mbar_test4(b0, p0, b1, p1, b2, p2, b3, p3)))
        if (wait_over(t0, W)) return false;
    return true;
}
// the phases of the last `n` of `issued` trips around a ring of n slots are complete: this warp's copies have landed
template <typename Full> __device__ __forceinline__ void drain_ring(int issued, int n, Full full, const Waits& W) {
    const Waits late = {W.word, kWaitCycles};
    for (int i = issued > n ? issued - n : 0; i < issued; i++)
        if (!mbar_wait_lim(full(i % n), (uint32_t)((i / n) & 1), late)) return;
}
__device__ __forceinline__ uint32_t elect_leader() {
    uint32_t pred;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(pred));
    return pred;
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ uint4 lds128(uint32_t a) {
    uint4 r;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "r"(a));
    return r;
}
__device__ __forceinline__ uint32_t h2u(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }
__device__ __forceinline__ __half2 u2h(uint32_t u) { return *reinterpret_cast<__half2*>(&u); }
__device__ __forceinline__ uint32_t h2_to_bf2(uint32_t h) {
    const float2 f = __half22float2(u2h(h));
    __nv_bfloat162 b = __floats2bfloat162_rn(f.x, f.y);
    return *reinterpret_cast<uint32_t*>(&b);
}
__device__ __forceinline__ uint32_t and_or(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}

// Scaled fp16 values of k-step s of one 16x64 tile for lane (g,t): out[0] = row g (4s,4s+1),
// out[1] = row g+8 (4s,4s+1), out[2] = row g (4s+2,4s+3), out[3] = row g+8 (4s+2,4s+3); the same
// register order as the mma.sync fragments of the GEMV kernel (the tile layout is shared).
template <int QT> struct Expand;

// The same order of codes in bf16 pairs, exact and unscaled, for formats whose value is code x scale (bf16(), gemm_exact.cu): 4-bit codes
// under the magic number 128, 8- and 6-bit floats as the upper halves of their 32-bit values.  A way that ends in cvt.rn.bf16x2.f32
// (7 clocks of a quarter of an SM) took twice the clocks.
__device__ __forceinline__ __nv_bfloat162 u2bf(uint32_t u) { return *reinterpret_cast<__nv_bfloat162*>(&u); }
__device__ __forceinline__ uint32_t bf2u(__nv_bfloat162 v) { return *reinterpret_cast<uint32_t*>(&v); }
__device__ __forceinline__ uint32_t h2_to_bf2_exact(uint32_t h) {            // at most 8 bits of significand
    const float2 f = __half22float2(u2h(h));
    return __byte_perm(__float_as_uint(f.x), __float_as_uint(f.y), 0x7632u);
}
template <int OFFSET> struct Expand4 {          // sym_int4 (OFFSET 1) / asym_int4 (OFFSET 2)
    static constexpr int kTileBytes = 512;
    static constexpr bool kHasMin = OFFSET == 2;
    static constexpr int kLutBytes = 0;
    // the lane's 16 bytes of the tile in one conflict-free LDS.128 (four LDS.32 at a 16-byte lane stride cost 4 wavefronts each)
    struct Codes { uint4 q; };
    __device__ static __forceinline__ void load(uint32_t codes, int lane, Codes& c) { c.q = lds128(codes + lane * 16); }
    __device__ static __forceinline__ void bf16(const Codes& c, int s, uint32_t (&out)[4]) {
        const uint32_t w = s == 0 ? c.q.x : s == 1 ? c.q.y : s == 2 ? c.q.z : c.q.w;
#pragma unroll
        for (int i = 0; i < 4; i++) out[i] = bf2u(__hsub2(u2bf(and_or(w >> (4 * i), 0x000f000fu, 0x43004300u)), u2bf(0x43084308u)));      // 128 + n - 136
    }
    __device__ static __forceinline__ void run(const Codes& c, int s, __half2 dlo, __half2 dhi, __half2 mlo,
                                               __half2 mhi, uint32_t, uint32_t (&out)[4]) {
        const uint32_t w = s == 0 ? c.q.x : s == 1 ? c.q.y : s == 2 ? c.q.z : c.q.w;
        const uint32_t w2 = w >> 8;
        const __half2 k16th = __floats2half2_rn(0.0625f, 0.0625f);
        // 0x6400 | n = 1024 + n ; 0x6400 | (n << 4) = 1024 + 16 n  (exact in fp16)
        if (OFFSET == 1) {
            // n - 8 straight from the magic number (exact): one subtraction / one fma per pair, then the product, rounded once
            const __half2 k1032 = __floats2half2_rn(1032.0f, 1032.0f), km72 = __floats2half2_rn(-72.0f, -72.0f);
            const __half2 v0 = __hsub2(u2h(and_or(w, 0x000f000fu, 0x64006400u)), k1032);
            const __half2 v1 = __hfma2(u2h(and_or(w, 0x00f000f0u, 0x64006400u)), k16th, km72);
            const __half2 v2 = __hsub2(u2h(and_or(w2, 0x000f000fu, 0x64006400u)), k1032);
            const __half2 v3 = __hfma2(u2h(and_or(w2, 0x00f000f0u, 0x64006400u)), k16th, km72);
            out[0] = h2u(__hmul2(v0, dlo)); out[1] = h2u(__hmul2(v1, dhi));
            out[2] = h2u(__hmul2(v2, dlo)); out[3] = h2u(__hmul2(v3, dhi));
        } else {
            const __half2 k1024 = __floats2half2_rn(1024.0f, 1024.0f), km64 = __floats2half2_rn(-64.0f, -64.0f);
            const __half2 v0 = __hsub2(u2h(and_or(w, 0x000f000fu, 0x64006400u)), k1024);                 // n
            const __half2 v1 = __hfma2(u2h(and_or(w, 0x00f000f0u, 0x64006400u)), k16th, km64);           // n
            const __half2 v2 = __hsub2(u2h(and_or(w2, 0x000f000fu, 0x64006400u)), k1024);
            const __half2 v3 = __hfma2(u2h(and_or(w2, 0x00f000f0u, 0x64006400u)), k16th, km64);
            out[0] = h2u(__hfma2(v0, dlo, mlo)); out[1] = h2u(__hfma2(v1, dhi, mhi));
            out[2] = h2u(__hfma2(v2, dlo, mlo)); out[3] = h2u(__hfma2(v3, dhi, mhi));
        }
    }
};
template <> struct Expand<QT_SYM_INT4> : Expand4<1> {};
template <> struct Expand<QT_ASYM_INT4> : Expand4<2> {};

template <int QT> struct Expand8 {
    static constexpr int kTileBytes = 1024;
    static constexpr bool kHasMin = false;
    __device__ static __forceinline__ uint32_t pair(uint32_t w, int hi) {
        uint32_t h;
        if (QT == QT_FP8_E5M2) h = __byte_perm(w, 0u, hi ? 0x3424u : 0x1404u);
        else {
            const unsigned short two = (unsigned short)(hi ? (w >> 16) : (w & 0xffffu));
            asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h) : "h"(two));
        }
        return h;
    }
    static constexpr int kLutBytes = 0;
    struct Codes { uint4 q0, q1; };
    __device__ static __forceinline__ void bf16(const Codes& c, int s, uint32_t (&out)[4]) {
        const uint32_t w[2] = {s == 0 ? c.q0.x : s == 1 ? c.q0.y : s == 2 ? c.q0.z : c.q0.w, s == 0 ? c.q1.x : s == 1 ? c.q1.y : s == 2 ? c.q1.z : c.q1.w};
#pragma unroll
        for (int i = 0; i < 4; i++) out[i] = h2_to_bf2_exact(pair(w[i & 1], i >> 1));
    }
    __device__ static __forceinline__ void load(uint32_t codes, int lane, Codes& c) {
        c.q0 = lds128(codes + lane * 16); c.q1 = lds128(codes + 512 + lane * 16);
    }
    __device__ static __forceinline__ void run(const Codes& c, int s, __half2 dlo, __half2 dhi, __half2, __half2,
                                               uint32_t, uint32_t (&out)[4]) {
        const uint32_t w0 = s == 0 ? c.q0.x : s == 1 ? c.q0.y : s == 2 ? c.q0.z : c.q0.w;
        const uint32_t w1 = s == 0 ? c.q1.x : s == 1 ? c.q1.y : s == 2 ? c.q1.z : c.q1.w;
        out[0] = h2u(__hmul2(u2h(pair(w0, 0)), dlo)); out[1] = h2u(__hmul2(u2h(pair(w1, 0)), dhi));
        out[2] = h2u(__hmul2(u2h(pair(w0, 1)), dlo)); out[3] = h2u(__hmul2(u2h(pair(w1, 1)), dhi));
    }
};
template <> struct Expand<QT_FP8_E4M3> : Expand8<QT_FP8_E4M3> {};
template <> struct Expand<QT_FP8_E5M2> : Expand8<QT_FP8_E5M2> {};

template <> struct Expand<QT_FP6> {
    static constexpr int kTileBytes = 768;
    static constexpr bool kHasMin = false;
    __device__ static __forceinline__ uint32_t cvt2(unsigned short two) {
        uint32_t h;
        asm("cvt.rn.f16x2.e3m2x2 %0, %1;" : "=r"(h) : "h"(two));
        return h;
    }
    static constexpr int kLutBytes = 0;
    struct Codes { uint4 lo; uint2 hi; };
    __device__ static __forceinline__ void bf16(const Codes& c, int s, uint32_t (&out)[4]) {
        const int u = s >> 1;
        const uint32_t sh = (s & 1) ? 4u : 0u;
        const uint32_t l[2] = {u ? c.lo.y : c.lo.x, u ? c.lo.w : c.lo.z}, h[2] = {c.hi.x, c.hi.y};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint32_t e = ((l[i & 1] >> sh) & 0x0f0f0f0fu) | (((h[i & 1] >> (2 * s)) & 0x03030303u) << 4);
            out[i] = h2_to_bf2_exact(cvt2((unsigned short)(i >> 1 ? e >> 16 : e & 0xffffu)));
        }
    }
    __device__ static __forceinline__ void load(uint32_t codes, int lane, Codes& c) {
        c.lo = lds128(codes + lane * 16);
        asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(c.hi.x), "=r"(c.hi.y) : "r"(codes + 512 + lane * 8));
    }
    __device__ static __forceinline__ void run(const Codes& c, int s, __half2 dlo, __half2 dhi, __half2, __half2,
                                               uint32_t, uint32_t (&out)[4]) {
        const int u = s >> 1;
        const uint32_t l0 = u ? c.lo.y : c.lo.x, l1 = u ? c.lo.w : c.lo.z, h0 = c.hi.x, h1 = c.hi.y;
        const uint32_t sh = (s & 1) ? 4u : 0u;
        const uint32_t e0 = ((l0 >> sh) & 0x0f0f0f0fu) | (((h0 >> (2 * s)) & 0x03030303u) << 4);
        const uint32_t e1 = ((l1 >> sh) & 0x0f0f0f0fu) | (((h1 >> (2 * s)) & 0x03030303u) << 4);
        out[0] = h2u(__hmul2(u2h(cvt2((unsigned short)(e0 & 0xffffu))), dlo));
        out[1] = h2u(__hmul2(u2h(cvt2((unsigned short)(e1 & 0xffffu))), dhi));
        out[2] = h2u(__hmul2(u2h(cvt2((unsigned short)(e0 >> 16))), dlo));
        out[3] = h2u(__hmul2(u2h(cvt2((unsigned short)(e1 >> 16))), dhi));
    }
};

// nf4: byte b of the lane's word s is the code pair of out[b] (tilednf4_pos); a 256-entry table of
// fp16 pairs of NormalFloat values sits in shared memory, 128 bytes per entry = one 4-byte slot per lane, so that no two
// lanes of a lookup meet in a bank (the first layout, 8 slots per entry, cost 3.1 wavefronts per LDS -- see the GEMV codec).
template <> struct Expand<QT_NF4> {
    static constexpr int kTileBytes = 512;
    static constexpr bool kHasMin = false;
    static constexpr int kLutBytes = 256 * 128;
    __device__ static __forceinline__ void fill_lut(uint8_t* lut, int tid, int nthreads) {
        for (int e = tid; e < 256; e += nthreads) {
            const uint32_t v = h2u(__floats2half2_rn(kNF4Table[e & 15], kNF4Table[e >> 4]));
            uint4* dst = reinterpret_cast<uint4*>(lut + e * 128);
#pragma unroll
            for (int c = 0; c < 8; c++) dst[c] = make_uint4(v, v, v, v);
        }
    }
    struct Codes { uint4 q; };
    __device__ static __forceinline__ void load(uint32_t codes, int lane, Codes& c) { c.q = lds128(codes + lane * 16); }
    // lut = table address + 4 * lane
    __device__ static __forceinline__ void run(const Codes& c, int s, __half2 dlo, __half2 dhi, __half2, __half2,
                                               uint32_t lut, uint32_t (&out)[4]) {
        const uint32_t w = s == 0 ? c.q.x : s == 1 ? c.q.y : s == 2 ? c.q.z : c.q.w;
        uint32_t v0, v1, v2, v3;
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v0) : "r"(lut + __byte_perm(w, 0u, 0x4440u) * 128u));
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v1) : "r"(lut + __byte_perm(w, 0u, 0x4441u) * 128u));
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v2) : "r"(lut + __byte_perm(w, 0u, 0x4442u) * 128u));
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v3) : "r"(lut + __byte_perm(w, 0u, 0x4443u) * 128u));
        out[0] = h2u(__hmul2(u2h(v0), dlo)); out[1] = h2u(__hmul2(u2h(v1), dhi));
        out[2] = h2u(__hmul2(u2h(v2), dlo)); out[3] = h2u(__hmul2(u2h(v3), dhi));
    }
};

template <bool BF> __device__ __forceinline__ uint32_t pack2(float a, float b) {
    if (BF) return bf2u(__floats2bfloat162_rn(a, b));
    return h2u(__floats2half2_rn(a, b));
}

// The same order of weights rounded ONCE to the activation type from their 32-bit value, the bits that dequantising (layout.cu) gives, for
// the product with the transposed weights.  code x scale: the product of an fp16 code and an fp16 scale is rounded once as it is; to bf16
// with the scale in two parts, d = hi + lo, exact, as the code times lo is (at most 4 + 3 bits): fma(code, hi, code * lo).  Minima and
// table: in 32 bits.
struct ScaleBf { __nv_bfloat162 hi, lo; };
__device__ __forceinline__ ScaleBf split_scale(__half d) {
    const float f = __half2float(d);
    const __nv_bfloat16 hi = __float2bfloat16_rn(f);
    ScaleBf s;
    s.hi = __bfloat162bfloat162(hi);
    s.lo = __bfloat162bfloat162(__float2bfloat16_rn(fabsf(f) <= 65504.0f ? f - __bfloat162float(hi) : 0.0f));      // none of an infinite scale
    return s;
}
__device__ __forceinline__ uint32_t scaled_bf(uint32_t code, const ScaleBf& d) { return bf2u(__hfma2(u2bf(code), d.hi, __hmul2(u2bf(code), d.lo))); }
// rows g (lo) and g + 8 (hi) of one 16 x 64 tile; registers 2 k4, 2 k4 + 1 of either row are k-step k4
template <int QT, bool BF>
__device__ __forceinline__ void expand_once(const typename Expand<QT>::Codes& c, uint32_t dq, uint32_t mq, uint32_t lut, uint32_t (&lo)[8], uint32_t (&hi)[8]) {
    using E = Expand<QT>;
    const __half2 d2 = u2h(dq), m2 = u2h(mq);
    ScaleBf sl, sh;
    if constexpr (BF && QT != QT_NF4 && QT != QT_ASYM_INT4) { sl = split_scale(__low2half(d2)); sh = split_scale(__high2half(d2)); }
    const float f[2] = {__low2float(d2), __high2float(d2)}, b[2] = {__low2float(m2), __high2float(m2)};
#pragma unroll
    for (int k4 = 0; k4 < 4; k4++) {
        uint32_t a[4];
        if constexpr (QT == QT_NF4) {
            const uint32_t w = k4 == 0 ? c.q.x : k4 == 1 ? c.q.y : k4 == 2 ? c.q.z : c.q.w;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                float x, y;
                asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(x), "=f"(y) : "r"(lut + __byte_perm(w, 0u, 0x4440u + i) * 128u));
                a[i] = pack2<BF>(x * f[i & 1], y * f[i & 1]);
            }
        } else if constexpr (QT == QT_ASYM_INT4 && BF) {
            const __half2 one = __floats2half2_rn(1.0f, 1.0f), zero = __floats2half2_rn(0.0f, 0.0f);
            E::run(c, k4, one, one, zero, zero, 0u, a);              // the codes
#pragma unroll
            for (int i = 0; i < 4; i++) { const float2 n = __half22float2(u2h(a[i])); a[i] = pack2<BF>(fmaf(n.x, f[i & 1], b[i & 1]), fmaf(n.y, f[i & 1], b[i & 1])); }
        } else if constexpr (BF) {
            E::bf16(c, k4, a);
#pragma unroll
            for (int i = 0; i < 4; i++) a[i] = scaled_bf(a[i], i & 1 ? sh : sl);
        } else {
            E::run(c, k4, __low2half2(d2), __high2half2(d2), __low2half2(m2), __high2half2(m2), lut, a);
        }
        lo[2 * k4] = a[0]; lo[2 * k4 + 1] = a[2]; hi[2 * k4] = a[1]; hi[2 * k4 + 1] = a[3];
    }
}
// nf4's table for it: entry b = the two 32-bit values of code byte b, in 16 slots (a 64-bit load is served half a warp at a time)
__device__ __forceinline__ void fill_nf4_pairs(uint8_t* lut, int tid, int nthreads) {
    for (int e = tid; e < 256; e += nthreads) {
        const float4 v = make_float4(kNF4Table[e & 15], kNF4Table[e >> 4], kNF4Table[e & 15], kNF4Table[e >> 4]);
        float4* dst = reinterpret_cast<float4*>(lut + e * 128);
#pragma unroll
        for (int c = 0; c < 8; c++) dst[c] = v;
    }
}

// bytes of one 64-row group x one k-block as the kernels stage it: codes, fp16 scales [, minima]
template <int QT> struct PackedBlock {
    static constexpr int kSuper = RG_TILES * Expand<QT>::kTileBytes;
    static constexpr int kGroup = kSuper + 128 + (Expand<QT>::kHasMin ? 128 : 0);
};

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
        else cudaGetLastError();
    });
    return fn;
}
// activations [rows][k] of a 16-bit type as boxes of `box_rows` rows x 64 elements, 128-byte swizzle; out-of-range rows read zero
static int encode_rows(CUtensorMap* map, const void* x, bool bf, int64_t rows, int64_t k, int box_rows) {
    EncodeTiledFn enc = encode_fn();
    if (!enc) { set_error(LB_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver"); return LB_ERR_CUDA; }
    const cuuint64_t gdim[2] = {(cuuint64_t)k, (cuuint64_t)rows};
    const cuuint64_t gstride[1] = {(cuuint64_t)k * 2};
    const cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    auto encode = [&] { return enc(map, bf ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(x), gdim,
                           gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE); };
    CUresult r = encode();
    if (r == CUDA_ERROR_INVALID_CONTEXT) {                // a thread (autograd's, say) before its first runtime call: bind its device's context
        int dev = 0;
        cudaGetDevice(&dev);
        cudaSetDevice(dev);
        r = encode();
    }
    if (r != CUDA_SUCCESS) { set_error(LB_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r); return LB_ERR_CUDA; }
    return LB_OK;
}

}  // namespace gemmtc
}  // namespace lowbit
