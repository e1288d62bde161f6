// tc_pair.cuh -- what the kernels on pairs of SMs share (gemm_pair.cu, gemm_exact.cu): signals across the cluster, cta_group::2 wrappers,
// TMEM reads, direct stores, the reduction behind a split K range.
#pragma once
#include "tc_common.cuh"

namespace lowbit {
namespace gemmtc {

// one arrival at the barrier at this shared-memory offset of CTA `rank` of the cluster
__device__ __forceinline__ void mbar_arrive_at(uint32_t bar, uint32_t rank) {
    asm volatile("{\n\t.reg .b32 ra;\n\tmapa.shared::cluster.u32 ra, %0, %1;\n\t"
                 "mbarrier.arrive.shared::cluster.b64 _, [ra];\n\t}" ::"r"(bar), "r"(rank) : "memory");
}
__device__ __forceinline__ void umma2_f16_w(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate, uint32_t leader) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(leader) : "memory");
}
// arrives at the barrier at this offset in BOTH CTAs when the MMAs issued so far are done
__device__ __forceinline__ void umma2_commit_w(uint32_t bar, uint32_t leader) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "setp.ne.b32 q, %1, 0;\n\t"
        "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %2;\n\t}"
        ::"r"(bar), "r"(leader), "h"((uint16_t)3) : "memory");
}
// 16 TMEM lanes x 32 columns as mma fragments: v[4 i + ..] = (lane g, columns 8 i + 2 t, + 1), (lane g + 8, the same) for thread 4 g + t.
// No wait
__device__ __forceinline__ void tmem_ld_frag32(uint32_t taddr, float (&v)[16]) {
    uint32_t* r = reinterpret_cast<uint32_t*>(v);
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
// four 8 x 8 matrices of 16-bit elements, each stored turned: lane 8 j + i gives the address of row i (a column of the fragment) of matrix j
__device__ __forceinline__ void stmatrix4_trans(uint32_t addr, const uint32_t (&m)[4]) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(m[0]), "r"(m[1]), "r"(m[2]), "r"(m[3]) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
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
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// one feature's values of up to 16 consecutive tokens, straight to memory: 32-bit results and partial sums, whose two runs of 16
// features per token are 64 bytes each
__device__ __forceinline__ void store_feature(float* p, int64_t stride, const float (&v)[16], int cnt, float bias, bool accumulate) {
#pragma unroll
    for (int j = 0; j < 16; j++) if (j < cnt) p[j * stride] = accumulate ? v[j] + bias + p[j * stride] : v[j] + bias;
}
// K split: y[token][n] = sum over splits (in split order) of the fp32 partials, + bias, + y when accumulating
static __global__ void __launch_bounds__(256) reduce_partials_kernel(const float* part, int ksplit, int64_t mn, int64_t n_cols,
                                                              void* y, int y_dtype, const void* bias, int accumulate) {
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) * 4; i < mn; i += (int64_t)gridDim.x * blockDim.x * 4) {
        float4 a = *reinterpret_cast<const float4*>(part + i);
        for (int ks = 1; ks < ksplit; ks++) {
            const float4 b = *reinterpret_cast<const float4*>(part + ks * mn + i);
            a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
        }
        float v[4] = {a.x, a.y, a.z, a.w};
        const int64_t col = i % n_cols;                           // n_cols % 128 == 0: the four values share a row
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if (bias) v[j] += y_dtype == DT_F32 ? ((const float*)bias)[col + j]
                            : (y_dtype == DT_F16 ? __half2float(((const __half*)bias)[col + j]) : __bfloat162float(((const __nv_bfloat16*)bias)[col + j]));
            if (y_dtype == DT_F32) { float* p = (float*)y + i + j; *p = accumulate ? *p + v[j] : v[j]; }
            else if (y_dtype == DT_F16) { __half* p = (__half*)y + i + j; *p = __float2half_rn(accumulate ? __half2float(*p) + v[j] : v[j]); }
            else { __nv_bfloat16* p = (__nv_bfloat16*)y + i + j; *p = __float2bfloat16_rn(accumulate ? __bfloat162float(*p) + v[j] : v[j]); }
        }
    }
}

}  // namespace gemmtc
}  // namespace lowbit
