// experts.cu -- the routed feed-forwards of many tokens (reference models/qwen3_moe.py:106-132, deepseek.py:313-330: a loop over the
// experts, each a handful of operators on its tokens' rows):
//   sort      the (token, choice) pairs by expert: counts, row offsets, a row per pair (one block, shared-memory counters);
//   gather    the tokens' activations into sorted rows;
//   act(gate) * up of every expert's rows, then down, both by the two-SM matmul kernel over all experts at once (gemm_pair.cu);
//             experts of at most kExactRows rows by the GEMV, two launches each, whose weights stay code x scale in 32 bits;
//   combine   y[token] = sum over its choices, in choice order, of weight * row, in 32 bits, rounded once.
// The host learns the counts while the two large products run: it waits for the sort only.
// The loop it replaces was bound by its launches, 30 per expert with two host synchronisations: 1.89 ms for 512 tokens, two of eight
// experts of 4096 x 14336, of which the matmuls were 0.9; so 0.49 ms.
#include "lowbit_common.cuh"
#include "lowbit_internal.h"

namespace lowbit {

namespace {
constexpr int kSortThreads = 1024, kSortExperts = 256;

// what the host reads: row offsets, then the three address tables
struct HostView {
    int offs[kSortExperts + 2];
    unsigned long long tab[3][kSortExperts];
};

__global__ void __launch_bounds__(kSortThreads) experts_sort_kernel(const void* __restrict__ ids, int ids_i64, int pairs, int top_k, int n_experts,
                                                                    const unsigned long long* __restrict__ gates, const unsigned long long* __restrict__ ups,
                                                                    const unsigned long long* __restrict__ downs, HostView* __restrict__ view,
                                                                    int* __restrict__ row_of, int* __restrict__ token_of) {
    int* const offs = view->offs;
    for (int e = threadIdx.x; e < n_experts; e += kSortThreads) { view->tab[0][e] = gates[e]; view->tab[1][e] = ups[e]; view->tab[2][e] = downs[e]; }
    __shared__ int count[kSortExperts], next[kSortExperts];
    for (int e = threadIdx.x; e < kSortExperts; e += kSortThreads) count[e] = 0;
    __syncthreads();
    auto id_at = [&](int p) { return ids_i64 ? ((const long long*)ids)[p] : (long long)((const int*)ids)[p]; };
    for (int p = threadIdx.x; p < pairs; p += kSortThreads) {
        const long long e = id_at(p);
        if (e >= 0 && e < n_experts) atomicAdd(&count[(int)e], 1);
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        int before = 0;
        for (int e0 = 0; e0 < n_experts; e0 += 32) {
            const int e = e0 + (int)threadIdx.x, c = e < n_experts ? count[e] : 0;
            int t = c;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) { const int o = __shfl_up_sync(0xffffffffu, t, d); if ((int)threadIdx.x >= d) t += o; }
            if (e < n_experts) { next[e] = before + t - c; offs[e] = before + t - c; }
            before += __shfl_sync(0xffffffffu, t, 31);
        }
        if (threadIdx.x == 0) offs[n_experts] = before;
    }
    __syncthreads();
    for (int p = threadIdx.x; p < pairs; p += kSortThreads) {
        const long long e = id_at(p);
        int r = -1;                                            // an id outside the table contributes nothing
        if (e >= 0 && e < n_experts) { r = atomicAdd(&next[(int)e], 1); token_of[r] = p / top_k; }
        row_of[p] = r;
    }
}

// rows beyond the last routed one hold whatever the scratch held: nothing reads their products
__global__ void __launch_bounds__(256) experts_gather_kernel(const uint4* __restrict__ x, uint4* __restrict__ rows, const int* __restrict__ token_of,
                                                             const int* __restrict__ n_rows, int vec) {
    const int r = blockIdx.x;
    if (r >= *n_rows) return;
    const uint4* src = x + (int64_t)token_of[r] * vec;
    uint4* dst = rows + (int64_t)r * vec;
    for (int i = threadIdx.x; i < vec; i += 256) dst[i] = src[i];
}

template <bool BF>
__global__ void __launch_bounds__(256) experts_combine_kernel(const uint4* __restrict__ rows, const int* __restrict__ row_of, const void* __restrict__ weight,
                                                              int w_dtype, int top_k, uint4* __restrict__ y, int vec) {
    const int64_t t = blockIdx.x;
    for (int i = threadIdx.x; i < vec; i += 256) {
        float a[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        for (int s = 0; s < top_k; s++) {
            const int r = row_of[t * top_k + s];
            if (r < 0) continue;
            const float w = w_dtype == DT_F32 ? ((const float*)weight)[t * top_k + s] : w_dtype == DT_F16 ? __half2float(((const __half*)weight)[t * top_k + s])
                                                                                                        : __bfloat162float(((const __nv_bfloat16*)weight)[t * top_k + s]);
            const uint4 q = rows[(int64_t)r * vec + i];
            const uint32_t u[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                float lo, hi;
                if (BF) { lo = __uint_as_float(u[j] << 16); hi = __uint_as_float(u[j] & 0xffff0000u); }
                else { const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&u[j])); lo = f.x; hi = f.y; }
                a[2 * j] += w * lo; a[2 * j + 1] += w * hi;
            }
        }
        uint32_t o[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if (BF) { const __nv_bfloat162 b = __floats2bfloat162_rn(a[2 * j], a[2 * j + 1]); o[j] = *reinterpret_cast<const uint32_t*>(&b); }
            else { const __half2 h = __floats2half2_rn(a[2 * j], a[2 * j + 1]); o[j] = *reinterpret_cast<const uint32_t*>(&h); }
        }
        y[t * vec + i] = make_uint4(o[0], o[1], o[2], o[3]);
    }
}

struct ExpertsScratch { size_t view, row_of, token_of, x, h, out, total; };
ExpertsScratch experts_scratch(int64_t hidden, int64_t inter, int64_t pairs) {
    auto up = [](size_t b) { return (b + 255) / 256 * 256; };
    ExpertsScratch S;
    size_t at = 0;
    S.view = at; at += up(sizeof(HostView));
    S.row_of = at; at += up((size_t)pairs * 4);
    S.token_of = at; at += up((size_t)pairs * 4);
    S.x = at; at += up((size_t)pairs * hidden * 2);
    S.h = at; at += up((size_t)pairs * inter * 2);
    S.out = at; at += up((size_t)pairs * hidden * 2);
    S.total = at;
    return S;
}
// page-locked memory for one call's view, the calling thread's own (a call waits for the copy before it returns)
struct PinnedView {
    HostView* p = nullptr;
    HostView* get() {
        if (!p && cudaHostAlloc(&p, sizeof(HostView), cudaHostAllocPortable) != cudaSuccess) { cudaGetLastError(); p = nullptr; }
        return p;
    }
    ~PinnedView() { if (p) cudaFreeHost(p); }
};
thread_local PinnedView t_view;
thread_local int64_t t_unrouted = 0;

// the experts of few rows, whatever their number: weights exact
int experts_of_few_rows(const MoeParams& P, const HostView& V, char* x, char* h, char* out, cudaStream_t st) {
    for (int e = 0; e < P.n_experts; e++) {
        const int64_t lo = V.offs[e], n = V.offs[e + 1] - lo;
        if (n < 1 || n > kExactRows) continue;
        int rc = gemv_launch_ex((const void*)V.tab[0][e], (const void*)V.tab[1][e], P.act, P.qtype, P.inter, P.hidden, x + lo * P.hidden * 2, P.x_dtype, n,
                                h + lo * P.inter * 2, P.x_dtype, nullptr, 0, nullptr, 0, st);
        if (!rc) rc = gemv_launch((const void*)V.tab[2][e], P.qtype, P.hidden, P.inter, h + lo * P.inter * 2, P.x_dtype, n, out + lo * P.hidden * 2, P.x_dtype,
                                  nullptr, 0, nullptr, 0, st);
        if (rc) return rc;
    }
    return LB_OK;
}
}  // namespace

bool experts_supported(int qt, int64_t hidden, int64_t inter, int n_experts, int top_k) {
    return gemm_tc_supported(qt, inter, hidden) && gemm_tc_supported(qt, hidden, inter) && n_experts >= 1 && n_experts <= kSortExperts && top_k >= 1;
}
size_t experts_workspace_size(int64_t hidden, int64_t inter, int n_experts, int64_t n_tokens, int top_k) {
    (void)n_experts;
    return experts_scratch(hidden, inter, n_tokens * top_k).total;
}
int64_t experts_unrouted() { return t_unrouted; }
int experts_launch(const MoeParams& P, int64_t n_tokens, cudaStream_t st) {
    const int64_t pairs = n_tokens * P.top_k;
    t_unrouted = 0;
    if (!experts_supported(P.qtype, P.hidden, P.inter, P.n_experts, P.top_k) || pairs > 0x3fffffff || P.accumulate) return LB_ERR_ARG;
    if ((P.x_dtype != DT_F16 && P.x_dtype != DT_BF16) || P.y_dtype != P.x_dtype) return LB_ERR_ARG;
    if (((uintptr_t)P.x & 15) || ((uintptr_t)P.y & 15) || ((uintptr_t)P.workspace & 255)) return LB_ERR_ARG;
    const ExpertsScratch S = experts_scratch(P.hidden, P.inter, pairs);
    if (!P.workspace || P.workspace_bytes < S.total) return LB_ERR_WORKSPACE;
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &capture) != cudaSuccess || capture != cudaStreamCaptureStatusNone) { cudaGetLastError(); return LB_ERR_ARG; }
    HostView* const host = t_view.get();
    cudaEvent_t sorted = nullptr;
    if (!host || cudaEventCreateWithFlags(&sorted, cudaEventDisableTiming) != cudaSuccess) {
        cudaGetLastError();
        set_error(LB_ERR_CUDA, "lowbit_moe_tokens_cuda: no page-locked memory or event for the row counts");
        return LB_ERR_CUDA;
    }
    char* ws = (char*)P.workspace;
    HostView* const view = (HostView*)(ws + S.view);
    int *row_of = (int*)(ws + S.row_of), *token_of = (int*)(ws + S.token_of);
    char *x = ws + S.x, *h = ws + S.h, *out = ws + S.out;
    const int vec = (int)(P.hidden / 8);
    experts_sort_kernel<<<1, kSortThreads, 0, st>>>(P.ids, P.ids_i64, (int)pairs, P.top_k, P.n_experts, P.gates, P.ups, P.downs, view, row_of, token_of);
    cudaMemcpyAsync(host, view, sizeof(HostView), cudaMemcpyDeviceToHost, st);
    cudaEventRecord(sorted, st);
    experts_gather_kernel<<<(unsigned)pairs, 256, 0, st>>>((const uint4*)P.x, (uint4*)x, token_of, view->offs + P.n_experts, vec);
    note_launch(); note_launch();
    int rc = LB_OK;
    if (pairs > kExactRows) {
        rc = gemm_tc_experts_launch(P.gates, P.ups, P.act, view->offs, P.n_experts, P.qtype, P.inter, P.hidden, x, P.x_dtype, pairs, h, P.x_dtype, st);
        if (!rc) rc = gemm_tc_experts_launch(P.downs, nullptr, 0, view->offs, P.n_experts, P.qtype, P.hidden, P.inter, h, P.x_dtype, pairs, out, P.x_dtype, st);
    }
    const cudaError_t waited = cudaEventSynchronize(sorted);
    cudaEventDestroy(sorted);
    if (rc) return rc;
    if (waited != cudaSuccess) { set_error(LB_ERR_CUDA, "CUDA error: %s", cudaGetErrorString(waited)); cudaGetLastError(); return LB_ERR_CUDA; }
    t_unrouted = pairs - host->offs[P.n_experts];
    if ((rc = experts_of_few_rows(P, *host, x, h, out, st))) return rc;
    if (P.x_dtype == DT_BF16) experts_combine_kernel<true><<<(unsigned)n_tokens, 256, 0, st>>>((const uint4*)out, row_of, P.weights, P.w_dtype, P.top_k, (uint4*)P.y, vec);
    else experts_combine_kernel<false><<<(unsigned)n_tokens, 256, 0, st>>>((const uint4*)out, row_of, P.weights, P.w_dtype, P.top_k, (uint4*)P.y, vec);
    note_launch();
    return check_launch();
}

}  // namespace lowbit
