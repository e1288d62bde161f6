// lowbit_internal.h -- declarations shared between the .cu translation units of
// libb200lowbit.so (not installed; the public ABI is include/b200_lowbit.h).
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace lowbit {

enum {
    LB_OK = 0,
    LB_ERR_ARG = 1,        // bad qtype / shape / pointer combination
    LB_ERR_CUDA = 2,       // a CUDA runtime call failed (see last_error_string)
    LB_ERR_NO_DEVICE = 3,  // no usable CUDA device: there is no CPU fallback
    LB_ERR_WORKSPACE = 4,  // caller workspace too small
};

// per-thread error / launch bookkeeping (capi.cu)
void set_error(int code, const char* fmt, ...);
void note_launch();
void reset_launch_count();
int check_launch();   // cudaGetLastError() -> LB_OK / LB_ERR_CUDA (records the message)
int sm_count();       // SMs of the current device (cached per device)

// layout.cu
int relayout_launch(const void* src, void* dst, int64_t rows, int64_t k, int qt, bool to_device,
                    cudaStream_t st);
int dequant_canonical_launch(const void* src, void* dst, size_t n, int qt, int out_dtype, cudaStream_t st);
int dequant_tiled_launch(const void* src, void* dst, int64_t rows, int64_t k, int qt, int out_dtype,
                         cudaStream_t st);

int dequant_rows_launch(const void* src, void* dst, const void* ids, int ids_i64, int64_t n_ids, int64_t rows, int64_t k,
                        int qt, int out_dtype, cudaStream_t st);

// quantize.cu
int quantize_launch(const float* src, void* dst, int qt, size_t n, int k, int64_t* hist, bool scale_search,
                    cudaStream_t st);

// gemv.cu
void gemv_set_pdl(int on);
int gemv_get_pdl();
// Launches outside a recorded step overlap their starts: a kernel is launched as a programmatic dependent of the one in front and waits
// (griddepcontrol.wait) before it touches global memory, so that what it reads and overwrites is ordered as without.  That pays behind another
// call of the library, 1 to 2 us; a kernel of torch or a copy releases nothing before it ends.  Off the chain are the scheduling of the blocks
// and what stands in front of the wait: the barriers and TMEM of the kernel for 17 to 64 rows, nf4's table, barriers in the prompt matmul,
// little or nothing in the GEMV, both attentions and the delta rule.  The GEMV, the decode attention, the reductions and the delta rule
// release their dependents at their start, the prompt attention when it holds its TMEM, the others at their end or in their last unit.
// Who releases early has his TMEM by then (a dependent may allocate in front of its wait), and no parameter is const __restrict__.
// In a recorded step (the switch on) the launches of these kernels stay ordinary: kernels there read inputs ahead of their wait because an
// ordinary launch lies in front of them; and in a stream that is being captured the graph's edges are left as they were.
inline bool launch_overlaps(cudaStream_t st) {
    if (gemv_get_pdl()) return false;
    cudaStreamCaptureStatus state = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(st, &state) == cudaSuccess && state == cudaStreamCaptureStatusNone;
}
inline int add_overlap(cudaLaunchAttribute* at, int n, bool on) {
    if (!on) return n;
    at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[n].val.programmaticStreamSerializationAllowed = 1;
    return n + 1;
}
template <typename... P, typename... Q>
inline void launch_behind(void (*kern)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, bool overlap, Q... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = dim3((unsigned)threads); cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cudaLaunchAttribute at[1];
    cfg.attrs = at; cfg.numAttrs = add_overlap(at, 0, overlap);
    cudaLaunchKernelEx(&cfg, kern, P(args)...);
}
struct GemvPush;
void gemv_set_push(const GemvPush* p);   // the next gemv_launch_ex on this thread pushes its result to the peers (comm.cu)
void gemv_set_next_weights(const void* w, size_t bytes);
void gemv_set_debug_timestamps(void* p);
size_t gemv_workspace_size(int64_t n_rows, int64_t k, int64_t m, int x_dtype);
int gemv_launch(const void* w, int qt, int64_t n_rows, int64_t k, const void* x, int x_dtype, int64_t m,
                void* y, int y_dtype, const void* bias, int accumulate, void* workspace,
                size_t workspace_bytes, cudaStream_t st);

int gemv_launch_ex(const void* w, const void* w2, int act, int qt, int64_t n_rows, int64_t k, const void* x, int x_dtype,
                   int64_t m, void* y, int y_dtype, const void* bias, int accumulate, void* workspace,
                   size_t workspace_bytes, cudaStream_t st);
bool gemv_mlp_fused_supported(int qt, int64_t n_rows, int64_t k, int64_t m, int x_dtype);
int act_mul_launch(const float* gate, const float* up, void* y, int y_dtype, int64_t n, int act, cudaStream_t st);

// one-token mixture-of-experts (reference xe_linear.moe_forward_vec)
struct MoeParams {
    const void* x; int x_dtype;                  // [hidden]
    const void* ids; int ids_i64;                // [top_k] routed expert ids (device)
    const void* weights; int w_dtype;            // [top_k] routing weights (device)
    int top_k;
    const unsigned long long* gates;             // [n_experts] device addresses of the tiled [inter][hidden] weights
    const unsigned long long* ups;
    const unsigned long long* downs;             // ... of the tiled [hidden][inter] weights
    int n_experts;
    int64_t hidden, inter;
    int qtype, act;
    void* y; int y_dtype; int accumulate;        // [hidden]
    void* workspace; size_t workspace_bytes;
};
bool moe_supported(int qt, int64_t hidden, int64_t inter, int top_k);
size_t moe_workspace_size(int64_t hidden, int64_t inter, int top_k, int x_dtype);
int moe_launch(const MoeParams& P, cudaStream_t st);

// bounded waits of the prompt kernels: a wait that runs out writes the device's word, which lies in host memory, and the launch's results
// are undefined; the next check_launch() on the device reports and clears it
struct Waits { unsigned int* word; long long limit; };       // limit: SM clocks
int make_waits(Waits* w, long long limit);                   // the current device's, with this limit unless the calling thread has set one

// up to this many half-precision rows a product keeps the weights as code x scale in 32 bits (the GEMV); above, the tensor cores take them
// rounded once to the activation dtype.  Measured line: see use_skinny in capi.cu
constexpr int64_t kExactRows = 16;

// many-token mixture-of-experts (experts.cu): MoeParams with x / y [n_tokens][hidden], ids / weights [n_tokens][top_k]
bool experts_supported(int qt, int64_t hidden, int64_t inter, int n_experts, int top_k);
size_t experts_workspace_size(int64_t hidden, int64_t inter, int n_experts, int64_t n_tokens, int top_k);
int experts_launch(const MoeParams& P, int64_t n_tokens, cudaStream_t st);
int64_t experts_unrouted();       // pairs of the calling thread's last launch whose id was outside the table

// gemm_pair.cu (tcgen05 prompt matmul, two SMs per tile)
bool gemm_tc_supported(int qt, int64_t n_rows, int64_t k);
size_t gemm_tc_workspace_size(int64_t n_rows, int64_t k, int64_t m);
int gemm_tc_launch(const void* w, int qt, int64_t n_rows, int64_t k, const void* x, int x_dtype, int64_t m, void* y,
                   int y_dtype, const void* bias, int accumulate, void* workspace, size_t workspace_bytes, cudaStream_t st);
bool gemm_tc_grad_supported(int qt, int64_t n_rows, int64_t k);
size_t gemm_tc_grad_workspace_size(int64_t n_rows, int64_t k, int64_t m);
bool gemm_tc_grad_faster(int qt, int64_t n_rows, int64_t k, int64_t m);
int gemm_tc_grad_launch(const void* w, int qt, int64_t n_rows, int64_t k, const void* g, int dtype, int64_t m, void* dx, void* workspace,
                        size_t workspace_bytes, cudaStream_t st);
int gemm_tc_mlp_launch(const void* w_gate, const void* w_up, int act, int qt, int64_t n_rows, int64_t k, const void* x, int x_dtype,
                       int64_t m, void* y, int y_dtype, void* workspace, size_t workspace_bytes, cudaStream_t st);
size_t gemm_tc_mlp_workspace_size(int64_t n_rows, int64_t k, int64_t m);
int gemm_tc_experts_launch(const unsigned long long* tab, const unsigned long long* tab2, int act, const int* offs, int n_experts, int qt,
                           int64_t n_rows, int64_t k, const void* x, int x_dtype, int64_t rows, void* y, int y_dtype, cudaStream_t st);

// gemm_exact.cu (the fp32 prompt matmul: codes and activation planes exact on the tensor cores)
bool gemm_exact_supported(int qt, int64_t n_rows, int64_t k, int64_t m);
size_t gemm_exact_workspace_size(int qt, int64_t n_rows, int64_t k, int64_t m);
int gemm_exact_launch(const void* w, int qt, int64_t n_rows, int64_t k, const void* x, int64_t m, void* y, const void* bias, int accumulate,
                      void* workspace, size_t workspace_bytes, cudaStream_t st);

// M above this goes to the tensor-core GEMM when the shape allows, else to chunks of the GEMV
constexpr int64_t kGemvMaxM = 32;
// the tensor-core GEMM with the operands swapped (weights = the 128-row operand, tokens = N): 17 <= m <= 64
bool gemm_skinny_supported(int qt, int64_t n_rows, int64_t k, int64_t m, int x_dtype);
size_t gemm_skinny_workspace_size(int64_t n_rows, int64_t k, int64_t m);
size_t gemm_skinny_mlp_workspace_size(int64_t n_rows, int64_t k, int64_t m);
int gemm_skinny_mlp_launch(const void* w_gate, const void* w_up, int act, int qt, int64_t n_rows, int64_t k, const void* x, int x_dtype,
                           int64_t m, void* y, int y_dtype, void* workspace, size_t workspace_bytes, cudaStream_t st, int pdl);
int gemm_skinny_launch(const void* w, int qt, int64_t n_rows, int64_t k, const void* x, int x_dtype, int64_t m, void* y, int y_dtype,
                       const void* bias, int accumulate, void* workspace, size_t workspace_bytes, cudaStream_t st, int pdl);

}  // namespace lowbit
