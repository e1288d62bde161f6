// capi.cu -- the extern "C" surface declared in include/b200_lowbit.h.
//
// Family (1): reference-named symbols with host pointers (reference
// ggml/model/llama/llama_cpp.py:945-1185).  They stage through library-owned device buffers,
// run the same CUDA kernels as family (2) and copy the result back.  No CPU arithmetic: if
// CUDA is unusable the call records LB_ERR_NO_DEVICE and returns without writing.
// Family (2): *_cuda symbols on device pointers + stream.
#include <atomic>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <mutex>
#include "../../include/b200_lowbit.h"
#include "lowbit_common.cuh"
#include "lowbit_internal.h"

namespace lowbit {

static thread_local int t_err = 0;
static thread_local char t_msg[512] = "";
static thread_local int t_launches = 0;
static thread_local int t_row_len = 0;

void set_error(int code, const char* fmt, ...) {
    t_err = code;
    va_list ap; va_start(ap, fmt);
    vsnprintf(t_msg, sizeof(t_msg), fmt, ap);
    va_end(ap);
}
void note_launch() { t_launches++; }
void reset_launch_count() { t_launches = 0; }
// a word per device, each in a cache line of its own, in host memory that every device writes; never freed (recorded graphs hold it)
constexpr int kWaitStride = 32;
static std::atomic<unsigned int*> g_wait_words{nullptr};
static thread_local long long t_wait_limit = 0;
static unsigned int* wait_word() {
    unsigned int* const w = g_wait_words.load(std::memory_order_acquire);
    int dev = 0;
    return w && cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64 ? w + dev * kWaitStride : nullptr;
}
int make_waits(Waits* out, long long limit) {
    if (!g_wait_words.load(std::memory_order_acquire)) {
        static std::mutex mu;
        std::lock_guard<std::mutex> lk(mu);
        if (!g_wait_words.load(std::memory_order_relaxed)) {
            // the first launch may be one that is being captured: page-locking is no part of it
            cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
            cudaThreadExchangeStreamCaptureMode(&mode);
            void* p = nullptr;
            const cudaError_t e = cudaHostAlloc(&p, 64 * kWaitStride * sizeof(unsigned int), cudaHostAllocPortable | cudaHostAllocMapped);
            cudaThreadExchangeStreamCaptureMode(&mode);
            if (e != cudaSuccess) { set_error(LB_ERR_CUDA, "cudaHostAlloc failed: %s", cudaGetErrorString(e)); cudaGetLastError(); return LB_ERR_CUDA; }
            memset(p, 0, 64 * kWaitStride * sizeof(unsigned int));
            g_wait_words.store((unsigned int*)p, std::memory_order_release);
        }
    }
    out->word = wait_word();
    out->limit = t_wait_limit ? t_wait_limit : limit;
    if (!out->word) { set_error(LB_ERR_NO_DEVICE, "no current CUDA device"); return LB_ERR_NO_DEVICE; }
    return LB_OK;
}
int check_launch() {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { set_error(LB_ERR_CUDA, "CUDA error: %s", cudaGetErrorString(e)); return LB_ERR_CUDA; }
    unsigned int* const word = wait_word();
    if (word && *(volatile unsigned int*)word) {
        *(volatile unsigned int*)word = 0;
        set_error(LB_ERR_CUDA, "a wait inside an earlier prompt matmul or prompt attention on this device ran out: the results since then are undefined");
        return LB_ERR_CUDA;
    }
    return LB_OK;
}
int sm_count() {
    static int cached[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { cudaGetLastError(); return 148; }
    if (!cached[dev]) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) { cudaGetLastError(); n = 148; }
        cached[dev] = n;
    }
    return cached[dev];
}

static bool have_device() {
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || n <= 0) { cudaGetLastError(); return false; }
    return true;
}

// ---- library-owned per-device buffers: staging for family (1), default matmul workspace ----
struct DevBuf {
    void* p = nullptr; size_t cap = 0;
    int ensure(size_t bytes, bool zero_new) {
        if (bytes <= cap) return LB_OK;
        if (p) cudaFree(p);
        p = nullptr; cap = 0;
        size_t want = bytes + bytes / 8;
        cudaError_t e = cudaMalloc(&p, want);
        if (e != cudaSuccess) { set_error(LB_ERR_CUDA, "cudaMalloc(%zu) failed: %s", want, cudaGetErrorString(e)); cudaGetLastError(); return LB_ERR_CUDA; }
        cap = want;
        if (zero_new) cudaMemset(p, 0, want);
        return LB_OK;
    }
};
struct DevState { DevBuf in, out, aux, ws; };
static std::mutex g_mu;
static DevState g_dev[64];
static DevState* dev_state() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { cudaGetLastError(); return nullptr; }
    return &g_dev[dev];
}

#define HOST_PROLOGUE(retval)                                                              \
    t_launches = 0;                                                                        \
    if (!have_device()) {                                                                  \
        set_error(LB_ERR_NO_DEVICE, "%s: no CUDA device (this library has no CPU path)", __func__); \
        return retval;                                                                     \
    }                                                                                      \
    std::lock_guard<std::mutex> lk(g_mu);                                                  \
    DevState* S = dev_state();                                                             \
    if (!S) { set_error(LB_ERR_NO_DEVICE, "%s: cudaGetDevice failed", __func__); return retval; }

static bool cuda_ok(cudaError_t e, const char* what) {
    if (e == cudaSuccess) return true;
    set_error(LB_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
    cudaGetLastError();
    return false;
}

}  // namespace lowbit

using namespace lowbit;

extern "C" {

void llama_init_backend(void) {}

size_t ggml_type_size(int qtype) { return (size_t)type_size(qtype); }
int ggml_qk_size(int qtype) { return supported(qtype) ? QK : 0; }

int b200_lowbit_last_error(void) { return t_err; }
const char* b200_lowbit_last_error_string(void) { return t_msg; }
void b200_lowbit_clear_error(void) { t_err = 0; t_msg[0] = 0; }
int b200_lowbit_last_launch_count(void) { return t_launches; }
int b200_lowbit_sm_count(void) { return have_device() ? sm_count() : 0; }
void b200_lowbit_set_row_length(int k) { t_row_len = k; }
void lowbit_set_programmatic_dependent_launch(int on) { gemv_set_pdl(on); }
int lowbit_get_programmatic_dependent_launch(void) { return gemv_get_pdl(); }
void lowbit_hint_next_weights(const void* d_w, size_t bytes) { gemv_set_next_weights(d_w, bytes); }
/* development aid, not in the public header: per-warp phase timestamps of the GEMV kernel */
void lowbit_debug_set_timestamps(void* dev_ptr) { gemv_set_debug_timestamps(dev_ptr); }

// ------------------------------------------------------------------ family (2)
int ggml_quantize_tensor_cuda(const float* d_src, void* d_dst, int qtype, size_t n, int k, int64_t* d_hist,
                              bool scale_search, void* stream) {
    t_launches = 0;
    int rc = quantize_launch(d_src, d_dst, qtype, n, k, d_hist, scale_search, (cudaStream_t)stream);
    if (rc == LB_ERR_ARG) set_error(rc, "ggml_quantize_tensor_cuda: bad argument (qtype %d, n %zu, k %d)", qtype, n, k);
    return rc;
}

int ggml_dequantize_cuda(const void* d_src, void* d_dst, size_t k, int qtype, int out_dtype, void* stream) {
    t_launches = 0;
    int rc = dequant_canonical_launch(d_src, d_dst, k, qtype, out_dtype, (cudaStream_t)stream);
    if (rc == LB_ERR_ARG) set_error(rc, "ggml_dequantize_cuda: bad argument (qtype %d, k %zu)", qtype, k);
    return rc;
}

int lowbit_dequantize_device_layout_cuda(const void* d_src, void* d_dst, int64_t rows, int64_t k, int qtype,
                                         int out_dtype, void* stream) {
    t_launches = 0;
    int rc = dequant_tiled_launch(d_src, d_dst, rows, k, qtype, out_dtype, (cudaStream_t)stream);
    if (rc == LB_ERR_ARG) set_error(rc, "lowbit_dequantize_device_layout_cuda: bad argument");
    return rc;
}

int lowbit_dequantize_rows_cuda(const void* d_w, int qtype, int64_t rows, int64_t k, const void* d_ids, int ids_dtype,
                                int64_t n_ids, void* d_out, int out_dtype, void* stream) {
    t_launches = 0;
    if (!d_w || (n_ids > 0 && (!d_ids || !d_out)) || (ids_dtype != 0 && ids_dtype != 1)) {
        set_error(LB_ERR_ARG, "lowbit_dequantize_rows_cuda: null pointer or bad ids_dtype");
        return LB_ERR_ARG;
    }
    int rc = dequant_rows_launch(d_w, d_out, d_ids, ids_dtype, n_ids, rows, k, qtype, out_dtype, (cudaStream_t)stream);
    if (rc == LB_ERR_ARG) set_error(rc, "lowbit_dequantize_rows_cuda: bad argument (rows %lld, k %lld, qtype %d)", (long long)rows, (long long)k, qtype);
    return rc;
}

int lowbit_relayout_cuda(const void* d_src, void* d_dst, int64_t rows, int64_t k, int qtype, int to_device,
                         void* stream) {
    t_launches = 0;
    int rc = relayout_launch(d_src, d_dst, rows, k, qtype, to_device != 0, (cudaStream_t)stream);
    if (rc == LB_ERR_ARG) set_error(rc, "lowbit_relayout_cuda: bad argument (rows %lld, k %lld, qtype %d)", (long long)rows, (long long)k, qtype);
    return rc;
}

// fp32 activations never take this kernel: it rounds them to one 16-bit value, while their contract keeps them to 2^-24 (three bf16
// planes) -- the fp32-in / fp32-out contract of ggml_compute_forward_mul_mat_q_fp32 (LBL:494-529), on the GEMV or in gemm_exact.cu.  A
// caller that accepts half precision casts first, as the reference's XPU path does (LBL:700-705, conver_to_half).
static bool use_gemm(int qtype, int64_t n_rows, int64_t k, int64_t m, int x_dtype) {
    static const int64_t max_m = [] { const char* e = getenv("LOWBIT_GEMV_MAX_M"); return e ? (int64_t)atoi(e) : kGemvMaxM; }();   // development
    return x_dtype != DT_F32 && m > max_m && gemm_tc_supported(qtype, n_rows, k);
}

// fp32 rows beyond one pass of the GEMV, fp32 results: the same arithmetic on pairs of SMs (gemm_exact.cu), in every format.
// The line lies at the GEMV's 32 rows: at 33 rows, two passes against one launch, 33.8 -> 17.4 us at 4096 x 4096, 18.2 -> 12.4 at 1024 x 1024
static bool use_exact(int qtype, int64_t n_rows, int64_t k, int64_t m, int x_dtype, int y_dtype) {
    return x_dtype == DT_F32 && y_dtype == DT_F32 && m > kGemvMaxM && gemm_exact_supported(qtype, n_rows, k, m);
}

// Batches between the GEMV's best range and a full 128-token tile take the tensor-core kernel with the operands swapped
// (gemm_skinny_launch): weights rounded once to the activation dtype, the prefill kernel's precision contract.
// The window is 17..64 rows, in every format (fresh weights, back to back): 11008 x 4096 in sym_int4, this kernel against the GEMV 13.0 / 23.2 us at 17
// rows and 13.3 / 24.3 at 32, against the prompt kernel 13.7 / 19.0 at 33, 15.3 / 19.0 at 64 and, in 128 columns, 21.7 / 19.8 at 65;
// fp8_e4m3 15.4 / 20.9, 15.6 / 22.0, 15.9 / 18.7, 16.9 / 18.9, 20.7 / 19.8.  At 9 to 16 rows the GEMV takes 13.5 us against 12.8 there, 8.7 against 9.6
// at 4096 x 4096 and 4.5 against 6.9 at 1024 x 1024.
// LOWBIT_SKINNY_MIN_M / LOWBIT_SKINNY_MAX_M (development) move the window, up to 64 rows; MIN_M above MAX_M switches the kernel off.
static bool use_skinny(int qtype, int64_t n_rows, int64_t k, int64_t m, int x_dtype) {
    static const int64_t min_m = [] { const char* e = getenv("LOWBIT_SKINNY_MIN_M"); return e ? (int64_t)atoi(e) : kExactRows + 1; }();
    static const int64_t max_m = [] { const char* e = getenv("LOWBIT_SKINNY_MAX_M"); return e ? (int64_t)atoi(e) : (int64_t)64; }();
    return m >= min_m && m <= max_m && gemm_skinny_supported(qtype, n_rows, k, m, x_dtype);
}

static size_t matmul_workspace(int qtype, int64_t n_rows, int64_t k, int64_t m, int x_dtype) {
    if (use_skinny(B200_QT_SYM_INT4, n_rows, k, m, x_dtype)) return gemm_skinny_workspace_size(n_rows, k, m);
    if (use_gemm(B200_QT_SYM_INT4, n_rows, k, m, x_dtype)) return gemm_tc_workspace_size(n_rows, k, m);
    const size_t gemv = gemv_workspace_size(n_rows, k, m, x_dtype);
    if (!use_exact(B200_QT_SYM_INT4, n_rows, k, m, x_dtype, DT_F32)) return gemv;
    const size_t exact = gemm_exact_workspace_size(qtype, n_rows, k, m);
    return exact > gemv ? exact : gemv;
}
// asked without the format: enough for each, asym_int4's sums of activations among them
size_t lowbit_matmul_workspace_size(int64_t n_rows, int64_t k, int64_t m, int x_dtype) { return matmul_workspace(B200_QT_ASYM_INT4, n_rows, k, m, x_dtype); }

static int matmul_dispatch(const void* d_w, int qtype, int64_t n_rows, int64_t k, const void* d_x, int x_dtype, int64_t m,
                           void* d_y, int y_dtype, const void* d_bias, int accumulate, void* workspace, size_t workspace_bytes,
                           cudaStream_t st) {
    if (use_skinny(qtype, n_rows, k, m, x_dtype))
        return gemm_skinny_launch(d_w, qtype, n_rows, k, d_x, x_dtype, m, d_y, y_dtype, d_bias, accumulate, workspace,
                                  workspace_bytes, st, launch_overlaps(st) ? 2 : gemv_get_pdl());
    if (use_gemm(qtype, n_rows, k, m, x_dtype))
        return gemm_tc_launch(d_w, qtype, n_rows, k, d_x, x_dtype, m, d_y, y_dtype, d_bias, accumulate, workspace, workspace_bytes, st);
    // a caller's scratch of the GEMV's size still runs its chunks of 32 rows
    if (use_exact(qtype, n_rows, k, m, x_dtype, y_dtype) && workspace && workspace_bytes >= gemm_exact_workspace_size(qtype, n_rows, k, m) &&
        !(((uintptr_t)d_x | (uintptr_t)d_w | (uintptr_t)workspace) & 15))
        return gemm_exact_launch(d_w, qtype, n_rows, k, d_x, m, d_y, d_bias, accumulate, workspace, workspace_bytes, st);
    return gemv_launch(d_w, qtype, n_rows, k, d_x, x_dtype, m, d_y, y_dtype, d_bias, accumulate, workspace, workspace_bytes, st);
}

int lowbit_matmul_cuda(const void* d_w, int qtype, int64_t n_rows, int64_t k, const void* d_x, int x_dtype,
                       int64_t m, void* d_y, int y_dtype, const void* d_bias, int accumulate, void* workspace,
                       size_t workspace_bytes, void* stream) {
    t_launches = 0;
    if (m == 0 || n_rows == 0) return LB_OK;
    std::unique_lock<std::mutex> lk(g_mu, std::defer_lock);
    if (!workspace) {
        lk.lock();
        DevState* S = dev_state();
        if (!S) { set_error(LB_ERR_NO_DEVICE, "lowbit_matmul_cuda: no CUDA device"); return LB_ERR_NO_DEVICE; }
        const size_t need = lowbit_matmul_workspace_size(n_rows, k, m, x_dtype);
        if (need > S->ws.cap) {
            // growing frees the old buffer: wait for work that may still use it
            cudaDeviceSynchronize();
            int rc = S->ws.ensure(need, true);
            if (rc) return rc;
        }
        workspace = S->ws.p; workspace_bytes = S->ws.cap;
    }
    int rc = matmul_dispatch(d_w, qtype, n_rows, k, d_x, x_dtype, m, d_y, y_dtype, d_bias, accumulate, workspace,
                             workspace_bytes, (cudaStream_t)stream);
    if (rc == LB_ERR_ARG) set_error(rc, "lowbit_matmul_cuda: bad argument (qtype %d, N %lld, K %lld, M %lld)", qtype, (long long)n_rows, (long long)k, (long long)m);
    if (rc == LB_ERR_WORKSPACE) set_error(rc, "lowbit_matmul_cuda: workspace too small (%zu bytes)", workspace_bytes);
    return rc;
}

int lowbit_matmul_grad_supported(int qtype, int64_t n_rows, int64_t k) { return gemm_tc_grad_supported(qtype, n_rows, k) ? 1 : 0; }
int lowbit_matmul_grad_faster(int qtype, int64_t n_rows, int64_t k, int64_t m) {
    return gemm_tc_grad_supported(qtype, n_rows, k) && m > 0 && gemm_tc_grad_faster(qtype, n_rows, k, m) ? 1 : 0;
}
size_t lowbit_matmul_grad_workspace_size(int64_t n_rows, int64_t k, int64_t m) { return gemm_tc_grad_workspace_size(n_rows, k, m); }
int lowbit_matmul_grad_cuda(const void* d_w, int qtype, int64_t n_rows, int64_t k, const void* d_grad, int dtype, int64_t m, void* d_out,
                            void* workspace, size_t workspace_bytes, void* stream) {
    t_launches = 0;
    if (m == 0) return LB_OK;
    const int rc = !d_w || !d_grad || !d_out || m < 0 || m > 0x7fffffff ? LB_ERR_ARG
                 : gemm_tc_grad_launch(d_w, qtype, n_rows, k, d_grad, dtype, m, d_out, workspace, workspace_bytes, (cudaStream_t)stream);
    if (rc == LB_ERR_ARG) set_error(rc, "lowbit_matmul_grad_cuda: bad argument (qtype %d, N %lld, K %lld, M %lld)", qtype, (long long)n_rows, (long long)k, (long long)m);
    return rc;
}

size_t lowbit_mlp_workspace_size(int64_t n_rows, int64_t k, int64_t m, int x_dtype) {
    if (use_skinny(B200_QT_SYM_INT4, n_rows, k, m, x_dtype)) return gemm_skinny_mlp_workspace_size(n_rows, k, m);
    if (use_gemm(B200_QT_SYM_INT4, n_rows, k, m, x_dtype)) return gemm_tc_mlp_workspace_size(n_rows, k, m);
    const size_t base = (lowbit_matmul_workspace_size(n_rows, k, m, x_dtype) + 255) / 256 * 256;
    return base + 2 * (size_t)m * n_rows * sizeof(float);
}

int lowbit_mlp_cuda(const void* d_w_gate, const void* d_w_up, int qtype, int64_t n_rows, int64_t k, const void* d_x,
                    int x_dtype, int64_t m, void* d_y, int y_dtype, int act, void* workspace, size_t workspace_bytes,
                    void* stream) {
    t_launches = 0;
    if (m == 0 || n_rows == 0) return LB_OK;
    if (act != 0 && act != 1) { set_error(LB_ERR_ARG, "lowbit_mlp_cuda: act must be 0 (SILU) or 1 (GELU), got %d", act); return LB_ERR_ARG; }
    if (!d_w_gate || !d_w_up || !d_x || !d_y || m < 0 || n_rows < 0) { set_error(LB_ERR_ARG, "lowbit_mlp_cuda: null pointer or negative size"); return LB_ERR_ARG; }
    const bool fused = gemv_mlp_fused_supported(qtype, n_rows, k, m, x_dtype);
    // 32-bit prompts: in every format a workspace without room for asym_int4's sums of activations is enough, and asym_int4 then runs as it
    // does in lowbit_matmul_cuda without them
    const size_t parts = 2 * (size_t)m * n_rows * sizeof(float), full = lowbit_mlp_workspace_size(n_rows, k, m, x_dtype);
    size_t base = (matmul_workspace(qtype, n_rows, k, m, x_dtype) + 255) / 256 * 256;
    const size_t least = (matmul_workspace(B200_QT_SYM_INT4, n_rows, k, m, x_dtype) + 255) / 256 * 256;
    const size_t need = fused ? base : x_dtype == DT_F32 ? least + parts : full;
    std::unique_lock<std::mutex> lk(g_mu, std::defer_lock);
    if (!workspace) {
        lk.lock();
        DevState* S = dev_state();
        if (!S) { set_error(LB_ERR_NO_DEVICE, "lowbit_mlp_cuda: no CUDA device"); return LB_ERR_NO_DEVICE; }
        if ((fused ? need : full) > S->ws.cap) {
            cudaDeviceSynchronize();
            int rc = S->ws.ensure(fused ? need : full, true);
            if (rc) return rc;
        }
        workspace = S->ws.p; workspace_bytes = S->ws.cap;
    } else if (workspace_bytes < need) {
        set_error(LB_ERR_WORKSPACE, "lowbit_mlp_cuda: workspace too small (%zu < %zu bytes)", workspace_bytes, need);
        return LB_ERR_WORKSPACE;
    }
    cudaStream_t st = (cudaStream_t)stream;
    int rc;
    if (fused) {
        rc = gemv_launch_ex(d_w_gate, d_w_up, act + 1, qtype, n_rows, k, d_x, x_dtype, m, d_y, y_dtype, nullptr, 0, workspace,
                            workspace_bytes, st);
    } else if (use_skinny(qtype, n_rows, k, m, x_dtype)) {
        // 17..64 half-precision rows: both matrices in one pass of the skinny tensor-core kernel, act * up in its reduction launch
        rc = gemm_skinny_mlp_launch(d_w_gate, d_w_up, act + 1, qtype, n_rows, k, d_x, x_dtype, m, d_y, y_dtype, workspace, workspace_bytes,
                                    st, launch_overlaps(st) ? 2 : gemv_get_pdl());
    } else if (use_gemm(qtype, n_rows, k, m, x_dtype)) {
        rc = gemm_tc_mlp_launch(d_w_gate, d_w_up, act + 1, qtype, n_rows, k, d_x, x_dtype, m, d_y, y_dtype, workspace, workspace_bytes, st);
    } else {
        // behind the exact GEMV: the two intermediates in fp32
        if (workspace_bytes < base + parts) base = least;
        float* tg = (float*)((char*)workspace + base);
        float* tu = tg + (size_t)m * n_rows;
        rc = matmul_dispatch(d_w_gate, qtype, n_rows, k, d_x, x_dtype, m, tg, DT_F32, nullptr, 0, workspace, base, st);
        if (!rc) rc = matmul_dispatch(d_w_up, qtype, n_rows, k, d_x, x_dtype, m, tu, DT_F32, nullptr, 0, workspace, base, st);
        if (!rc) rc = act_mul_launch(tg, tu, d_y, y_dtype, m * n_rows, act + 1, st);
    }
    if (rc == LB_ERR_ARG) set_error(rc, "lowbit_mlp_cuda: bad argument (qtype %d, N %lld, K %lld, M %lld)", qtype, (long long)n_rows, (long long)k, (long long)m);
    if (rc == LB_ERR_WORKSPACE) set_error(rc, "lowbit_mlp_cuda: workspace too small (%zu bytes)", workspace_bytes);
    return rc;
}

int lowbit_moe_supported(int qtype, int64_t hidden, int64_t inter, int top_k) {
    return moe_supported(qtype, hidden, inter, top_k) ? 1 : 0;
}

size_t lowbit_moe_workspace_size(int64_t hidden, int64_t inter, int top_k, int x_dtype) {
    return moe_workspace_size(hidden, inter, top_k, x_dtype);
}

int lowbit_moe_cuda(const void* d_x, int x_dtype, const void* d_topk_ids, int ids_dtype, const void* d_topk_weight,
                    int weight_dtype, int top_k, const uint64_t* d_gates, const uint64_t* d_ups, const uint64_t* d_downs,
                    int n_experts, int64_t hidden, int64_t inter, int qtype, int act, void* d_y, int y_dtype, int accumulate,
                    void* workspace, size_t workspace_bytes, void* stream) {
    t_launches = 0;
    if (!d_x || !d_topk_ids || !d_topk_weight || !d_gates || !d_ups || !d_downs || !d_y || n_experts <= 0 ||
        (ids_dtype != 0 && ids_dtype != 1) || (act != 0 && act != 1)) {
        set_error(LB_ERR_ARG, "lowbit_moe_cuda: null pointer, bad ids_dtype / act or n_experts <= 0");
        return LB_ERR_ARG;
    }
    if (!moe_supported(qtype, hidden, inter, top_k)) {
        set_error(LB_ERR_ARG, "lowbit_moe_cuda: unsupported problem (qtype %d, hidden %lld, inter %lld, top_k %d)", qtype,
                  (long long)hidden, (long long)inter, top_k);
        return LB_ERR_ARG;
    }
    const size_t need = moe_workspace_size(hidden, inter, top_k, x_dtype);
    std::unique_lock<std::mutex> lk(g_mu, std::defer_lock);
    if (!workspace) {
        lk.lock();
        DevState* S = dev_state();
        if (!S) { set_error(LB_ERR_NO_DEVICE, "lowbit_moe_cuda: no CUDA device"); return LB_ERR_NO_DEVICE; }
        if (need > S->ws.cap) {
            cudaDeviceSynchronize();
            int rc = S->ws.ensure(need, true);
            if (rc) return rc;
        }
        workspace = S->ws.p; workspace_bytes = S->ws.cap;
    }
    MoeParams P;
    P.x = d_x; P.x_dtype = x_dtype; P.ids = d_topk_ids; P.ids_i64 = ids_dtype; P.weights = d_topk_weight; P.w_dtype = weight_dtype;
    P.top_k = top_k; P.gates = (const unsigned long long*)d_gates; P.ups = (const unsigned long long*)d_ups;
    P.downs = (const unsigned long long*)d_downs; P.n_experts = n_experts; P.hidden = hidden; P.inter = inter;
    P.qtype = qtype; P.act = act + 1; P.y = d_y; P.y_dtype = y_dtype; P.accumulate = accumulate;
    P.workspace = workspace; P.workspace_bytes = workspace_bytes;
    int rc = moe_launch(P, (cudaStream_t)stream);
    if (rc == LB_ERR_ARG) set_error(rc, "lowbit_moe_cuda: bad argument (dtype codes or alignment)");
    if (rc == LB_ERR_WORKSPACE) set_error(rc, "lowbit_moe_cuda: workspace too small (%zu < %zu bytes)", workspace_bytes, need);
    return rc;
}

int lowbit_moe_tokens_supported(int qtype, int64_t hidden, int64_t inter, int n_experts, int top_k) {
    return experts_supported(qtype, hidden, inter, n_experts, top_k) ? 1 : 0;
}

size_t lowbit_moe_tokens_workspace_size(int64_t hidden, int64_t inter, int n_experts, int64_t n_tokens, int top_k) {
    return experts_workspace_size(hidden, inter, n_experts, n_tokens, top_k);
}

int lowbit_moe_tokens_cuda(const void* d_x, int x_dtype, int64_t n_tokens, const void* d_topk_ids, int ids_dtype, const void* d_topk_weight,
                           int weight_dtype, int top_k, const uint64_t* d_gates, const uint64_t* d_ups, const uint64_t* d_downs,
                           int n_experts, int64_t hidden, int64_t inter, int qtype, int act, void* d_y, void* workspace,
                           size_t workspace_bytes, void* stream) {
    t_launches = 0;
    if (n_tokens == 0) return LB_OK;
    if (!d_x || !d_topk_ids || !d_topk_weight || !d_gates || !d_ups || !d_downs || !d_y || n_experts <= 0 || n_tokens < 0 ||
        (ids_dtype != 0 && ids_dtype != 1) || (act != 0 && act != 1) || weight_dtype < 0 || weight_dtype > 2) {
        set_error(LB_ERR_ARG, "lowbit_moe_tokens_cuda: null pointer, bad ids_dtype / weight_dtype / act, n_tokens < 0 or n_experts <= 0");
        return LB_ERR_ARG;
    }
    if (!experts_supported(qtype, hidden, inter, n_experts, top_k)) {
        set_error(LB_ERR_ARG, "lowbit_moe_tokens_cuda: unsupported problem (qtype %d, hidden %lld, inter %lld, %d experts, top_k %d)", qtype,
                  (long long)hidden, (long long)inter, n_experts, top_k);
        return LB_ERR_ARG;
    }
    MoeParams P = {};
    P.x = d_x; P.x_dtype = x_dtype; P.ids = d_topk_ids; P.ids_i64 = ids_dtype; P.weights = d_topk_weight; P.w_dtype = weight_dtype;
    P.top_k = top_k; P.gates = (const unsigned long long*)d_gates; P.ups = (const unsigned long long*)d_ups;
    P.downs = (const unsigned long long*)d_downs; P.n_experts = n_experts; P.hidden = hidden; P.inter = inter;
    P.qtype = qtype; P.act = act + 1; P.y = d_y; P.y_dtype = x_dtype;
    P.workspace = workspace; P.workspace_bytes = workspace_bytes;
    const int rc = experts_launch(P, n_tokens, (cudaStream_t)stream);
    if (rc == LB_ERR_ARG) set_error(rc, "lowbit_moe_tokens_cuda: bad argument (dtype codes or alignment), or the stream is being captured");
    if (rc == LB_ERR_WORKSPACE) set_error(rc, "lowbit_moe_tokens_cuda: workspace too small (%zu bytes)", workspace_bytes);
    return rc;
}

int64_t lowbit_moe_tokens_last_unrouted(void) { return experts_unrouted(); }

int lowbit_gemm_wait_expired(void) {
    if (cudaDeviceSynchronize() != cudaSuccess) { cudaGetLastError(); return -1; }
    const unsigned int* const word = wait_word();
    return word && *(const volatile unsigned int*)word ? 1 : 0;
}
/* development aid, not in the public header: the limit, in SM clocks, of the waits in this thread's launches (0: the usual one; below
 * zero: the launches' copies stop half-way, and the waits for them run out after that many clocks) */
void lowbit_debug_set_wait_limit(long long clocks) { t_wait_limit = clocks; }

// ------------------------------------------------------------------ family (1)
size_t ggml_quantize_tensor(const float* src, void* dst, int qtype, size_t n, int k, int64_t* hist,
                            bool scale_search) {
    HOST_PROLOGUE(0)
    const int bs = type_size(qtype);
    if (!bs || k <= 0 || k % QK || n % QK) { set_error(LB_ERR_ARG, "ggml_quantize_tensor: bad argument (qtype %d, n %zu, k %d)", qtype, n, k); return 0; }
    const size_t out_bytes = n / QK * bs;
    if (n == 0) return 0;
    if (S->in.ensure(n * sizeof(float), false) || S->out.ensure(out_bytes, false) || S->aux.ensure(256, false)) return 0;
    if (!cuda_ok(cudaMemcpy(S->in.p, src, n * sizeof(float), cudaMemcpyHostToDevice), "H2D")) return 0;
    if (quantize_launch((const float*)S->in.p, S->out.p, qtype, n, k, hist ? (int64_t*)S->aux.p : nullptr, scale_search, 0)) return 0;
    if (!cuda_ok(cudaMemcpy(dst, S->out.p, out_bytes, cudaMemcpyDeviceToHost), "D2H")) return 0;
    if (hist && !cuda_ok(cudaMemcpy(hist, S->aux.p, 16 * sizeof(int64_t), cudaMemcpyDeviceToHost), "D2H hist")) return 0;
    return out_bytes;
}

void ggml_dequantize(const void* src, void* dst, size_t k, int qtype) {
    HOST_PROLOGUE()
    const int bs = type_size(qtype);
    if (!bs || k % QK) { set_error(LB_ERR_ARG, "ggml_dequantize: bad argument (qtype %d, k %zu)", qtype, k); return; }
    if (k == 0) return;
    const size_t in_bytes = k / QK * bs;
    if (S->in.ensure(in_bytes, false) || S->out.ensure(k * sizeof(float), false)) return;
    if (!cuda_ok(cudaMemcpy(S->in.p, src, in_bytes, cudaMemcpyHostToDevice), "H2D")) return;
    if (dequant_canonical_launch(S->in.p, S->out.p, k, qtype, DT_F32, 0)) return;
    cuda_ok(cudaMemcpy(dst, S->out.p, k * sizeof(float), cudaMemcpyDeviceToHost), "D2H");
}

void ggml_dequantize_q4_0(const void* src, void* dst, size_t k) { ggml_dequantize(src, dst, k, QT_SYM_INT4); }

static int relayout_host(const void* src, void* dst, int64_t rows, int64_t k, int qtype, bool to_device, const char* who) {
    HOST_PROLOGUE(LB_ERR_NO_DEVICE)
    const int bs = type_size(qtype);
    if (!bs || k <= 0 || k % QK || rows <= 0) { set_error(LB_ERR_ARG, "%s: bad argument (rows %lld, k %lld, qtype %d)", who, (long long)rows, (long long)k, qtype); return LB_ERR_ARG; }
    const size_t bytes = (size_t)rows * (k / QK) * bs;
    if (S->in.ensure(bytes, false) || S->out.ensure(bytes, false)) return LB_ERR_CUDA;
    if (!cuda_ok(cudaMemcpy(S->in.p, src, bytes, cudaMemcpyHostToDevice), "H2D")) return LB_ERR_CUDA;
    int rc = relayout_launch(S->in.p, S->out.p, rows, k, qtype, to_device, 0);
    if (rc) return rc;
    if (!cuda_ok(cudaMemcpy(dst, S->out.p, bytes, cudaMemcpyDeviceToHost), "D2H")) return LB_ERR_CUDA;
    return LB_OK;
}

int ggml_q_format_convert_cpu2cuda_2d(const void* src, void* dst, int64_t rows, int64_t k, int qtype) {
    return relayout_host(src, dst, rows, k, qtype, true, "ggml_q_format_convert_cpu2cuda_2d");
}
int ggml_q_format_convert_cuda2cpu_2d(const void* src, void* dst, int64_t rows, int64_t k, int qtype) {
    return relayout_host(src, dst, rows, k, qtype, false, "ggml_q_format_convert_cuda2cpu_2d");
}

static void relayout_shapeless(const void* src, void* dst, size_t n, int qtype, bool to_device, const char* who) {
    const int k = t_row_len;
    if (k <= 0 || n % (size_t)k) {
        set_error(LB_ERR_ARG, "%s: the B200 device layout is tiled by rows; call b200_lowbit_set_row_length(k) first "
                  "(n = %zu, registered row length = %d)", who, n, k);
        return;
    }
    relayout_host(src, dst, (int64_t)(n / (size_t)k), k, qtype, to_device, who);
}
void ggml_q_format_convet_cpu2xpu(const void* src, void* dst, size_t n, int qtype) {
    relayout_shapeless(src, dst, n, qtype, true, "ggml_q_format_convet_cpu2xpu");
}
void ggml_q_format_convet_xpu2cpu(const void* src, void* dst, size_t n, int qtype) {
    relayout_shapeless(src, dst, n, qtype, false, "ggml_q_format_convet_xpu2cpu");
}

void ggml_compute_forward_mul_mat_q_fp32(const int64_t* src0_ne, const void* w, int qtype, const int64_t* src1_ne,
                                         const void* x, void* result) {
    HOST_PROLOGUE()
    const int64_t K = src0_ne[0], N = src0_ne[1], M = src1_ne[1];
    const int bs = type_size(qtype);
    if (!bs || K <= 0 || K % QK || src1_ne[0] != K || N <= 0 || M < 0) {
        set_error(LB_ERR_ARG, "ggml_compute_forward_mul_mat_q_fp32: bad shapes (K %lld, N %lld, M %lld, qtype %d)", (long long)K, (long long)N, (long long)M, qtype);
        return;
    }
    if (M == 0) return;
    const size_t w_bytes = (size_t)N * (K / QK) * bs, x_bytes = (size_t)M * K * 4, y_bytes = (size_t)M * N * 4;
    const size_t ws_bytes = lowbit_matmul_workspace_size(N, K, M, DT_F32);
    // in: [canonical w][x]   out: [tiled w]   aux: y
    const size_t w_al = (w_bytes + 255) / 256 * 256;
    if (S->in.ensure(w_al + x_bytes, false) || S->out.ensure(w_bytes, false) || S->aux.ensure(y_bytes, false)) return;
    if (ws_bytes > S->ws.cap) { cudaDeviceSynchronize(); if (S->ws.ensure(ws_bytes, true)) return; }
    if (!cuda_ok(cudaMemcpy(S->in.p, w, w_bytes, cudaMemcpyHostToDevice), "H2D w")) return;
    if (!cuda_ok(cudaMemcpy((char*)S->in.p + w_al, x, x_bytes, cudaMemcpyHostToDevice), "H2D x")) return;
    if (relayout_launch(S->in.p, S->out.p, N, K, qtype, true, 0)) return;
    if (matmul_dispatch(S->out.p, qtype, N, K, (char*)S->in.p + w_al, DT_F32, M, S->aux.p, DT_F32, nullptr, 0, S->ws.p, S->ws.cap, 0)) {
        if (!t_err) set_error(LB_ERR_CUDA, "ggml_compute_forward_mul_mat_q_fp32: launch failed");
        return;
    }
    cuda_ok(cudaMemcpy(result, S->aux.p, y_bytes, cudaMemcpyDeviceToHost), "D2H y");
}

}  // extern "C"
