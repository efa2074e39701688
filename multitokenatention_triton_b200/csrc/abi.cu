// C ABI of the library: argument validation, error text, and dispatch to the kernel launchers.
// See include/mta_b200.h for the contract of every entry point.
#include <atomic>
#include <cstring>
#include <string>

#include "kernels.cuh"

namespace mta {
namespace {
thread_local char g_error[512] = "";
thread_local long g_launches = 0;
// Kernel selection for tests and measurements: process-wide, read on every launch, written by mta_set_variant from any
// thread (relaxed atomics: a launch sees either the old or the new value of each key, never a torn one).
std::atomic<int> g_variant_head_linear{0}, g_variant_conv2d{0}, g_variant_gemm{0}, g_variant_fused{0}, g_variant_mix_softmax{0};
}  // namespace

void set_error(const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_error, sizeof(g_error), fmt, ap);
    va_end(ap);
}

void count_launch(int n) { g_launches += n; }

int variant(const char* key) {
    if (!strcmp(key, "head_linear")) return g_variant_head_linear.load(std::memory_order_relaxed);
    if (!strcmp(key, "conv2d")) return g_variant_conv2d.load(std::memory_order_relaxed);
    if (!strcmp(key, "gemm")) return g_variant_gemm.load(std::memory_order_relaxed);
    if (!strcmp(key, "fused")) return g_variant_fused.load(std::memory_order_relaxed);
    if (!strcmp(key, "mix_softmax")) return g_variant_mix_softmax.load(std::memory_order_relaxed);
    return 0;
}

int check_device() {
    int dev = 0;
    MTA_CUDA_OK(cudaGetDevice(&dev));
    static std::atomic<int> known[MAX_DEVICES_KNOWN];         // major compute capability, 0 = not looked up yet
    int major = dev < MAX_DEVICES_KNOWN ? known[dev].load(std::memory_order_relaxed) : 0;
    if (major == 0) {
        MTA_CUDA_OK(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev));
        if (dev < MAX_DEVICES_KNOWN) known[dev].store(major, std::memory_order_relaxed);
    }
    if (major != 10) {
        set_error("device %d has compute capability %d.x; this library is built for sm_100a only", dev, major);
        return MTA_ERR_ARCH;
    }
    if (wait_flag_raised()) {
        set_error("a bounded wait of an earlier kernel on device %d gave up: results since then are invalid; "
                  "mta_device_status() reports and clears the condition", dev);
        return MTA_ERR_TIMEOUT;
    }
    return MTA_OK;
}

int sm_count(int* out) {
    static std::atomic<int> known[MAX_DEVICES_KNOWN];
    int dev = 0;
    MTA_CUDA_OK(cudaGetDevice(&dev));
    int n = dev < MAX_DEVICES_KNOWN ? known[dev].load(std::memory_order_relaxed) : 0;
    if (n == 0) {
        MTA_CUDA_OK(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
        if (dev < MAX_DEVICES_KNOWN) known[dev].store(n, std::memory_order_relaxed);
    }
    *out = n;
    return MTA_OK;
}

PlaneView full_view(int rows, int cols) { return PlaneView{(long)rows * cols, 0, cols}; }

namespace {
// `op(copy of x, copy of y)` on padded copies in the workspace; y's is copied back.
template <typename OP>
int on_padded(const void* x, void* y, PlaneView v, const PadPlan& p, void* workspace, long planes, int H, int W, int causal, float fill, int dtype,
              cudaStream_t st, OP op) {
    char* xp = static_cast<char*>(workspace);
    char* yp = xp + p.bytes;
    if (int rc = pad_planes(x, v, xp, p, planes, H, W, causal, dtype, st)) return rc;
    if (int rc = op(xp, yp)) return rc;
    return unpad_planes(yp, p, y, v, planes, H, W, causal, fill, dtype, st);
}

int head_mix_maybe_padded(const void* x, const void* Wm, int w_dtype, void* y, void* workspace, size_t workspace_bytes, int N, int C, int P, int Q,
                          int causal, float fill, bool w_transposed, int dtype, cudaStream_t st) {
    const PlaneView v = full_view(P, Q);
    const PadPlan p = pad_plan((long)N * C, P, Q, dtype);
    // B1 H12 S601 (4M scores) 21 us without copies, 26 with; B1 H16 S1022 48 / 42; B3 H12 S1739 251 / 189; 64 heads, B2 S1001: 914 / 226
    const bool pays = C > 32 || (long)N * C * P * Q >= 8L << 20;
    if (p.use && pays && workspace && workspace_bytes >= 2 * p.bytes && variant("head_linear") == 0 && aligned16(workspace) &&
        (C <= 32 || head_linear_tc05_supported(workspace, p.view, static_cast<char*>(workspace) + p.bytes, p.view, C, Q, dtype, w_dtype)))
        return on_padded(x, y, v, p, workspace, (long)N * C, P, Q, causal, fill, dtype, st, [&](const void* xp, void* yp) {
            return head_linear_launch(xp, p.view, Wm, w_dtype, yp, p.view, N, C, P, Q, causal, fill, 0, P, false, dtype, st, w_transposed);
        });
    return head_linear_launch(x, v, Wm, w_dtype, y, v, N, C, P, Q, causal, fill, 0, P, true, dtype, st, w_transposed);
}
}  // namespace

}  // namespace mta

using namespace mta;

extern "C" {

int mta_abi_version(void) { return 2; }

const char* mta_last_error(void) { return g_error; }

long mta_launch_count(void) { return g_launches; }
void mta_reset_launch_count(void) { g_launches = 0; }

int mta_set_variant(const char* key, int value) {
    if (!key || value < 0 || value > 3) return MTA_ERR_INVALID;
    if (!strcmp(key, "head_linear")) g_variant_head_linear.store(value, std::memory_order_relaxed);
    else if (!strcmp(key, "conv2d")) g_variant_conv2d.store(value, std::memory_order_relaxed);
    else if (!strcmp(key, "gemm")) g_variant_gemm.store(value, std::memory_order_relaxed);
    else if (!strcmp(key, "fused")) g_variant_fused.store(value, std::memory_order_relaxed);
    else if (!strcmp(key, "mix_softmax")) g_variant_mix_softmax.store(value, std::memory_order_relaxed);
    else return MTA_ERR_INVALID;
    return MTA_OK;
}

size_t mta_planes_workspace_bytes(int N, int C, int P, int Q, int dtype) {
    if (N <= 0 || C <= 0 || P <= 0 || Q <= 0 || !dtype_ok(dtype)) return 0;
    const PadPlan p = pad_plan((long)N * C, P, Q, dtype);
    return p.use ? 2 * p.bytes : 0;
}

int mta_conv2d_fwd(const void* x, const void* w, void* y, int N, int C, int H, int W, int R, int S, int causal,
                   int x_dtype, int w_dtype, void* stream) {
    return mta_conv2d_fwd_ws(x, w, y, nullptr, 0, N, C, H, W, R, S, causal, x_dtype, w_dtype, stream);
}

int mta_conv2d_fwd_ws(const void* x, const void* w, void* y, void* workspace, size_t workspace_bytes, int N, int C, int H, int W, int R,
                      int S, int causal, int x_dtype, int w_dtype, void* stream) {
    g_error[0] = 0;
    MTA_REQUIRE(dtype_ok(x_dtype) && dtype_ok(w_dtype), "conv2d: unknown dtype code (x %d, w %d)", x_dtype, w_dtype);
    MTA_REQUIRE(N >= 0 && C >= 1 && H >= 0 && W >= 0, "conv2d: bad shape N=%d C=%d H=%d W=%d", N, C, H, W);
    MTA_REQUIRE(R >= 1 && S >= 1, "conv2d: kernel size %dx%d must be positive", R, S);
    if ((long)N * H * W == 0) return MTA_OK;
    MTA_REQUIRE(x && w && y, "conv2d: null pointer");
    MTA_REQUIRE(x != y, "conv2d: in-place operation is not supported");
    if (int rc = check_device()) return rc;
    const PlaneView v = full_view(H, W);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const PadPlan p = pad_plan((long)N * C, H, W, x_dtype);
    if (p.use && workspace && workspace_bytes >= 2 * p.bytes && variant("conv2d") == 0 &&
        conv2d_tc05_supported(workspace, p.view, workspace, p.view, W, R, S, x_dtype, w_dtype))
        return on_padded(x, y, v, p, workspace, (long)N * C, H, W, causal ? 1 : 0, 0.0f, x_dtype, st, [&](const void* xp, void* yp) {
            return conv2d_launch(xp, p.view, H, w, w_dtype, yp, p.view, (long)N * C, C, H, W, R, S, causal ? 1 : 0, 0, H, false, x_dtype, st);
        });
    return conv2d_launch(x, v, H, w, w_dtype, y, v, (long)N * C, C, H, W, R, S, causal ? 1 : 0, 0, H, true, x_dtype, st);
}

int mta_head_linear_fwd(const void* x, const void* Wm, void* y, int N, int C, int P, int Q, int causal, float fill,
                        int x_dtype, int w_dtype, void* stream) {
    return mta_head_linear_fwd_ws(x, Wm, y, nullptr, 0, N, C, P, Q, causal, fill, x_dtype, w_dtype, stream);
}

int mta_head_linear_fwd_ws(const void* x, const void* Wm, void* y, void* workspace, size_t workspace_bytes, int N, int C, int P, int Q,
                           int causal, float fill, int x_dtype, int w_dtype, void* stream) {
    g_error[0] = 0;
    MTA_REQUIRE(dtype_ok(x_dtype) && dtype_ok(w_dtype), "head_linear: unknown dtype code (x %d, w %d)", x_dtype, w_dtype);
    MTA_REQUIRE(N >= 0 && C >= 1 && P >= 0 && Q >= 0, "head_linear: bad shape N=%d C=%d P=%d Q=%d", N, C, P, Q);
    if ((long)N * P * Q == 0) return MTA_OK;
    MTA_REQUIRE(x && Wm && y, "head_linear: null pointer");
    MTA_REQUIRE(x != y, "head_linear: in-place operation is not supported");
    if (int rc = check_device()) return rc;
    return head_mix_maybe_padded(x, Wm, w_dtype, y, workspace, workspace_bytes, N, C, P, Q, causal ? 1 : 0, fill, false, x_dtype,
                                 static_cast<cudaStream_t>(stream));
}

int mta_softmax_fwd(const void* x, void* y, int N, int C, int P, int Q, int causal, int dtype, void* stream) {
    g_error[0] = 0;
    MTA_REQUIRE(dtype_ok(dtype), "softmax: unknown dtype code %d", dtype);
    MTA_REQUIRE(N >= 0 && C >= 1 && P >= 0 && Q >= 0, "softmax: bad shape N=%d C=%d P=%d Q=%d", N, C, P, Q);
    if ((long)N * P * Q == 0) return MTA_OK;
    MTA_REQUIRE(x && y, "softmax: null pointer");
    if (int rc = check_device()) return rc;
    const PlaneView v = full_view(P, Q);
    return softmax_launch(x, v, y, v, (long)N * C, P, Q, causal ? 1 : 0, 0, P, true, 1.0f, dtype,
                          static_cast<cudaStream_t>(stream));
}

int mta_head_linear_softmax_fwd(const void* x, const void* Wm, void* y, int N, int C, int P, int Q, int x_dtype, int w_dtype,
                                void* stream) {
    g_error[0] = 0;
    MTA_REQUIRE(dtype_ok(x_dtype) && dtype_ok(w_dtype), "head_linear_softmax: unknown dtype code (x %d, w %d)", x_dtype, w_dtype);
    MTA_REQUIRE(N >= 0 && C >= 1 && P >= 0 && Q >= 0, "head_linear_softmax: bad shape N=%d C=%d P=%d Q=%d", N, C, P, Q);
    if ((long)N * P * Q == 0) return MTA_OK;
    MTA_REQUIRE(x && Wm && y, "head_linear_softmax: null pointer");
    MTA_REQUIRE(x != y, "head_linear_softmax: in-place operation is not supported");
    if (int rc = check_device()) return rc;
    const PlaneView v = full_view(P, Q);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (variant("fused") != 1 && head_mix_softmax_supported(x, v, y, v, C, Q, 1, x_dtype, w_dtype))
        return head_mix_softmax_launch(x, v, Wm, w_dtype, y, v, N, C, Q, 0, P, true, x_dtype, st);
    // shapes the one-pass kernel does not take: the two stages, the softmax in place
    if (int rc = head_linear_launch(x, v, Wm, w_dtype, y, v, N, C, P, Q, 1, 0.0f, 0, P, false, x_dtype, st)) return rc;
    return softmax_launch(y, v, y, v, (long)N * C, P, Q, 1, 0, P, true, 1.0f, x_dtype, st);
}

int mta_conv2d_bwd_input(const void* dy, const void* w, void* dx, int N, int C, int H, int W, int R, int S, int causal,
                         int dtype, int w_dtype, void* stream) {
    return mta_conv2d_bwd_input_ws(dy, w, dx, nullptr, 0, N, C, H, W, R, S, causal, dtype, w_dtype, stream);
}

int mta_conv2d_bwd_input_ws(const void* dy, const void* w, void* dx, void* workspace, size_t workspace_bytes, int N, int C, int H, int W,
                            int R, int S, int causal, int dtype, int w_dtype, void* stream) {
    g_error[0] = 0;
    MTA_REQUIRE(dtype_ok(dtype) && dtype_ok(w_dtype), "conv2d_bwd_input: unknown dtype code (dy %d, w %d)", dtype, w_dtype);
    MTA_REQUIRE(N >= 0 && C >= 1 && H >= 0 && W >= 0, "conv2d_bwd_input: bad shape N=%d C=%d H=%d W=%d", N, C, H, W);
    MTA_REQUIRE(R >= 1 && S >= 1, "conv2d_bwd_input: kernel size %dx%d must be positive", R, S);
    if ((long)N * H * W == 0) return MTA_OK;
    MTA_REQUIRE(dy && w && dx, "conv2d_bwd_input: null pointer");
    MTA_REQUIRE(dy != dx, "conv2d_bwd_input: in-place operation is not supported");
    if (int rc = check_device()) return rc;
    const PlaneView v = full_view(H, W);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const PadPlan p = pad_plan((long)N * C, H, W, dtype);
    if (p.use && workspace && workspace_bytes >= 2 * p.bytes && variant("conv2d") == 0 && S % 2 == 1 &&
        conv2d_tc05_supported(workspace, p.view, workspace, p.view, W, R, S, dtype, w_dtype))
        return on_padded(dy, dx, v, p, workspace, (long)N * C, H, W, causal ? 1 : 0, 0.0f, dtype, st, [&](const void* xp, void* yp) {
            return conv2d_bwd_input_launch(xp, p.view, w, w_dtype, yp, p.view, (long)N * C, C, H, W, R, S, causal ? 1 : 0, false, dtype, st);
        });
    return conv2d_bwd_input_launch(dy, v, w, w_dtype, dx, v, (long)N * C, C, H, W, R, S, causal ? 1 : 0, true, dtype, st);
}

size_t mta_conv2d_bwd_weight_workspace_bytes(int N, int C, int H, int W, int R, int S) {
    if (N <= 0 || C <= 0 || H <= 0 || W <= 0 || R < 1 || S < 1) return 0;
    return conv2d_bwd_weight_workspace(N, C, H, W, R, S);
}

size_t mta_conv2d_bwd_weight_workspace_for(int N, int C, int H, int W, int R, int S, int dtype) {
    if (N <= 0 || C <= 0 || H <= 0 || W <= 0 || R < 1 || S < 1 || !dtype_ok(dtype)) return 0;
    return conv2d_bwd_weight_padded_workspace(N, C, H, W, R, S, dtype);
}

int mta_conv2d_bwd_weight(const void* x, const void* dy, float* dw, void* workspace, size_t workspace_bytes, int N, int C,
                          int H, int W, int R, int S, int causal, int dtype, void* stream) {
    return mta_conv2d_bwd_weight_as(x, dy, dw, MTA_F32, workspace, workspace_bytes, N, C, H, W, R, S, causal, dtype, stream);
}

int mta_conv2d_bwd_weight_as(const void* x, const void* dy, void* dw, int dw_dtype, void* workspace, size_t workspace_bytes, int N,
                             int C, int H, int W, int R, int S, int causal, int dtype, void* stream) {
    g_error[0] = 0;
    MTA_REQUIRE(dtype_ok(dtype) && dtype_ok(dw_dtype), "conv2d_bwd_weight: unknown dtype code (x %d, dw %d)", dtype, dw_dtype);
    MTA_REQUIRE(N >= 0 && C >= 1 && H >= 0 && W >= 0, "conv2d_bwd_weight: bad shape N=%d C=%d H=%d W=%d", N, C, H, W);
    MTA_REQUIRE(R >= 1 && S >= 1, "conv2d_bwd_weight: kernel size %dx%d must be positive", R, S);
    MTA_REQUIRE(dw, "conv2d_bwd_weight: null pointer");
    if (int rc = check_device()) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if ((long)N * H * W == 0) {
        MTA_CUDA_OK(cudaMemsetAsync(dw, 0, (size_t)C * R * S * dtype_size(dw_dtype), st));
        return MTA_OK;
    }
    MTA_REQUIRE(x && dy, "conv2d_bwd_weight: null pointer");
    const size_t need = conv2d_bwd_weight_workspace(N, C, H, W, R, S);
    MTA_REQUIRE(workspace && workspace_bytes >= need, "conv2d_bwd_weight: workspace of %zu bytes is smaller than the %zu needed",
                workspace_bytes, need);
    return conv2d_bwd_weight_padded(x, full_view(H, W), dy, full_view(H, W), dw, dw_dtype, workspace, workspace_bytes, N, C, H, W, R, S, causal ? 1 : 0, dtype, st);
}

int mta_head_linear_bwd_input(const void* dy, const void* Wm, void* dx, int N, int C, int P, int Q, int causal, int dtype,
                              int w_dtype, void* stream) {
    return mta_head_linear_bwd_input_ws(dy, Wm, dx, nullptr, 0, N, C, P, Q, causal, dtype, w_dtype, stream);
}

int mta_head_linear_bwd_input_ws(const void* dy, const void* Wm, void* dx, void* workspace, size_t workspace_bytes, int N, int C, int P,
                                 int Q, int causal, int dtype, int w_dtype, void* stream) {
    g_error[0] = 0;
    MTA_REQUIRE(dtype_ok(dtype) && dtype_ok(w_dtype), "head_linear_bwd_input: unknown dtype code (dy %d, w %d)", dtype, w_dtype);
    MTA_REQUIRE(N >= 0 && C >= 1 && P >= 0 && Q >= 0, "head_linear_bwd_input: bad shape N=%d C=%d P=%d Q=%d", N, C, P, Q);
    if ((long)N * P * Q == 0) return MTA_OK;
    MTA_REQUIRE(dy && Wm && dx, "head_linear_bwd_input: null pointer");
    MTA_REQUIRE(dy != dx, "head_linear_bwd_input: in-place operation is not supported");
    if (int rc = check_device()) return rc;
    return head_mix_maybe_padded(dy, Wm, w_dtype, dx, workspace, workspace_bytes, N, C, P, Q, causal ? 1 : 0, 0.0f, true, dtype,
                                 static_cast<cudaStream_t>(stream));
}

size_t mta_head_linear_bwd_weight_workspace_bytes(int C) {
    if (C < 1 || C > 128) return 0;
    return head_linear_bwd_weight_workspace(C);
}

size_t mta_head_linear_bwd_weight_workspace_for(int N, int C, int P, int Q, int dtype) {
    if (C < 1 || C > 128 || N < 0 || P < 0 || Q < 0 || !dtype_ok(dtype)) return 0;
    return head_linear_bwd_weight_padded_workspace(N, C, P, Q, dtype);
}

int mta_head_linear_bwd_weight(const void* x, const void* dy, float* dW, void* workspace, size_t workspace_bytes, int N,
                               int C, int P, int Q, int causal, int dtype, void* stream) {
    return mta_head_linear_bwd_weight_as(x, dy, dW, MTA_F32, workspace, workspace_bytes, N, C, P, Q, causal, dtype, stream);
}

int mta_head_linear_bwd_weight_as(const void* x, const void* dy, void* dW, int dw_dtype, void* workspace, size_t workspace_bytes,
                                  int N, int C, int P, int Q, int causal, int dtype, void* stream) {
    g_error[0] = 0;
    MTA_REQUIRE(dtype_ok(dtype) && dtype_ok(dw_dtype), "head_linear_bwd_weight: unknown dtype code (x %d, dW %d)", dtype, dw_dtype);
    MTA_REQUIRE(N >= 0 && C >= 1 && C <= 128 && P >= 0 && Q >= 0, "head_linear_bwd_weight: bad shape N=%d C=%d P=%d Q=%d", N, C, P, Q);
    MTA_REQUIRE(dW, "head_linear_bwd_weight: null pointer");
    if (int rc = check_device()) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if ((long)N * P * Q == 0) {
        MTA_CUDA_OK(cudaMemsetAsync(dW, 0, (size_t)C * C * dtype_size(dw_dtype), st));
        return MTA_OK;
    }
    MTA_REQUIRE(x && dy, "head_linear_bwd_weight: null pointer");
    const size_t need = head_linear_bwd_weight_workspace(C);
    MTA_REQUIRE(workspace && workspace_bytes >= need, "head_linear_bwd_weight: workspace of %zu bytes is smaller than the %zu needed",
                workspace_bytes, need);
    return head_linear_bwd_weight_padded(x, full_view(P, Q), dy, full_view(P, Q), dW, dw_dtype, workspace, workspace_bytes, N, C, P, Q, causal ? 1 : 0, dtype, st);
}

int mta_qk_scores_fwd(const void* q, const void* k, void* s, int B, int H, int S, int D, float scale, int round_scale,
                      int causal, int dtype, void* stream) {
    g_error[0] = 0;
    MTA_REQUIRE(dtype_ok(dtype), "qk_scores: unknown dtype code %d", dtype);
    MTA_REQUIRE(B >= 0 && H >= 1 && S >= 0 && D >= 1, "qk_scores: bad shape B=%d H=%d S=%d D=%d", B, H, S, D);
    if ((long)B * S == 0) return MTA_OK;
    MTA_REQUIRE(q && k && s, "qk_scores: null pointer");
    MTA_REQUIRE((long)B * H <= 65535, "qk_scores: B*H = %ld exceeds 65535", (long)B * H);
    if (int rc = check_device()) return rc;
    return qk_scores_launch(q, k, s, full_view(S, S), B, H, S, D, scale, round_scale, causal ? 1 : 0, 0, S, dtype,
                            static_cast<cudaStream_t>(stream));
}

int mta_pv_fwd(const void* p, const void* v, void* o, int B, int H, int S, int D, int causal, int dtype, void* stream) {
    g_error[0] = 0;
    MTA_REQUIRE(dtype_ok(dtype), "pv: unknown dtype code %d", dtype);
    MTA_REQUIRE(B >= 0 && H >= 1 && S >= 0 && D >= 1, "pv: bad shape B=%d H=%d S=%d D=%d", B, H, S, D);
    if ((long)B * S == 0) return MTA_OK;
    MTA_REQUIRE(p && v && o, "pv: null pointer");
    MTA_REQUIRE((long)B * H <= 65535, "pv: B*H = %ld exceeds 65535", (long)B * H);
    if (int rc = check_device()) return rc;
    return pv_launch(p, full_view(S, S), S, v, o, B, H, S, D, causal ? 1 : 0, 0, S, dtype, static_cast<cudaStream_t>(stream));
}

int mta_device_status(void* stream) {
    g_error[0] = 0;
    int timed_out = 0;
    if (int rc = device_wait_status(static_cast<cudaStream_t>(stream), &timed_out)) return rc;
    if (timed_out) {
        set_error("a device-side bounded wait (mbarrier) gave up: results of the kernels launched since the last check are invalid");
        return MTA_ERR_TIMEOUT;
    }
    return MTA_OK;
}

int mta_inject_wait_timeout(void* stream) {
    g_error[0] = 0;
    return wait_flag_inject(static_cast<cudaStream_t>(stream));
}

int mta_inject_late_wait_timeout(void* stream) {
    g_error[0] = 0;
    if (int rc = check_device()) return rc;
    return wait_flag_inject_late(static_cast<cudaStream_t>(stream));
}

}  // extern "C"
