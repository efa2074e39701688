// The MTA forward of a training step and its backward as two calls (use_mask=False, causal, no dropout):
//
//   mta_train_fwd   scores -> conv -> head mix -> softmax -> conv -> head mix -> P V, keeping the five planes that the
//                   backward reads: scores, conv 1, probabilities, conv 2, head mix 2
//   mta_train_bwd   the gradients of q, k, v and the four weights from the gradient of the output
//
// Stand in for MTAAttentionTriton.forward under autograd (mta_attention_triton.py:61-92 with the backward kernels of
// convolution_2d_trit.py:143-295 and triton_linear_head.py:142-278, and torch's own backward of the softmax and of the two
// matrix products).  Every plane has padded rows (any sequence length runs on the tensor cores) and is read and written in
// the lower triangle only: the stage-by-stage autograd path writes zeros above the diagonal after each stage, masks the
// planes again before each product, converts them to float32 for the softmax's gradient and multiplies whole squares.
// The gradients of the products are the forward's own kernels: dP = dO V^T is a score product, dQ = dS K a P V product, and
// dV = P^T dO, dK = dS^T Q read the plane transposed.
#include "kernels.cuh"

namespace mta {
namespace {

constexpr int SAVED = 5;      // scores, conv 1, probabilities, conv 2, head mix 2
enum { SCORES, CONV1, PROBS, CONV2, MIX2 };

struct TrainPlan {
    PlaneView v;
    size_t plane_bytes;       // all B * H planes of one kind
    long planes;
};

TrainPlan train_plan(int B, int H, int S, int dtype) {
    TrainPlan t;
    const int step = dtype == MTA_F32 ? 32 : 64;          // rows on 128-byte boundaries
    t.v.width = (S + step - 1) / step * step;
    t.v.row0 = 0;
    t.v.plane_stride = (long)S * t.v.width;
    t.planes = (long)B * H;
    t.plane_bytes = ((size_t)t.planes * t.v.plane_stride * dtype_size(dtype) + 255) & ~size_t(255);
    return t;
}

size_t partial_bytes(int B, int H, int S, int cq, int ck, int cq2, int ck2) {
    size_t n = conv2d_bwd_weight_workspace(B, H, S, S, cq, ck);
    const size_t n2 = conv2d_bwd_weight_workspace(B, H, S, S, cq2, ck2), n3 = head_linear_bwd_weight_workspace(H);
    if (n2 > n) n = n2;
    if (n3 > n) n = n3;
    return (n + 255) & ~size_t(255);
}

int check_shape(const char* what, int B, int H, int S, int D, int cq, int ck, int cq2, int ck2, int dtype, int w_dtype) {
    MTA_REQUIRE(dtype_ok(dtype) && dtype_ok(w_dtype), "%s: unknown dtype code (%d, %d)", what, dtype, w_dtype);
    MTA_REQUIRE(B >= 0 && H >= 1 && H <= 128 && S >= 0 && D >= 1, "%s: bad shape B=%d H=%d S=%d D=%d", what, B, H, S, D);
    MTA_REQUIRE(cq >= 1 && ck >= 1 && cq2 >= 1 && ck2 >= 1 && ck % 2 == 1 && ck2 % 2 == 1,
                "%s: kernel sizes %dx%d and %dx%d must be positive with odd key extents", what, cq, ck, cq2, ck2);
    MTA_REQUIRE((long)B * H <= 65535, "%s: B*H = %ld exceeds 65535", what, (long)B * H);
    return MTA_OK;
}

}  // namespace
}  // namespace mta

using namespace mta;

extern "C" {

size_t mta_train_saved_bytes(int B, int H, int S, int dtype) {
    if (B <= 0 || H <= 0 || S <= 0 || !dtype_ok(dtype)) return 0;
    return SAVED * train_plan(B, H, S, dtype).plane_bytes;
}

size_t mta_train_workspace_bytes(int B, int H, int S, int D, int cq, int ck, int cq2, int ck2, int dtype) {
    if (B <= 0 || H <= 0 || S <= 0 || D <= 0 || cq < 1 || ck < 1 || cq2 < 1 || ck2 < 1 || !dtype_ok(dtype)) return 0;
    return 2 * train_plan(B, H, S, dtype).plane_bytes + partial_bytes(B, H, S, cq, ck, cq2, ck2) + (size_t)B * H * S * D * dtype_size(dtype);
}

int mta_train_fwd(const void* q, const void* k, const void* v, const void* w1, const void* W1, const void* w2, const void* W2, void* o,
                  void* saved, size_t saved_bytes, int B, int H, int S, int D, int cq, int ck, int cq2, int ck2, int dtype, int w_dtype,
                  void* stream) {
    set_error("%s", "");
    if (int rc = check_shape("train_fwd", B, H, S, D, cq, ck, cq2, ck2, dtype, w_dtype)) return rc;
    if ((long)B * S == 0) return MTA_OK;
    MTA_REQUIRE(q && k && v && w1 && W1 && w2 && W2 && o && saved, "train_fwd: null pointer");
    MTA_REQUIRE(saved_bytes >= mta_train_saved_bytes(B, H, S, dtype), "train_fwd: %zu bytes for the saved planes, %zu are needed", saved_bytes,
                mta_train_saved_bytes(B, H, S, dtype));
    MTA_REQUIRE(aligned16(saved), "train_fwd: the saved planes must be 16-byte aligned");
    if (int rc = check_device()) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const TrainPlan t = train_plan(B, H, S, dtype);
    char* base = static_cast<char*>(saved);
    void* pl[SAVED];
    for (int i = 0; i < SAVED; ++i) pl[i] = base + i * t.plane_bytes;
    int rc;
    if ((rc = qk_scores_launch(q, k, pl[SCORES], t.v, B, H, S, D, 1.0f / sqrtf((float)D), dtype != MTA_F32, 1, 0, S, dtype, st))) return rc;
    if ((rc = conv2d_launch(pl[SCORES], t.v, S, w1, w_dtype, pl[CONV1], t.v, t.planes, H, S, S, cq, ck, 1, 0, S, false, dtype, st, true))) return rc;
    if (head_mix_softmax_supported(pl[CONV1], t.v, pl[PROBS], t.v, H, S, 1, dtype, w_dtype)) {
        if ((rc = head_mix_softmax_launch(pl[CONV1], t.v, W1, w_dtype, pl[PROBS], t.v, B, H, S, 0, S, false, dtype, st, true))) return rc;
    } else {
        if ((rc = head_linear_launch(pl[CONV1], t.v, W1, w_dtype, pl[PROBS], t.v, B, H, S, S, 1, 0.0f, 0, S, false, dtype, st, false, true))) return rc;
        if ((rc = softmax_launch(pl[PROBS], t.v, pl[PROBS], t.v, t.planes, S, S, 1, 0, S, false, 1.0f, dtype, st))) return rc;
    }
    if ((rc = conv2d_launch(pl[PROBS], t.v, S, w2, w_dtype, pl[CONV2], t.v, t.planes, H, S, S, cq2, ck2, 1, 0, S, false, dtype, st, true))) return rc;
    if ((rc = head_linear_launch(pl[CONV2], t.v, W2, w_dtype, pl[MIX2], t.v, B, H, S, S, 1, 0.0f, 0, S, false, dtype, st, false, true))) return rc;
    return pv_launch(pl[MIX2], t.v, S, v, o, B, H, S, D, 1, 0, S, dtype, st);
}

int mta_train_bwd(const void* q, const void* k, const void* v, const void* w1, const void* W1, const void* w2, const void* W2,
                  const void* dout, const void* saved, void* dq, void* dk, void* dv, void* dw1, void* dW1, void* dw2, void* dW2,
                  void* workspace, size_t workspace_bytes, int B, int H, int S, int D, int cq, int ck, int cq2, int ck2, int dout_heads_inner,
                  int dtype, int w_dtype, void* stream) {
    set_error("%s", "");
    if (int rc = check_shape("train_bwd", B, H, S, D, cq, ck, cq2, ck2, dtype, w_dtype)) return rc;
    MTA_REQUIRE((long)B * S > 0, "train_bwd: empty problem");
    MTA_REQUIRE(q && k && v && w1 && W1 && w2 && W2 && dout && saved && workspace, "train_bwd: null pointer");
    const size_t need = mta_train_workspace_bytes(B, H, S, D, cq, ck, cq2, ck2, dtype);
    MTA_REQUIRE(workspace_bytes >= need, "train_bwd: workspace of %zu bytes is smaller than the %zu needed", workspace_bytes, need);
    MTA_REQUIRE(aligned16(saved) && aligned16(workspace), "train_bwd: saved planes and workspace must be 16-byte aligned");
    if (int rc = check_device()) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const TrainPlan t = train_plan(B, H, S, dtype);
    const char* base = static_cast<const char*>(saved);
    const void* pl[SAVED];
    for (int i = 0; i < SAVED; ++i) pl[i] = base + i * t.plane_bytes;
    char* ws = static_cast<char*>(workspace);
    void* ga = ws;                                        // the running gradient plane alternates between the two
    void* gb = ws + t.plane_bytes;
    void* partial = ws + 2 * t.plane_bytes;
    const float scale = 1.0f / sqrtf((float)D);
    int rc;
    if (dout_heads_inner) {                               // (B,S,H,D), as autograd hands it over: the products want (B,H,S,D)
        void* swapped = ws + 2 * t.plane_bytes + partial_bytes(B, H, S, cq, ck, cq2, ck2);
        if ((rc = swap_heads_launch(dout, swapped, B, H, S, D, dtype, st))) return rc;
        dout = swapped;
    }
    if (dv && (rc = ptx_launch(pl[MIX2], t.v, dout, dv, B, H, S, D, 1, 1.0f, dtype, st))) return rc;
    // how far back the chain of plane gradients has to go
    const bool to_scores = dq || dk, to_conv1 = to_scores || dw1, to_mix1 = to_conv1 || dW1, to_conv2 = to_mix1 || dw2;
    if (!to_conv2 && !dW2) return MTA_OK;
    // d(head mix 2) = dO V^T
    if ((rc = qk_scores_launch(dout, v, ga, t.v, B, H, S, D, 1.0f, 0, 1, 0, S, dtype, st))) return rc;
    if (dW2 && (rc = head_linear_bwd_weight_launch(pl[CONV2], t.v, ga, t.v, dW2, w_dtype, partial, B, H, S, S, 1, dtype, st))) return rc;
    if (!to_conv2) return MTA_OK;
    if ((rc = head_linear_launch(ga, t.v, W2, w_dtype, gb, t.v, B, H, S, S, 1, 0.0f, 0, S, false, dtype, st, true, true))) return rc;      // d(conv 2)
    if (dw2 && (rc = conv2d_bwd_weight_launch(pl[PROBS], t.v, gb, t.v, dw2, w_dtype, partial, B, H, S, S, cq2, ck2, 1, dtype, st))) return rc;
    if (!to_mix1) return MTA_OK;
    if ((rc = conv2d_bwd_input_launch(gb, t.v, w2, w_dtype, ga, t.v, t.planes, H, S, S, cq2, ck2, 1, false, dtype, st, true))) return rc;  // d(probabilities)
    if ((rc = softmax_bwd_launch(pl[PROBS], t.v, ga, t.v, ga, t.v, t.planes, S, S, 1, dtype, st))) return rc;                       // d(head mix 1)
    if (dW1 && (rc = head_linear_bwd_weight_launch(pl[CONV1], t.v, ga, t.v, dW1, w_dtype, partial, B, H, S, S, 1, dtype, st))) return rc;
    if (!to_conv1) return MTA_OK;
    if ((rc = head_linear_launch(ga, t.v, W1, w_dtype, gb, t.v, B, H, S, S, 1, 0.0f, 0, S, false, dtype, st, true, true))) return rc;      // d(conv 1)
    if (dw1 && (rc = conv2d_bwd_weight_launch(pl[SCORES], t.v, gb, t.v, dw1, w_dtype, partial, B, H, S, S, cq, ck, 1, dtype, st))) return rc;
    if (!to_scores) return MTA_OK;
    if ((rc = conv2d_bwd_input_launch(gb, t.v, w1, w_dtype, ga, t.v, t.planes, H, S, S, cq, ck, 1, false, dtype, st, true))) return rc;    // d(scores)
    if (dq && (rc = pv_launch(ga, t.v, S, k, dq, B, H, S, D, 1, 0, S, dtype, st, DropoutSpec(), scale))) return rc;
    if (dk && (rc = ptx_launch(ga, t.v, q, dk, B, H, S, D, 1, scale, dtype, st))) return rc;
    return MTA_OK;
}

}  // extern "C"
