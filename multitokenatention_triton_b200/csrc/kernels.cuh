// Internal launch interface between the C ABI (abi.cu), the fused forward (fused.cu) and the kernel
// translation units.  Every function enqueues work on `st` and returns an MTA_* status.
#pragma once

#include "common.cuh"
#include "dropout.cuh"

namespace mta {

// Keys that no query may see, one bit each (bit k % 32 of word k / 32), `words` words per batch element; null: every key may
// be seen.
struct DeadKeys {
    const uint32_t* bits = nullptr;
    int words = 0;
    // The bits of keys [key, key + 32) of batch element n, key a multiple of 32.
    __device__ uint32_t word(long n, int key) const { return bits ? __ldg(bits + n * words + (key >> 5)) : 0u; }
};
// Copies of unaligned 16-bit planes in padded rows (pad.cu): `use` says whether they pay, `bytes` is the size of one.
struct PadPlan {
    bool use;
    PlaneView view;
    size_t bytes;
};
PadPlan pad_plan(long planes, int H, int W, int dtype);
// The lower triangle only when causal; unpad_planes writes the whole of `out`, `fill` above the diagonal.
int pad_planes(const void* in, PlaneView iv, void* copy, const PadPlan& p, long planes, int H, int W, int causal, int dtype, cudaStream_t st);
int unpad_planes(const void* copy, const PadPlan& p, void* out, PlaneView ov, long planes, int H, int W, int causal, float fill, int dtype,
                 cudaStream_t st);
// out (B,H,S,D) contiguous = in (B,S,H,D) contiguous (mask.cu).
int swap_heads_launch(const void* in, void* out, int B, int H, int S, int D, int dtype, cudaStream_t st);
// Prepares them from a (B,S) byte mask (0 = dead), together with copies of k and v (B,H,S,D) whose rows of dead keys are zero
// (mask.cu).  Zero rows of K make the scores of dead keys zero; zero rows of V drop whatever the later stages hold there.
int mask_prepare_launch(const unsigned char* key_mask, const void* k, const void* v, uint32_t* bits, void* k_out, void* v_out, int B, int H,
                        int S, int D, int dtype, cudaStream_t st);

// `early_weights` below: this is not the first kernel of the library call (see pdl_wait() in common.cuh).
//
// Depthwise causal conv over planes; computes output rows [row_begin,row_end) of every plane.
// When `write_upper` the entries above the diagonal of those rows are written as 0, otherwise they
// are left untouched (internal scratch whose upper triangle nobody reads).
// `x_rows_stored` = rows each plane of x holds (from xv.row0 on).
int conv2d_launch(const void* x, PlaneView xv, long x_rows_stored, const void* w, int w_dtype, void* y, PlaneView yv,
                  long planes, int C, int H, int W, int R, int S, int causal, int row_begin, int row_end,
                  bool write_upper, int dtype, cudaStream_t st, bool early_weights = false);
// CUDA cores, odd key extents 3 .. 15 (conv2d_fma.cu): the conv or its input gradient, and the weight gradient's per-part sums.
bool conv2d_fma_supported(int R, int S, long planes);
int conv2d_fma_launch(const void* x, PlaneView xv, const void* w, int w_dtype, void* y, PlaneView yv, long planes, int C, int H, int W, int R,
                      int S, int causal, int row_begin, int row_end, bool write_upper, bool grad_input, int dtype, cudaStream_t st);
int conv2d_dw_fma_launch(const void* x, PlaneView xv, const void* dy, PlaneView dyv, float* partial, int max_parts, int* parts_out, long planes,
                         int H, int W, int R, int S, int causal, int dtype, cudaStream_t st);
// Tensor-core version (conv2d_mma.cu): 16-bit dtypes, S <= 17, W a multiple of 8, 16-byte aligned planes.
bool conv2d_mma_supported(const void* x, PlaneView xv, const void* y, PlaneView yv, int W, int R, int S, int dtype);
int conv2d_mma_launch(const void* x, PlaneView xv, long x_rows_stored, const void* w, int w_dtype, void* y, PlaneView yv,
                      long planes, int C, int H, int W, int R, int S, int causal, int row_begin, int row_end,
                      bool write_upper, int dtype, cudaStream_t st);

// Head mix over groups of C planes; rows [row_begin,row_end).  `write_upper` as above (value `fill`).
// `w_transposed`: y[o] = sum_h Wm[h,o] x[h] (the gradient with respect to the head mix's input).
int head_linear_launch(const void* x, PlaneView xv, const void* Wm, int w_dtype, void* y, PlaneView yv, int N,
                       int C, int P, int Q, int causal, float fill, int row_begin, int row_end, bool write_upper,
                       int dtype, cudaStream_t st, bool w_transposed = false, bool early_weights = false);

// Gradients of the two stand-alone ops (backward.cu, conv2d.cu).  dx of the conv: zeros above the diagonal when causal and
// `write_upper`.  The weight gradients come in `dw_dtype`, reduced in a fixed order through a caller workspace.
int conv2d_bwd_input_launch(const void* dy, PlaneView dyv, const void* w, int w_dtype, void* dx, PlaneView dxv, long planes, int C, int H,
                            int W, int R, int S, int causal, bool write_upper, int dtype, cudaStream_t st, bool early_weights = false);
size_t conv2d_bwd_weight_workspace(int N, int C, int H, int W, int R, int S);
int conv2d_bwd_weight_launch(const void* x, PlaneView xv, const void* dy, PlaneView dyv, void* dw, int dw_dtype, void* workspace, int N, int C,
                             int H, int W, int R, int S, int causal, int dtype, cudaStream_t st);
// The same with a workspace that may also hold padded copies of x and dy (the size is what makes them possible).
size_t conv2d_bwd_weight_padded_workspace(int N, int C, int H, int W, int R, int S, int dtype);
int conv2d_bwd_weight_padded(const void* x, PlaneView xv, const void* dy, PlaneView dyv, void* dw, int dw_dtype, void* workspace,
                             size_t workspace_bytes, int N, int C, int H, int W, int R, int S, int causal, int dtype, cudaStream_t st);
size_t head_linear_bwd_weight_padded_workspace(int N, int C, int P, int Q, int dtype);
int head_linear_bwd_weight_padded(const void* x, PlaneView xv, const void* dy, PlaneView dyv, void* dW, int dw_dtype, void* workspace,
                                  size_t workspace_bytes, int N, int C, int P, int Q, int causal, int dtype, cudaStream_t st);
// The conv's weight gradient on tcgen05 (conv2d_dw_tc05.cu).
bool conv2d_dw_tc05_supported(const void* x, PlaneView xv, const void* dy, PlaneView dyv, int R, int S, int dtype);
size_t conv2d_dw_tc05_workspace(int N, int C, int H, int W, int R, int S);
int conv2d_dw_tc05_launch(const void* x, PlaneView xv, const void* dy, PlaneView dyv, void* dw, int dw_dtype, void* workspace, int N, int C, int H,
                          int W, int R, int S, int causal, int dtype, cudaStream_t st);
size_t head_linear_bwd_weight_workspace(int C);
int head_linear_bwd_weight_launch(const void* x, PlaneView xv, const void* dy, PlaneView dyv, void* dW, int dw_dtype, void* workspace, int N, int C,
                                  int P, int Q, int causal, int dtype, cudaStream_t st);

// The head mix's weight gradient on tcgen05 (head_dw_tc05.cu).
bool head_dw_tc05_supported(const void* x, PlaneView xv, const void* dy, PlaneView dyv, int C, int dtype);
int head_dw_tc05_launch(const void* x, PlaneView xv, const void* dy, PlaneView dyv, float* partial, int* slots_out, int N, int C, int P, int Q,
                        int causal, int dtype, cudaStream_t st);

// Head mix followed by the causal row softmax of the mixed logits, in one pass (causal; 16-bit dtypes with C <= 32, float32 with rows that fit);
// entries above the diagonal of y are written as 0 when `write_upper`, else left untouched.
bool head_mix_softmax_supported(const void* x, PlaneView xv, const void* y, PlaneView yv, int C, int Q, int causal, int dtype,
                                int w_dtype);
int head_mix_softmax_launch(const void* x, PlaneView xv, const void* Wm, int w_dtype, void* y, PlaneView yv, int N, int C,
                            int Q, int row_begin, int row_end, bool write_upper, int dtype, cudaStream_t st, bool early_weights = false);

// The same in float32 (head_mix_softmax_f32.cu), rows whose C logits fit into shared memory, 16-byte aligned.
bool head_mix_softmax_f32_supported(const void* x, PlaneView xv, const void* y, PlaneView yv, int C, int Q, int causal, int dtype);
int head_mix_softmax_f32_launch(const void* x, PlaneView xv, const void* Wm, int w_dtype, void* y, PlaneView yv, int N, int C, int Q, int row_begin,
                                int row_end, bool write_upper, cudaStream_t st, bool early_weights);

// The same on tcgen05 (head_mix_tc05.cu): C a power of two in 8..128, weights in the activations' 16-bit dtype; entries
// above the diagonal are written as 0 up to the end of the diagonal's 128-key tile, and up to Q when `write_upper`.
bool head_mix_softmax_tc05_supported(const void* x, PlaneView xv, const void* y, PlaneView yv, int C, int Q, int causal, int dtype,
                                     int w_dtype);
int head_mix_softmax_tc05_launch(const void* x, PlaneView xv, const void* Wm, void* y, PlaneView yv, int N, int C, int Q,
                                 int row_begin, int row_end, bool write_upper, int dtype, cudaStream_t st, DeadKeys dead = DeadKeys(),
                                 bool early_weights = false);

// The plain head mix on the same kernel (one pass): y = Wm x over the head axis (Wm read transposed when `wt`), `fill`
// above the diagonal when causal (written up to the end of the diagonal's key tile, and up to Q when `write_upper`).
bool head_linear_tc05_supported(const void* x, PlaneView xv, const void* y, PlaneView yv, int C, int Q, int dtype, int w_dtype);
int head_linear_tc05_launch(const void* x, PlaneView xv, const void* Wm, void* y, PlaneView yv, int N, int C, int Q, int causal,
                            float fill, int row_begin, int row_end, bool write_upper, bool wt, int dtype, cudaStream_t st, bool early_weights = false);

// A small causal conv (2 or 3 row taps, 3 key taps) and the head mix that follows it in one kernel (conv_mix_tc05.cu): the conv's
// output never reaches memory.  16-bit dtypes, weights in the same one, C = 8, 16, 32 or 64, rows [row_begin,row_end).
bool conv_mix_supported(const void* x, PlaneView xv, const void* y, PlaneView yv, int C, int CQ, int CK, int causal, int dtype, int w_dtype);
int conv_mix_launch(const void* x, PlaneView xv, const void* w, const void* Wm, void* y, PlaneView yv, int N, int C, int Q, int CQ, int CK, int row_begin,
                    int row_end, int dtype, cudaStream_t st);

// Causal row softmax of pre_scale * x; rows [row_begin,row_end).  `dead` (planes of one batch element: `heads`): keys that get
// probability 0, in a row with no other key too.
int softmax_launch(const void* x, PlaneView xv, void* y, PlaneView yv, long planes, int P, int Q, int causal,
                   int row_begin, int row_end, bool write_upper, float pre_scale, int dtype, cudaStream_t st, DeadKeys dead = DeadKeys(), int heads = 1);

// ds = p (g - sum over the row of g p), keys k <= query when causal; ds may be g.  Nothing above the diagonal is touched.
int softmax_bwd_launch(const void* p, PlaneView pv, const void* g, PlaneView gv, void* ds, PlaneView dv, long planes, int P, int Q,
                       int causal, int dtype, cudaStream_t st);

// s = round(round(Q K^T) * scale) for rows [row_begin,row_end), keys k <= q when causal.
int qk_scores_launch(const void* q, const void* k, void* s, PlaneView sv, int B, int H, int S, int D, float scale,
                     int round_scale, int causal, int row_begin, int row_end, int dtype, cudaStream_t st);

// o[rows] = p[rows, k<=q] V.  `p_rows_stored` = number of rows each plane of p holds (from pview.row0 on).
// `drop`: dropout on the weights as they are read (dropout.cuh); the default leaves them as they are.
int pv_launch(const void* p, PlaneView pview, long p_rows_stored, const void* v, void* o, int B, int H, int S, int D,
              int causal, int row_begin, int row_end, int dtype, cudaStream_t st, DropoutSpec drop = DropoutSpec(), float scale = 1.0f);
// o[key] = scale * sum over queries >= key (all when not causal) of p[query, key] x[query]: the product with the transposed plane.
int ptx_launch(const void* p, PlaneView pview, const void* x, void* o, int B, int H, int S, int D, int causal, float scale, int dtype,
               cudaStream_t st);

// CUDA-core versions of the two contractions (gemm_simt.cu).
int qk_scores_simt_launch(const void* q, const void* k, void* s, PlaneView sv, int B, int H, int S, int D, float scale,
                          int round_scale, int causal, int row_begin, int row_end, int dtype, cudaStream_t st);
int pv_simt_launch(const void* p, PlaneView pview, const void* v, void* o, int B, int H, int S, int D, int causal,
                   int row_begin, int row_end, int dtype, cudaStream_t st, DropoutSpec drop = DropoutSpec(), bool trans = false,
                   float scale = 1.0f);

// float32 with 16-byte aligned rows (gemm_f32.cu).
bool gemm_f32_supported(const void* a, const void* b, const void* c, PlaneView plane, int S, int D, int dtype);
int qk_f32_launch(const void* q, const void* k, void* s, PlaneView sv, int B, int H, int S, int D, float scale, int causal, int row_begin,
                  int row_end, cudaStream_t st);
int pv_f32_launch(const void* p, PlaneView pview, const void* v, void* o, int B, int H, int S, int D, int causal, int row_begin, int row_end,
                  bool trans, float scale, cudaStream_t st);

// tcgen05 version of the conv (conv2d_tc05.cu): 16-bit dtypes, S <= 17, any W on rows whose pitch is a multiple of 8 elements, R <= 16;
// weights of the same type or float32 (then in two 16-bit parts).
bool conv2d_tc05_supported(const void* x, PlaneView xv, const void* y, PlaneView yv, int W, int R, int S, int dtype,
                           int w_dtype);
// `grad_input` (odd S): the same kernel evaluates the gradient with respect to the conv's input - taps reversed, rows
// looking forward - with x = dy and y = dx.
int conv2d_tc05_launch(const void* x, PlaneView xv, long x_rows_stored, const void* w, int w_dtype, void* y, PlaneView yv,
                       long planes, int C, int H, int W, int R, int S, int causal, int row_begin, int row_end,
                       bool write_upper, int dtype, cudaStream_t st, bool grad_input = false, bool early_weights = false);

// tcgen05 tensor-core versions (gemm_tc05.cu): 16-bit dtypes, D in {64,128}, any S on planes whose row pitch is a multiple of 8 elements.
bool tc05_contractions_supported(int S, int D, int dtype, const void* a, const void* b, const void* c, PlaneView view);
int pv_tc05_launch(const void* p, PlaneView pview, long p_rows_stored, const void* v, void* o, int B, int H, int S, int D,
                   int causal, int row_begin, int row_end, int dtype, cudaStream_t st, DropoutSpec drop = DropoutSpec(),
                   bool trans = false, float scale = 1.0f);
// Persistent, warp-specialised score-tile kernel (qk_persistent.cu); same domain as the kernels above.
// NI = 1: c = scale * a b^T.  mode 0: all tiles with keys <= query; 1 / 2: the band of a (band_cq x (2 band_pw + 1))
// conv / the tiles wholly below it.
int qk_persistent_launch(const void* a, const void* b, void* c, PlaneView cv, int B, int H, int S, int D, int NI, float scale,
                         int round_scale, int causal, int mode, int band_cq, int band_pw, int row_begin, int row_end, int dtype,
                         cudaStream_t st);
// Scaled scores Q K^T and the causal conv of them in one kernel (qk_conv_tc05.cu): y = conv(round(round(Q K^T) scale)),
// rows [row_begin,row_end); the score planes never reach memory.  16-bit dtypes, D in {64,128}, odd key extent <= 17.
bool qk_conv_supported(const void* q, const void* k, const void* y, PlaneView yv, int S, int D, int R, int KS, int causal, int dtype,
                       int w_dtype);
int qk_conv_launch(const void* q, const void* k, const void* w, int w_dtype, void* y, PlaneView yv, int B, int H, int S, int D,
                   int R, int KS, float scale, int row_begin, int row_end, int dtype, cudaStream_t st);
// The conv attention forward softmax(sm_scale * conv(round(Q K^T))) V in one kernel with no score plane
// anywhere (conv_attn_tc05.cu); output rows [row_begin,row_end).  16-bit dtypes, D in {64,128}, odd key extent <= 17,
// causal, any S.
bool conv_attn_fused_shape_ok(int S, int D, int R, int KS, int causal, int dtype, int w_dtype);
bool conv_attn_fused_supported(const void* q, const void* k, const void* v, const void* o, int S, int D, int R, int KS, int causal,
                               int dtype, int w_dtype);
int conv_attn_fused_launch(const void* q, const void* k, const void* v, const void* w, int w_dtype, void* o, int B, int H, int S, int D,
                           int R, int KS, float sm_scale, int row_begin, int row_end, int dtype, cudaStream_t st);
// Scratch that mta_conv_attn_fwd needs at the least (0: none); with mta_conv_attn_workspace_bytes(...) its rows are padded.
size_t conv_attn_least_workspace(int B, int H, int S, int D, int cq, int ck, int causal, int dtype, int w_dtype);
// Reads and clears the flag raised by a device-side bounded wait that gave up (synchronises `st`).
int device_wait_status(cudaStream_t st, int* timed_out);
// True when such a wait has given up on the current device since the last device_wait_status; reads the flag's mirror in
// host memory, no synchronisation.
bool wait_flag_raised();
// Raises the flag from the host as a timed-out wait would.
int wait_flag_inject(cudaStream_t st);
// Launches a kernel whose bounded wait gives up after a few milliseconds.
int wait_flag_inject_late(cudaStream_t st);

}  // namespace mta
