// Chooses the implementation of the products with a score plane: tcgen05 tensor cores for 16-bit dtypes with D in {64,128}
// and 16-byte aligned rows, gemm_f32.cu for float32 with 16-byte aligned rows, the general CUDA-core kernels otherwise.
// mta_set_variant("gemm", 1) forces the general CUDA-core kernels, ("gemm", 2) requires the tensor-core ones.
#include "kernels.cuh"

namespace mta {

int qk_scores_launch(const void* q, const void* k, void* s, PlaneView sv, int B, int H, int S, int D, float scale,
                     int round_scale, int causal, int row_begin, int row_end, int dtype, cudaStream_t st) {
    if (B == 0 || row_end <= row_begin) return MTA_OK;
    const int want = variant("gemm");
    const bool ok = tc05_contractions_supported(S, D, dtype, q, k, s, sv);
    MTA_REQUIRE(want != 2 || ok, "qk_scores: the tensor-core variant needs a 16-bit dtype, D in {64,128}, S %% 8 == 0 and 16-byte aligned tensors");
    if (ok && want != 1)
        return qk_persistent_launch(q, k, s, sv, B, H, S, D, 1, scale, round_scale, causal, 0, 1, 0, row_begin, row_end, dtype, st);
    if (want != 1 && gemm_f32_supported(q, k, s, sv, S, D, dtype))
        return qk_f32_launch(q, k, s, sv, B, H, S, D, scale, causal, row_begin, row_end, st);
    return qk_scores_simt_launch(q, k, s, sv, B, H, S, D, scale, round_scale, causal, row_begin, row_end, dtype, st);
}

int pv_launch(const void* p, PlaneView pview, long p_rows_stored, const void* v, void* o, int B, int H, int S, int D,
              int causal, int row_begin, int row_end, int dtype, cudaStream_t st, DropoutSpec drop, float scale) {
    if (B == 0 || row_end <= row_begin) return MTA_OK;
    const int want = variant("gemm");
    const bool ok = tc05_contractions_supported(S, D, dtype, p, v, o, pview);
    MTA_REQUIRE(want != 2 || ok, "pv: the tensor-core variant needs a 16-bit dtype, D in {64,128}, S %% 8 == 0 and 16-byte aligned tensors");
    if (ok && want != 1)
        return pv_tc05_launch(p, pview, p_rows_stored, v, o, B, H, S, D, causal, row_begin, row_end, dtype, st, drop, false, scale);
    if (want != 1 && !drop.on() && gemm_f32_supported(p, v, o, pview, S, D, dtype))
        return pv_f32_launch(p, pview, v, o, B, H, S, D, causal, row_begin, row_end, false, scale, st);
    return pv_simt_launch(p, pview, v, o, B, H, S, D, causal, row_begin, row_end, dtype, st, drop, false, scale);
}

int ptx_launch(const void* p, PlaneView pview, const void* x, void* o, int B, int H, int S, int D, int causal, float scale, int dtype,
               cudaStream_t st) {
    if (B == 0 || S == 0) return MTA_OK;
    if (variant("gemm") != 1 && tc05_contractions_supported(S, D, dtype, p, x, o, pview))
        return pv_tc05_launch(p, pview, S, x, o, B, H, S, D, causal, 0, S, dtype, st, DropoutSpec(), true, scale);
    if (variant("gemm") != 1 && gemm_f32_supported(p, x, o, pview, S, D, dtype))
        return pv_f32_launch(p, pview, x, o, B, H, S, D, causal, 0, S, true, scale, st);
    return pv_simt_launch(p, pview, x, o, B, H, S, D, causal, 0, S, dtype, st, DropoutSpec(), true, scale);
}

}  // namespace mta
