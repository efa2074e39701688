// Preparation of the forward with a key mask (the (batch, keys) padding mask of MTAAttentionTriton._update_mask,
// mta_attention_triton.py:106-127): the mask as bits, and copies of K and V with the rows of dead keys zeroed.
//
// The reference zeroes the scores of dead keys before the first conv, adds -inf to their logits, zeroes their probabilities
// before the second conv and their weights after it (mta_attention_triton.py:72-86).  Zero rows of K give zero scores; the
// softmax reads the bits; zero rows of V make whatever the second conv and head mix leave at dead keys drop out.  So the
// causal kernels run as they are, on the lower triangle only, and the mask costs one pass over K and V.  Bound: memory.
#include "kernels.cuh"

namespace mta {
namespace {

constexpr int MP_THREADS = 256;

// A thread copies one 16-byte piece (or one element, PIECE = the element type) of a row of K or V.
template <typename PIECE>
__global__ void __launch_bounds__(MP_THREADS)
mask_prepare_kernel(const unsigned char* __restrict__ key_mask, const PIECE* __restrict__ k, const PIECE* __restrict__ v, uint32_t* __restrict__ bits,
                    PIECE* __restrict__ k_out, PIECE* __restrict__ v_out, int H, int S, int row_pieces, int words) {
    pdl_wait();
    const int i = (int)(blockIdx.x * MP_THREADS + threadIdx.x), plane = (int)blockIdx.y, b = plane / H;
    const unsigned char* mask = key_mask + (long)b * S;
    if (plane % H == 0 && i < words) {                   // the first plane of a batch element also writes its bits
        uint32_t d = 0;
        for (int e = 0; e < 32; ++e)
            if (i * 32 + e < S && mask[i * 32 + e] == 0) d |= 1u << e;
        bits[b * words + i] = d;
    }
    if (i >= S * row_pieces) return;
    const bool keep = mask[i / row_pieces] != 0;
    const long at = (long)plane * S * row_pieces + i;
    PIECE zero;
    memset(&zero, 0, sizeof(zero));
    k_out[at] = keep ? k[at] : zero;
    v_out[at] = keep ? v[at] : zero;
}

template <typename PIECE>
int launch(const unsigned char* key_mask, const void* k, const void* v, uint32_t* bits, void* k_out, void* v_out, int B, int H, int S, int row_pieces,
           cudaStream_t st) {
    const dim3 grid((unsigned)((S * row_pieces + MP_THREADS - 1) / MP_THREADS), (unsigned)(B * H));
    return launch_kernel<mask_prepare_kernel<PIECE>>("mask_prepare_kernel", grid, MP_THREADS, 0, st, key_mask, static_cast<const PIECE*>(k),
                                                     static_cast<const PIECE*>(v), bits, static_cast<PIECE*>(k_out), static_cast<PIECE*>(v_out), H, S,
                                                     row_pieces, (S + 31) / 32);
}

// One 16-byte piece (or element) per thread; consecutive threads along a row of D.
template <typename PIECE>
__global__ void __launch_bounds__(MP_THREADS)
swap_heads_kernel(const PIECE* __restrict__ in, PIECE* __restrict__ out, int H, int S, int row_pieces) {
    pdl_wait();
    const int i = (int)(blockIdx.x * MP_THREADS + threadIdx.x);
    if (i >= S * row_pieces) return;
    const int s = i / row_pieces, e = i - s * row_pieces, b = (int)blockIdx.y / H, h = (int)blockIdx.y % H;
    out[(long)blockIdx.y * S * row_pieces + i] = in[(((long)b * S + s) * H + h) * row_pieces + e];
}

template <typename PIECE> int launch_swap(const void* in, void* out, int B, int H, int S, int row_pieces, cudaStream_t st) {
    const dim3 grid((unsigned)((S * row_pieces + MP_THREADS - 1) / MP_THREADS), (unsigned)(B * H));
    return launch_kernel<swap_heads_kernel<PIECE>>("swap_heads_kernel", grid, MP_THREADS, 0, st, static_cast<const PIECE*>(in), static_cast<PIECE*>(out), H, S,
                                                   row_pieces);
}

}  // namespace

int swap_heads_launch(const void* in, void* out, int B, int H, int S, int D, int dtype, cudaStream_t st) {
    const size_t row = (size_t)D * dtype_size(dtype);
    if (row % 16 == 0 && aligned16(in) && aligned16(out)) return launch_swap<uint4>(in, out, B, H, S, (int)(row / 16), st);
    if (dtype == MTA_F32) return launch_swap<uint32_t>(in, out, B, H, S, D, st);
    return launch_swap<uint16_t>(in, out, B, H, S, D, st);
}

int mask_prepare_launch(const unsigned char* key_mask, const void* k, const void* v, uint32_t* bits, void* k_out, void* v_out, int B, int H,
                        int S, int D, int dtype, cudaStream_t st) {
    const size_t row = (size_t)D * dtype_size(dtype);
    if (row % 16 == 0 && aligned16(k) && aligned16(v) && aligned16(k_out) && aligned16(v_out))
        return launch<uint4>(key_mask, k, v, bits, k_out, v_out, B, H, S, (int)(row / 16), st);
    if (dtype == MTA_F32) return launch<uint32_t>(key_mask, k, v, bits, k_out, v_out, B, H, S, D, st);
    return launch<uint16_t>(key_mask, k, v, bits, k_out, v_out, B, H, S, D, st);
}

}  // namespace mta
