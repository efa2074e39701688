// The stand-alone conv and head mix, and their gradients, on 16-bit planes whose rows do not start on 16-byte boundaries.  TMA and the
// 16-byte loads of the tensor-core kernels need rows that do, so the planes are copied into rows padded to a multiple of 16 elements, the
// kernels run on the copies, and a result plane is copied back.  The copies sit in a workspace that the caller may leave out.
//
// Bound: memory.  A warp copies a row; a lane assembles 16 aligned bytes of the destination from the two aligned 16-byte pieces of the
// source that hold them (the second is its neighbour's first, from L1) and shifts them into place.
#include "kernels.cuh"

namespace mta {
namespace {

constexpr int CP_THREADS = 256;
// Measured on B200, bf16, 6 x 11 conv and head mix, us without / with copies.  conv: B1 H8 S401 (1.2M scores) 31 / 21, B2 H8 S1001 97 / 48,
// B3 H12 S1739 478 / 196, B4 H16 S2041 1093 / 413.  Smaller planes gain nothing from three launches instead of one.  The head mix, which
// the CUDA cores do well when there are few heads, has a line of its own where it is called.
constexpr long PAD_MIN = 1L << 20;
constexpr size_t PAD_MAX = size_t(8) << 30;              // bytes of one copy: larger problems keep the memory that they needed before

// 8 elements from element `sh` (0 .. 7) of the 16 in (a, b) on; `sh` is the same in all lanes of a warp.
__device__ __forceinline__ uint4 shifted(uint4 a, uint4 b, int sh) {
    uint32_t t[5];
    switch (sh >> 1) {
        case 0: t[0] = a.x; t[1] = a.y; t[2] = a.z; t[3] = a.w; t[4] = b.x; break;
        case 1: t[0] = a.y; t[1] = a.z; t[2] = a.w; t[3] = b.x; t[4] = b.y; break;
        case 2: t[0] = a.z; t[1] = a.w; t[2] = b.x; t[3] = b.y; t[4] = b.z; break;
        default: t[0] = a.w; t[1] = b.x; t[2] = b.y; t[3] = b.z; t[4] = b.w; break;
    }
    if (sh & 1) return make_uint4(__funnelshift_r(t[0], t[1], 16), __funnelshift_r(t[1], t[2], 16), __funnelshift_r(t[2], t[3], 16), __funnelshift_r(t[3], t[4], 16));
    return make_uint4(t[0], t[1], t[2], t[3]);
}

// Columns [0, n) of a row are copied, n = row + 1 at most when causal; with `write_upper` the rest of the row becomes `fill`.
// in_mis, out_mis: elements between the last 16-byte boundary and the base; in_total: elements that may be read from the base on.
template <typename T>
__global__ void __launch_bounds__(CP_THREADS)
copy_planes_kernel(const uint16_t* __restrict__ in, PlaneView iv, int in_mis, long in_total, uint16_t* __restrict__ out, PlaneView ov, int out_mis,
                   int out_padded, int H, int W, int causal, int write_upper, float fill) {
    pdl_wait();
    const int row = (int)blockIdx.x * (CP_THREADS / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= H) return;
    const T fill_t = from_f32<T>(fill);
    const uint32_t fill16 = *reinterpret_cast<const uint16_t*>(&fill_t);
    const int n = causal ? min(row + 1, W) : W, nd = write_upper ? W : n;
    const uint16_t* src = in + iv.at(blockIdx.y, row, 0);
    uint16_t* dst = out + ov.at(blockIdx.y, row, 0);
    const long s0 = in_mis + iv.at(blockIdx.y, row, 0);   // from the 16-byte boundary below `in`
    const int lead = (int)((out_mis + ov.at(blockIdx.y, row, 0)) & 7);
    const int sh = (int)((s0 - lead) & 7);
    const uint4* pieces = reinterpret_cast<const uint4*>(in - in_mis);
#pragma unroll 2
    for (int c = lane * 8 - lead; c < nd; c += 256) {    // the lane's 8 columns, the first of them on a 16-byte boundary of `out`
        uint32_t v[4];
        if (c < n) {
            const long at = (s0 + c) >> 3;
            if (at * 8 >= in_mis && (at + (sh ? 2 : 1)) * 8 <= in_mis + in_total) {
                const uint4 a = __ldg(pieces + at);
                const uint4 r = sh ? shifted(a, __ldg(pieces + at + 1), sh) : a;
                v[0] = r.x; v[1] = r.y; v[2] = r.z; v[3] = r.w;
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int c0 = c + 2 * e;
                    v[e] = (c0 >= 0 && c0 < n ? (uint32_t)src[c0] : 0u) | (c0 + 1 >= 0 && c0 + 1 < n ? (uint32_t)src[c0 + 1] << 16 : 0u);
                }
            }
        }
        if (c + 8 > n) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int c0 = c + 2 * e;
                if (c0 >= n) v[e] = fill16 | fill16 << 16;
                else if (c0 + 1 >= n) v[e] = (v[e] & 0xffffu) | fill16 << 16;
            }
        }
        if (c >= 0 && (c + 8 <= nd || out_padded)) {
            *reinterpret_cast<uint4*>(dst + c) = make_uint4(v[0], v[1], v[2], v[3]);
        } else {
#pragma unroll
            for (int e = 0; e < 8; ++e)
                if (c + e >= 0 && c + e < nd) dst[c + e] = (uint16_t)(v[e >> 1] >> (16 * (e & 1)));
        }
    }
}

int copy_planes(const void* in, PlaneView iv, void* out, PlaneView ov, long planes, int H, int W, int causal, bool write_upper, float fill,
                int dtype, cudaStream_t st) {
    const dim3 grid((unsigned)((H + CP_THREADS / 32 - 1) / (CP_THREADS / 32)), (unsigned)planes);
    const int in_mis = (int)(reinterpret_cast<uintptr_t>(in) / 2 % 8), out_mis = (int)(reinterpret_cast<uintptr_t>(out) / 2 % 8);
    const int out_padded = out_mis == 0 && ov.width % 8 == 0;
    const uint16_t* i16 = static_cast<const uint16_t*>(in);
    uint16_t* o16 = static_cast<uint16_t*>(out);
    const long total = planes * iv.plane_stride;
    if (dtype == MTA_BF16)
        return launch_kernel<copy_planes_kernel<__nv_bfloat16>>("copy_planes_kernel", grid, CP_THREADS, 0, st, i16, iv, in_mis, total, o16, ov, out_mis,
                                                                out_padded, H, W, causal, write_upper ? 1 : 0, fill);
    return launch_kernel<copy_planes_kernel<__half>>("copy_planes_kernel", grid, CP_THREADS, 0, st, i16, iv, in_mis, total, o16, ov, out_mis, out_padded, H, W,
                                                     causal, write_upper ? 1 : 0, fill);
}

}  // namespace

PadPlan pad_plan(long planes, int H, int W, int dtype) {
    PadPlan p;
    const int width = (W + 15) / 16 * 16;
    p.view = PlaneView{(long)H * width, 0, width};
    p.bytes = ((size_t)planes * p.view.plane_stride * 2 + 255) & ~size_t(255);
    p.use = dtype != MTA_F32 && W % 8 != 0 && planes * H * W >= PAD_MIN && planes <= 65535 && p.bytes <= PAD_MAX;
    return p;
}

int pad_planes(const void* in, PlaneView iv, void* copy, const PadPlan& p, long planes, int H, int W, int causal, int dtype, cudaStream_t st) {
    return copy_planes(in, iv, copy, p.view, planes, H, W, causal, false, 0.0f, dtype, st);
}

int unpad_planes(const void* copy, const PadPlan& p, void* out, PlaneView ov, long planes, int H, int W, int causal, float fill, int dtype,
                 cudaStream_t st) {
    return copy_planes(copy, p.view, out, ov, planes, H, W, causal, true, fill, dtype, st);
}

}  // namespace mta
