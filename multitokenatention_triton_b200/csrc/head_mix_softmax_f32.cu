// Head mix followed by the causal row softmax in float32 as one kernel:
//   y[n,o,p,:p+1] = softmax_k( sum_h Wm[o,h] * x[n,h,p,k] ),   0 above the diagonal when the whole row is wanted
// (mta_attention_triton.py:76-79, triton_linear_head.py:76-139).
//
// A CTA owns one query row of all heads.  Its mixed logits live in shared memory: the keys are spread over the threads (a thread takes V
// neighbouring keys of all heads, as head_linear_simt_kernel does, same sums in the same order), then a warp per head takes the maximum,
// the exponentials and their sum, and writes the probabilities.  Bound: HBM, the planes are read once and written once; as two
// kernels they were read and written twice.  It takes rows whose C logits fit into shared memory (16 heads: 3504 keys).
// Measured, both stages, B1 H16: S1024 45 -> 32 us, S2048 125 -> 108 (one CTA an SM); B2 H8 S256 18 -> 9.  With the row in the warp's
// registers instead of three passes over shared memory: S1024 42, S256 11, S2048 the same.
// Every head count and every length that fits take it: a whole forward (1x1 convs) with one / two kernels, us: H4 B1 S1024 81 / 83, H8 B4 S256 53 / 59,
// H32 B1 S128 45 / 45, S512 137 / 146, S1700 1012 / 1040, H48 B1 S1024 710 / 711, H64 B1 S128 70 / 81, B4 S256 353 / 366, S860 (the longest) 711 / 711;
// over 9 head counts and 64 to 3000 keys 0.83 to 1.02 of the time of two, 1.01 or 1.02 at three of 90 sizes.
#include <algorithm>

#include "kernels.cuh"

namespace mta {
namespace {

constexpr int OG = 8;                                 // heads mixed at a time, as packed pairs

constexpr size_t MSF_SMEM_LIMIT = 220 * 1024;
int padded_keys(int Q) { return (Q + 3) & ~3; }
int padded_heads(int C) { return C <= 8 ? 8 : (C <= 16 ? 16 : (C <= 32 ? 32 : 64)); }
size_t msf_smem(int C, int Q) { return ((size_t)C * padded_keys(Q) + (size_t)padded_heads(C) * ((C + OG - 1) / OG * OG)) * sizeof(float); }

__device__ __forceinline__ float row_max(float v) {
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, s));
    return v;
}
__device__ __forceinline__ float row_sum(float v) {
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) v += __shfl_xor_sync(0xffffffffu, v, s);
    return v;
}
// (a row of nothing but -inf becomes NaN, as in softmax.cu without a mask)
__device__ __forceinline__ float4 exp4(float4 v, float mx) { return make_float4(__expf(v.x - mx), __expf(v.y - mx), __expf(v.z - mx), __expf(v.w - mx)); }

template <int CP, int V, int THREADS>
__global__ void __launch_bounds__(THREADS)
head_mix_softmax_f32_kernel(const float* __restrict__ x, PlaneView xv, const void* __restrict__ Wm, int w_dtype, float* __restrict__ y, PlaneView yv,
                            int C, int Q, int row_end, int write_upper, int early_weights) {
    extern __shared__ __align__(16) float smem[];
    const int OP = (C + OG - 1) / OG * OG, pitch = (Q + 3) & ~3;
    float* ws = smem;                                 // [h][o]
    float* rows = smem + CP * OP;                     // [o][key]
    if (!early_weights) pdl_wait();
    for (int i = threadIdx.x; i < CP * OP; i += THREADS) {
        const int h = i / OP, o = i - h * OP;
        ws[i] = h < C && o < C ? load_weight(Wm, (long)o * C + h, w_dtype) : 0.0f;
    }
    if (early_weights) pdl_wait();
    __syncthreads();
    const int p = row_end - 1 - (int)blockIdx.x;      // the longest rows first
    const long plane0 = (long)blockIdx.y * C;
    const int n = min(p + 1, Q), padded = (n + 3) & ~3;
    const float* xr = x + xv.at(plane0, p, 0);
#pragma unroll 1
    for (int k = (int)threadIdx.x * V; k < padded; k += THREADS * V) {
        float xs[CP][V];
        const int live = n - k;
#pragma unroll
        for (int h = 0; h < CP; ++h) {
            const float* src = xr + h * xv.plane_stride + k;
            if (V > 1 && live >= V && h < C) {
                if constexpr (V == 4) {
                    const float4 t = *reinterpret_cast<const float4*>(src);
                    xs[h][0] = t.x; xs[h][1] = t.y; xs[h][2] = t.z; xs[h][3] = t.w;
                } else if constexpr (V == 2) {
                    const float2 t = *reinterpret_cast<const float2*>(src);
                    xs[h][0] = t.x; xs[h][1] = t.y;
                }
            } else {
#pragma unroll
                for (int e = 0; e < V; ++e) xs[h][e] = e < live && h < C ? src[e] : 0.0f;
            }
        }
#pragma unroll 1
        for (int o0 = 0; o0 < OP; o0 += OG) {
            float2 acc[V][OG / 2];
#pragma unroll
            for (int e = 0; e < V; ++e)
#pragma unroll
                for (int j = 0; j < OG / 2; ++j) acc[e][j] = make_float2(0.0f, 0.0f);
#pragma unroll
            for (int h = 0; h < CP; ++h) {
                const float4 w0 = *reinterpret_cast<const float4*>(ws + h * OP + o0), w1 = *reinterpret_cast<const float4*>(ws + h * OP + o0 + 4);
                const float2 wv[4] = {make_float2(w0.x, w0.y), make_float2(w0.z, w0.w), make_float2(w1.x, w1.y), make_float2(w1.z, w1.w)};
#pragma unroll
                for (int e = 0; e < V; ++e) {
                    const float2 x2 = make_float2(xs[h][e], xs[h][e]);
#pragma unroll
                    for (int j = 0; j < OG / 2; ++j) acc[e][j] = __ffma2_rn(wv[j], x2, acc[e][j]);
                }
            }
#pragma unroll
            for (int j = 0; j < OG; ++j) {
                if (o0 + j >= C) break;
                float* dst = rows + (o0 + j) * pitch + k;
                float r[V];
#pragma unroll
                for (int e = 0; e < V; ++e) r[e] = e < live ? (j & 1 ? acc[e][j / 2].y : acc[e][j / 2].x) : -INFINITY;
                if constexpr (V == 4) *reinterpret_cast<float4*>(dst) = make_float4(r[0], r[1], r[2], r[3]);
                else if constexpr (V == 2) *reinterpret_cast<float2*>(dst) = make_float2(r[0], r[1]);
                else *dst = r[0];
            }
        }
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (int o = threadIdx.x >> 5; o < C; o += THREADS / 32) {
        float4* row = reinterpret_cast<float4*>(rows + o * pitch);
        const int n4 = padded / 4;
        float* yr = y + yv.at(plane0 + o, p, 0);
        auto store = [&](int i, float4 v, float inv) {
            v.x *= inv; v.y *= inv; v.z *= inv; v.w *= inv;
            if (4 * i + 3 < n) {
                *reinterpret_cast<float4*>(yr + 4 * i) = v;
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (4 * i + e < n) yr[4 * i + e] = (&v.x)[e];
            }
        };
        float mx = -INFINITY;
        for (int i = lane; i < n4; i += 32) {
            const float4 v = row[i];
            mx = fmaxf(mx, fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w)));
        }
        mx = row_max(mx);
        float sum = 0.0f;
        for (int i = lane; i < n4; i += 32) {
            const float4 v = exp4(row[i], mx);
            row[i] = v;
            sum += (v.x + v.y) + (v.z + v.w);
        }
        const float inv = 1.0f / row_sum(sum);
        for (int i = lane; i < n4; i += 32) store(i, row[i], inv);
        if (write_upper)
            for (int k = n + lane; k < Q; k += 32) yr[k] = 0.0f;
    }
}

template <int CP, int V>
int launch_msf(const void* x, PlaneView xv, const void* Wm, int w_dtype, void* y, PlaneView yv, int N, int C, int Q, int row_begin, int row_end,
               bool write_upper, bool early, cudaStream_t st) {
    const dim3 grid((unsigned)(row_end - row_begin), (unsigned)N);
    const float* xf = static_cast<const float*>(x);
    float* yf = static_cast<float*>(y);
#define MTA_MSF(THREADS)                                                                                                                        \
    return launch_kernel<head_mix_softmax_f32_kernel<CP, V, THREADS>>("head_mix_softmax_f32_kernel", grid, THREADS, msf_smem(C, Q), st, xf, xv, Wm, \
                                                                      w_dtype, yf, yv, C, Q, row_end, write_upper ? 1 : 0, early ? 1 : 0)
    // a thread's keys once or twice through the row
    if (Q <= 128 * V) MTA_MSF(128);
    if (Q <= 256 * V) MTA_MSF(256);
    MTA_MSF(512);
#undef MTA_MSF
}

}  // namespace

bool head_mix_softmax_f32_supported(const void* x, PlaneView xv, const void* y, PlaneView yv, int C, int Q, int causal, int dtype) {
    return causal && dtype == MTA_F32 && C >= 1 && C <= 64 && x != y && msf_smem(C, Q) <= MSF_SMEM_LIMIT && aligned16(x) && aligned16(y) &&
           xv.width % 4 == 0 && xv.plane_stride % 4 == 0 && yv.width % 4 == 0 && yv.plane_stride % 4 == 0;
}

int head_mix_softmax_f32_launch(const void* x, PlaneView xv, const void* Wm, int w_dtype, void* y, PlaneView yv, int N, int C, int Q, int row_begin,
                                int row_end, bool write_upper, cudaStream_t st, bool early) {
    MTA_REQUIRE(N <= 65535, "head_mix_softmax: N = %d exceeds 65535", N);
#define MTA_MSF_CASE(CP, V) return launch_msf<CP, V>(x, xv, Wm, w_dtype, y, yv, N, C, Q, row_begin, row_end, write_upper, early, st)
    if (C <= 8) MTA_MSF_CASE(8, 4);
    if (C <= 16) MTA_MSF_CASE(16, 4);
    if (C <= 32) MTA_MSF_CASE(32, 2);
    MTA_MSF_CASE(64, 1);
#undef MTA_MSF_CASE
}

}  // namespace mta
