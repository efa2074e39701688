// Weight gradients of the two stand-alone ops (the input gradients reuse the forward kernels: conv2d.cu with the
// taps reversed and the rows looking forward, head_linear.cu with the weight read transposed).
//
//   conv2d_bwd_weight    dw[c,r,s] = sum_{n,q,k} xh[n,c,q+r-(R-1),k+s-(S-1)/2] * dyh[n,c,q,k]
//                        (reference: conv_bwd_weight_kernel, convolution_2d_trit.py:226-295); xh / dyh are x / dy inside
//                        the plane and, when causal, where key <= query, 0 elsewhere
//   head_linear_bwd_weight  dW[o,h] = sum_{n,p,q<=p} dy[n,o,p,q] * x[n,h,p,q]
//                        (reference: linear_head_kernel_backward_weight, triton_linear_head.py:210-278)
//
// Both reduce over every position of every plane.  The reference accumulates with floating-point atomics; here each
// CTA writes its partial sums to a workspace and a second kernel adds them in a fixed order in double precision, so
// the result does not depend on scheduling.
#include <algorithm>

#include "kernels.cuh"

namespace mta {
namespace {

__device__ __forceinline__ float warp_sum_f(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// ------------------------------------------------------------------------------------------------
constexpr int WT_M = 32, WT_N = 128, WT_CPT = 8;
constexpr int WT_THREADS = WT_M * (WT_N / WT_CPT) / 2;     // 256: a thread owns 2 rows x 8 columns of output positions

// SC = the key extent when it is one of the common sizes (the window of a row tap then sits in registers and every tap
// indexes it statically), 0 = any size (the window is re-read from shared memory per tap).
template <typename T, int SC>
__global__ void __launch_bounds__(WT_THREADS)
conv2d_bwd_weight_kernel(const T* __restrict__ x, PlaneView xv, const T* __restrict__ dy, PlaneView dyv, float* __restrict__ partial,
                         int H, int W, int R, int S, int causal, int tiles_n) {
    extern __shared__ __align__(16) float smem[];
    const int pad_h = R - 1, pad_w = (S - 1) / 2;
    const int tw = (WT_N + S - 1 + 3) & ~3, th = WT_M + R - 1;      // row pitch a multiple of 4 floats: 16-byte window loads
    float* xs = smem;                               // th x tw, masked input
    float* part = smem + th * tw + 8;               // (WT_THREADS / 32) x R*S warp partials
    const long plane = blockIdx.y;
    const int tile_m = blockIdx.x / tiles_n, tile_n = blockIdx.x % tiles_n;
    const int m0 = tile_m * WT_M, n0 = tile_n * WT_N;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int taps = R * S;
    float* out = partial + ((long)plane * gridDim.x + blockIdx.x) * taps;
    if (causal && n0 > min(m0 + WT_M, H) - 1) {     // every dy of the tile is masked
        for (int i = tid; i < taps; i += WT_THREADS) out[i] = 0.0f;
        return;
    }
    const T* xp = x + plane * xv.plane_stride;
    const T* dp = dy + plane * dyv.plane_stride;
    for (int idx = tid; idx < th * tw; idx += WT_THREADS) {
        const int rr = idx / tw, cc = idx - rr * tw;
        const int qq = m0 - pad_h + rr, kk = n0 - pad_w + cc;
        float v = 0.0f;
        if (qq >= 0 && qq < H && kk >= 0 && kk < W && (!causal || kk <= qq)) v = to_f32<T>(xp[(long)qq * xv.width + kk]);
        xs[idx] = v;
    }
    // this thread's output positions: rows (ry, ry + WT_M/2), columns [cx, cx + 8)
    const int ry = tid / (WT_N / WT_CPT), cx = (tid % (WT_N / WT_CPT)) * WT_CPT;
    float g0[WT_CPT], g1[WT_CPT];
#pragma unroll
    for (int e = 0; e < WT_CPT; ++e) {
        const int k = n0 + cx + e, q0 = m0 + ry, q1 = m0 + ry + WT_M / 2;
        g0[e] = (q0 < H && k < W && (!causal || k <= q0)) ? to_f32<T>(dp[(long)q0 * dyv.width + k]) : 0.0f;
        g1[e] = (q1 < H && k < W && (!causal || k <= q1)) ? to_f32<T>(dp[(long)q1 * dyv.width + k]) : 0.0f;
    }
    __syncthreads();
    for (int i = 0; i < R; ++i) {
        const float* r0 = xs + (ry + i) * tw + cx;
        const float* r1 = xs + (ry + WT_M / 2 + i) * tw + cx;
        if constexpr (SC > 0) {
            constexpr int WIN = (WT_CPT + SC - 1 + 3) & ~3;
            float w0[WIN], w1[WIN];
#pragma unroll
            for (int c4 = 0; c4 < WIN / 4; ++c4) {
                const float4 a = reinterpret_cast<const float4*>(r0)[c4], b = reinterpret_cast<const float4*>(r1)[c4];
                w0[4 * c4] = a.x; w0[4 * c4 + 1] = a.y; w0[4 * c4 + 2] = a.z; w0[4 * c4 + 3] = a.w;
                w1[4 * c4] = b.x; w1[4 * c4 + 1] = b.y; w1[4 * c4 + 2] = b.z; w1[4 * c4 + 3] = b.w;
            }
#pragma unroll
            for (int j = 0; j < SC; ++j) {
                float v = 0.0f;
#pragma unroll
                for (int e = 0; e < WT_CPT; ++e) v = fmaf(w0[j + e], g0[e], fmaf(w1[j + e], g1[e], v));
                v = warp_sum_f(v);
                if (lane == 0) part[warp * taps + i * SC + j] = v;
            }
        } else {
            for (int j = 0; j < S; ++j) {
                float v = 0.0f;
#pragma unroll
                for (int e = 0; e < WT_CPT; ++e) v = fmaf(r0[j + e], g0[e], fmaf(r1[j + e], g1[e], v));
                v = warp_sum_f(v);
                if (lane == 0) part[warp * taps + i * S + j] = v;
            }
        }
    }
    __syncthreads();
    for (int i = tid; i < taps; i += WT_THREADS) {
        float v = 0.0f;
#pragma unroll
        for (int wv = 0; wv < WT_THREADS / 32; ++wv) v += part[wv * taps + i];
        out[i] = v;
    }
}

// dw[c, tap] = sum over the planes of channel c and their tiles, in a fixed order, in double.
__global__ void conv2d_bwd_weight_reduce_kernel(const float* __restrict__ partial, void* __restrict__ dw, int dw_dtype, int N, int C,
                                                int tiles, int taps) {
    __shared__ double red[256];
    pdl_wait();
    const int c = blockIdx.x / taps, tap = blockIdx.x % taps;
    double acc = 0.0;
    const long per_channel = (long)N * tiles;
    for (long i = threadIdx.x; i < per_channel; i += blockDim.x) {
        const long n = i / tiles, tile = i - n * tiles;
        acc += (double)partial[((n * C + c) * tiles + tile) * taps + tap];
    }
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) store_weight(dw, blockIdx.x, dw_dtype, (float)red[0]);
}

// ------------------------------------------------------------------------------------------------
// Weight gradient of the head mix on the CUDA cores.  Bound: the FP32 pipe, C * C multiply-adds per position.  A CTA walks
// tiles of KT keys of one row for all heads, staged as fp32 in two buffers (float32: asynchronous copies one tile ahead).  A
// thread owns a 4 x 4 block of (o, h) and every PG-th group of 4 positions: 8 16-byte loads for 32 packed FMAs (the packed
// halves are neighbouring positions, so both operands are pairs as they lie).  The 16-byte chunks of head r sit at chunk
// index c ^ ((r / 4 % 4) * 2): the four head blocks of a warp read different banks.  B1 H16 S1024 fp32: 80 us (280 with one
// (o, h) per thread).
constexpr int HW_THREADS = 256;

__device__ __forceinline__ int hw_at(int r, int k, int KT) { return r * KT + (k ^ (((r >> 2) & 3) << 3)); }

template <typename T>
__global__ void __launch_bounds__(HW_THREADS)
head_linear_bwd_weight_kernel(const T* __restrict__ x, PlaneView xv, const T* __restrict__ dy, PlaneView dyv,
                              float* __restrict__ partial, int N, int C, int P, int Q, int causal, int KT) {
    extern __shared__ __align__(16) float smem[];        // two buffers of (dy, x), C4 x KT each
    pdl_wait();
    const int CB = (C + 3) / 4, C4 = CB * 4, blocks = CB * CB;
    const int b_first = blockIdx.y * HW_THREADS, b_here = min(blocks - b_first, HW_THREADS);     // the (o, h) blocks of this CTA
    const int tid = threadIdx.x;
    const int PG = HW_THREADS / b_here, pg = tid / b_here, blk = b_first + tid % b_here;
    const int o0 = blk / CB * 4, h0 = blk % CB * 4;
    const int buf = 2 * C4 * KT;
    const int kblocks = (Q + KT - 1) / KT;
    const long tiles = (long)N * P * kblocks;
    float2 acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.0f, 0.0f);
    // the next tile from t on that has a visible key (heads C .. C4 - 1 are staged as 0)
    auto find = [&](long t) {
        while (t < tiles && causal && (int)(t % kblocks) * KT > (int)(t / kblocks % P)) t += gridDim.x;
        return t;
    };
    auto stage = [&](long t, int which) {
        if (t >= tiles) return;
        const int k0 = (int)(t % kblocks) * KT, p = (int)(t / kblocks % P);
        const long n = t / ((long)kblocks * P);
        float* gs = smem + which * buf;
        float* xs = gs + C4 * KT;
        const int n_keys = min(causal ? min(p + 1, Q) : Q, k0 + KT) - k0;
        for (int idx = tid; idx < C4 * KT; idx += HW_THREADS) {
            const int h = idx / KT, kk = idx - h * KT;
            const bool ok = h < C && kk < n_keys;
            const T* gp = ok ? dy + dyv.at(n * C + h, p, k0 + kk) : dy;
            const T* xp = ok ? x + xv.at(n * C + h, p, k0 + kk) : x;
            const int at = hw_at(h, kk, KT);
            if constexpr (sizeof(T) == 4) {
                const int bytes = ok ? 4 : 0;
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(gs + at)), "l"(gp), "r"(bytes) : "memory");
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(xs + at)), "l"(xp), "r"(bytes) : "memory");
            } else {
                gs[at] = ok ? to_f32<T>(*gp) : 0.0f;
                xs[at] = ok ? to_f32<T>(*xp) : 0.0f;
            }
        }
    };
    long t = find(blockIdx.x);
    stage(t, 0);
    asm volatile("cp.async.commit_group;" ::: "memory");
    for (int it = 0; t < tiles; ++it) {
        const long next = find(t + gridDim.x);
        stage(next, (it + 1) & 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        const int k0 = (int)(t % kblocks) * KT, p = (int)(t / kblocks % P);
        const int chunks = (min(causal ? min(p + 1, Q) : Q, k0 + KT) - k0 + 3) / 4;       // groups of 4 positions that hold a key
        const float* gs = smem + (it & 1) * buf;
        const float* xs = gs + C4 * KT;
        if (pg < PG) {
#pragma unroll 1
            for (int c = pg; c < chunks; c += PG) {
                float4 a[4], b[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    a[i] = *reinterpret_cast<const float4*>(gs + hw_at(o0 + i, c * 4, KT));
                    b[i] = *reinterpret_cast<const float4*>(xs + hw_at(h0 + i, c * 4, KT));
                }
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        acc[i][j] = __ffma2_rn(make_float2(a[i].z, a[i].w), make_float2(b[j].z, b[j].w),
                                               __ffma2_rn(make_float2(a[i].x, a[i].y), make_float2(b[j].x, b[j].y), acc[i][j]));
            }
        }
        __syncthreads();                                 // this buffer is refilled next
        t = next;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    // the position groups' sums, added in group order
    float* red = smem;                                   // [PG][b_here * 16]
    if (pg < PG) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) red[(pg * b_here + tid % b_here) * 16 + i * 4 + j] = acc[i][j].x + acc[i][j].y;
    }
    __syncthreads();
    for (int e = tid; e < b_here * 16; e += HW_THREADS) {
        const int bb = b_first + e / 16, o = bb / CB * 4 + (e & 15) / 4, h = bb % CB * 4 + (e & 3);
        float v = 0.0f;
        for (int gq = 0; gq < PG; ++gq) v += red[gq * b_here * 16 + e];
        if (o < C && h < C) partial[(long)blockIdx.x * C * C + o * C + h] = v;
    }
}

// dW = sum of the CTAs' partial sums, in a fixed order, in double.  A warp takes every 32nd slot of 32 pairs, HR_BATCH loads in flight:
// the kernel is a chain of dependent loads and additions, and 592 slots are two batches of loads and 32 + 32 additions long.
// 5.5 us for 592 slots of 256 pairs; with eight warps (74 slots each, loads and additions alternating) 23 us, twice in a training step.
constexpr int HR_SLICES = 32, HR_BATCH = 10;
__global__ void __launch_bounds__(32 * HR_SLICES)
head_linear_bwd_weight_reduce_kernel(const float* __restrict__ partial, void* __restrict__ dW, int dw_dtype, int ctas, int pairs) {
    __shared__ double red[HR_SLICES][32];
    pdl_wait();
    const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5, pair = blockIdx.x * 32 + lane;
    double acc = 0.0;
    if (pair < pairs)
        for (int i0 = slice; i0 < ctas; i0 += HR_SLICES * HR_BATCH) {
            float v[HR_BATCH];
#pragma unroll
            for (int j = 0; j < HR_BATCH; ++j) {
                const int i = i0 + j * HR_SLICES;
                v[j] = i < ctas ? partial[(long)i * pairs + pair] : 0.0f;
            }
#pragma unroll
            for (int j = 0; j < HR_BATCH; ++j) acc += (double)v[j];
        }
    red[slice][lane] = acc;
    __syncthreads();
    if (slice == 0 && pair < pairs) {
#pragma unroll
        for (int i = 1; i < HR_SLICES; ++i) acc += red[i][lane];
        store_weight(dW, pair, dw_dtype, (float)acc);
    }
}

int hw_grid(int sms) { return sms * 4; }

template <typename T>
int launch_hw(const void* x, PlaneView xv, const void* dy, PlaneView dyv, float* partial, int N, int C, int P, int Q, int causal, int grid,
              cudaStream_t st) {
    const int CB = (C + 3) / 4;
    const int KT = C <= 8 ? 512 : (C <= 16 ? 256 : (C <= 32 ? 128 : (C <= 64 ? 64 : 32)));        // 64 KB for the two buffers
    const size_t smem = (size_t)4 * CB * 4 * KT * sizeof(float);
    return launch_kernel<head_linear_bwd_weight_kernel<T>>("head_linear_bwd_weight_kernel", dim3((unsigned)grid, (unsigned)((CB * CB + HW_THREADS - 1) / HW_THREADS)),
                                                           HW_THREADS, smem, st, static_cast<const T*>(x), xv, static_cast<const T*>(dy), dyv, partial, N, C,
                                                           P, Q, causal, KT);
}

}  // namespace

// Weight gradients with a workspace that may hold padded copies of x and dy (pad.cu) behind the partial sums: 16-bit planes with unaligned
// rows then run on the tensor cores.  The CUDA-core kernels read element by element; bf16, us without / with copies: 6 x 11 conv
// N1 C8 S401 25 / 28, N1 C16 S515 40 / 32, N3 C12 S1739 435 / 192; head mix 42 / 32, 67 / 46, 650 / 204.
namespace {
// x and dy at `ws` in padded form; returns an MTA_* status.
int pad_both(const void*& x, PlaneView& xv, const void*& dy, PlaneView& dyv, const PadPlan& p, char* ws, long planes, int H, int W, int causal,
             int dtype, cudaStream_t st) {
    int rc;
    if ((rc = pad_planes(x, xv, ws, p, planes, H, W, causal, dtype, st))) return rc;
    if ((rc = pad_planes(dy, dyv, ws + p.bytes, p, planes, H, W, causal, dtype, st))) return rc;
    x = ws;
    dy = ws + p.bytes;
    xv = dyv = p.view;
    return MTA_OK;
}
}  // namespace

size_t conv2d_bwd_weight_padded_workspace(int N, int C, int H, int W, int R, int S, int dtype) {
    const PadPlan p = pad_plan((long)N * C, H, W, dtype);
    return ((conv2d_bwd_weight_workspace(N, C, H, W, R, S) + 255) & ~size_t(255)) + (p.use ? 2 * p.bytes : 0);
}

int conv2d_bwd_weight_padded(const void* x, PlaneView xv, const void* dy, PlaneView dyv, void* dw, int dw_dtype, void* workspace,
                             size_t workspace_bytes, int N, int C, int H, int W, int R, int S, int causal, int dtype, cudaStream_t st) {
    const PadPlan p = pad_plan((long)N * C, H, W, dtype);
    if (p.use && (long)N * C * H * W >= 2L << 20 && variant("conv2d") != 1 && workspace_bytes >= conv2d_bwd_weight_padded_workspace(N, C, H, W, R, S, dtype) &&
        conv2d_dw_tc05_supported(workspace, p.view, workspace, p.view, R, S, dtype)) {
        char* ws = static_cast<char*>(workspace) + ((conv2d_bwd_weight_workspace(N, C, H, W, R, S) + 255) & ~size_t(255));
        if (int rc = pad_both(x, xv, dy, dyv, p, ws, (long)N * C, H, W, causal, dtype, st)) return rc;
    }
    return conv2d_bwd_weight_launch(x, xv, dy, dyv, dw, dw_dtype, workspace, N, C, H, W, R, S, causal, dtype, st);
}

size_t head_linear_bwd_weight_padded_workspace(int N, int C, int P, int Q, int dtype) {
    const PadPlan p = pad_plan((long)N * C, P, Q, dtype);
    return ((head_linear_bwd_weight_workspace(C) + 255) & ~size_t(255)) + (p.use ? 2 * p.bytes : 0);
}

int head_linear_bwd_weight_padded(const void* x, PlaneView xv, const void* dy, PlaneView dyv, void* dW, int dw_dtype, void* workspace,
                                  size_t workspace_bytes, int N, int C, int P, int Q, int causal, int dtype, cudaStream_t st) {
    const PadPlan p = pad_plan((long)N * C, P, Q, dtype);
    if (p.use && variant("head_linear") != 1 && workspace_bytes >= head_linear_bwd_weight_padded_workspace(N, C, P, Q, dtype)) {
        char* ws = static_cast<char*>(workspace) + ((head_linear_bwd_weight_workspace(C) + 255) & ~size_t(255));
        if (int rc = pad_both(x, xv, dy, dyv, p, ws, (long)N * C, P, Q, causal, dtype, st)) return rc;
    }
    return head_linear_bwd_weight_launch(x, xv, dy, dyv, dW, dw_dtype, workspace, N, C, P, Q, causal, dtype, st);
}

size_t conv2d_bwd_weight_workspace(int N, int C, int H, int W, int R, int S) {
    const long tiles = (long)((H + WT_M - 1) / WT_M) * ((W + WT_N - 1) / WT_N);
    return std::max((size_t)N * C * tiles * R * S * sizeof(float), conv2d_dw_tc05_workspace(N, C, H, W, R, S));
}

int conv2d_bwd_weight_launch(const void* x, PlaneView xv, const void* dy, PlaneView dyv, void* dw, int dw_dtype, void* workspace, int N, int C,
                             int H, int W, int R, int S, int causal, int dtype, cudaStream_t st) {
    const int tiles_m = (H + WT_M - 1) / WT_M, tiles_n = (W + WT_N - 1) / WT_N;
    const long planes = (long)N * C;
    MTA_REQUIRE(planes <= 65535, "conv2d_bwd_weight: N*C = %ld exceeds 65535", planes);
    const int taps = R * S;
    float* partial = static_cast<float*>(workspace);
    // 16-bit dtypes with aligned rows: tensor cores (mta_set_variant("conv2d", 1): CUDA cores)
    if (variant("conv2d") != 1 && conv2d_dw_tc05_supported(x, xv, dy, dyv, R, S, dtype))
        return conv2d_dw_tc05_launch(x, xv, dy, dyv, dw, dw_dtype, workspace, N, C, H, W, R, S, causal, dtype, st);
    if (variant("conv2d") != 1 && conv2d_fma_supported(R, S, planes)) {
        int parts = 0;
        if (int rc = conv2d_dw_fma_launch(x, xv, dy, dyv, partial, tiles_m * tiles_n, &parts, planes, H, W, R, S, causal, dtype, st)) return rc;
        return launch_kernel<conv2d_bwd_weight_reduce_kernel>("conv2d_bwd_weight_reduce_kernel", (unsigned)(C * taps), 64, 0, st, partial, dw, dw_dtype, N, C,
                                                              parts, taps);
    }
    // rows padded to a multiple of 4 floats, plus slack for the last window's 16-byte over-read
    const size_t smem = ((size_t)(WT_M + R - 1) * ((WT_N + S - 1 + 3) & ~3) + 8 + (size_t)(WT_THREADS / 32) * taps) * sizeof(float);
    MTA_REQUIRE(smem <= 200 * 1024, "conv2d_bwd_weight: kernel %dx%d needs %zu bytes of shared memory (max 204800)", R, S, smem);
    dim3 grid((unsigned)(tiles_m * tiles_n), (unsigned)planes);
#define MTA_BW_LAUNCH(TT, SCV)                                                                                           \
    do {                                                                                                                 \
        if (smem > 48 * 1024)                                                                                            \
            MTA_CUDA_OK(cudaFuncSetAttribute(conv2d_bwd_weight_kernel<TT, SCV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); \
        conv2d_bwd_weight_kernel<TT, SCV><<<grid, WT_THREADS, smem, st>>>(static_cast<const TT*>(x), xv, static_cast<const TT*>(dy), dyv, \
                                                                          partial, H, W, R, S, causal, tiles_n);          \
    } while (0)
#define MTA_BW_CASE(TT)                                     \
    do {                                                    \
        switch (S) {                                        \
            case 3: MTA_BW_LAUNCH(TT, 3); break;            \
            case 5: MTA_BW_LAUNCH(TT, 5); break;            \
            case 7: MTA_BW_LAUNCH(TT, 7); break;            \
            case 11: MTA_BW_LAUNCH(TT, 11); break;          \
            case 15: MTA_BW_LAUNCH(TT, 15); break;          \
            default: MTA_BW_LAUNCH(TT, 0); break;           \
        }                                                   \
    } while (0)
    if (dtype == MTA_F32) MTA_BW_CASE(float);
    else if (dtype == MTA_BF16) MTA_BW_CASE(__nv_bfloat16);
    else MTA_BW_CASE(__half);
#undef MTA_BW_CASE
#undef MTA_BW_LAUNCH
    MTA_LAUNCH_OK("conv2d_bwd_weight_kernel");
    return launch_kernel<conv2d_bwd_weight_reduce_kernel>("conv2d_bwd_weight_reduce_kernel", (unsigned)(C * taps), 256, 0, st, partial, dw, dw_dtype, N, C,
                                                          tiles_m * tiles_n, taps);
}

size_t head_linear_bwd_weight_workspace(int C) {
    int sms = 148;
    if (sm_count(&sms) != MTA_OK) sms = 148;
    return (size_t)hw_grid(sms) * C * C * sizeof(float);
}

int head_linear_bwd_weight_launch(const void* x, PlaneView xv, const void* dy, PlaneView dyv, void* dW, int dw_dtype, void* workspace, int N, int C,
                                  int P, int Q, int causal, int dtype, cudaStream_t st) {
    int sms = 0;
    if (int bad = sm_count(&sms)) return bad;
    MTA_REQUIRE(C >= 1 && C <= 128, "head_linear_bwd_weight: C = %d heads is outside the supported range 1..128", C);
    const int grid = hw_grid(sms);
    float* partial = static_cast<float*>(workspace);
    int rc;
    int slots = grid;                                     // sums of C * C floats in `partial`
    // 16-bit dtypes with aligned rows: tensor cores (mta_set_variant("head_linear", 1): CUDA cores)
    if (variant("head_linear") != 1 && head_dw_tc05_supported(x, xv, dy, dyv, C, dtype)) {
        rc = head_dw_tc05_launch(x, xv, dy, dyv, partial, &slots, N, C, P, Q, causal, dtype, st);
    } else if (dtype == MTA_F32) rc = launch_hw<float>(x, xv, dy, dyv, partial, N, C, P, Q, causal, grid, st);
    else if (dtype == MTA_BF16) rc = launch_hw<__nv_bfloat16>(x, xv, dy, dyv, partial, N, C, P, Q, causal, grid, st);
    else rc = launch_hw<__half>(x, xv, dy, dyv, partial, N, C, P, Q, causal, grid, st);
    if (rc) return rc;
    const int pairs = C * C;
    return launch_kernel<head_linear_bwd_weight_reduce_kernel>("head_linear_bwd_weight_reduce_kernel", (unsigned)((pairs + 31) / 32), 32 * HR_SLICES, 0, st,
                                                               partial, dW, dw_dtype, slots, pairs);
}

}  // namespace mta
