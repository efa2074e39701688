// The depthwise conv and its weight gradient on the CUDA cores for the common odd key extents: float32, and 16-bit planes whose
// rows are not aligned for the tensor-core kernels.  Semantics: conv2d.cu (forward, and the gradient with respect to the input,
// which is the same sum with the taps reversed and the rows looking forward) and backward.cu (weight gradient).
//
// Bound: the FP32 pipe, R * S multiply-adds per position.  All sums run on the packed FMA along the key axis: a pair of
// neighbouring inputs (x[2p], x[2p+1]) meets the pair of taps that belongs to it - (w[2p], w[2p+1]) for an even output column,
// (w[2p-1], w[2p]) for an odd one - so no input pair ever has to be re-aligned; both pair tables of a row tap sit side by side
// in shared memory.  A thread owns 4 rows x 8 columns and walks the input rows: a window of 8 + S - 1 inputs is read once and
// meets the taps of every output row it belongs to (read per output row, the windows took as many shared-memory cycles as the
// FMAs).  The halo tile is staged as fp32 by 4-byte asynchronous copies (all in
// flight at once) with the causal zero applied on the way; 16-byte chunks are swizzled so that lanes 32 bytes apart hit
// different banks.
// Measured at B1 H16 S2048 11x15 float32: 295 us (conv2d_tile_kernel: 591); four CTAs an SM, which 15 key taps only get when the compiler is
// held to 128 registers (305 us with 129 and three).
#include <algorithm>

#include "kernels.cuh"

namespace mta {
namespace {

constexpr int TM = 32, TN = 128;      // output tile of a CTA
constexpr int THREADS = 128;          // 16 column groups of 8 x 8 row groups of 4

__device__ __forceinline__ void copy4(float* dst, const float* src, bool valid) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(valid ? 4 : 0) : "memory");
}
__device__ __forceinline__ void copy_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Position of column c in a staged row: 16-byte chunk c / 4 with its lowest bit flipped in every second group of 8 chunks.
__device__ __forceinline__ int staged_col(int c) { return c ^ ((c >> 3) & 4); }

// Stages rows [q_first, q_first + rows) x keys [k_first, k_first + cols) of a plane; what the conv must not see becomes 0.
template <typename T>
__device__ __forceinline__ void stage_tile(float* dst, int pitch, const T* plane, const PlaneView& v, int q_first, int rows, int q_lo, int q_hi,
                                           int k_first, int cols, int W, int causal, int tid, int nthreads) {
    const int lane = tid & 31, warp = tid >> 5, warps = nthreads >> 5;
    // a tile wholly inside what the conv sees, which most are: no comparison per element
    if (q_first >= q_lo && q_first + rows <= q_hi && k_first >= 0 && k_first + cols <= W && (!causal || k_first + cols - 1 <= q_first)) {
        const T* src = plane + (long)(q_first + warp - v.row0) * v.width + k_first + lane;
        float* d = dst + warp * pitch;
        for (int r = warp; r < rows; r += warps, src += (long)warps * v.width, d += warps * pitch) {
#pragma unroll
            for (int c = 0; c < 160; c += 32) {
                if (c >= cols) break;
                if (c + lane >= cols) continue;
                if constexpr (sizeof(T) == 4) copy4(d + staged_col(c + lane), src + c, true);
                else d[staged_col(c + lane)] = to_f32<T>(src[c]);
            }
        }
        return;
    }
    for (int r = warp; r < rows; r += warps) {
        const int q = q_first + r;
        const bool row_ok = q >= q_lo && q < q_hi;
        const int last = causal ? min(q, W - 1) : W - 1;
        const T* src = plane + (long)(q - v.row0) * v.width;
        float* d = dst + r * pitch;
#pragma unroll 5
        for (int c = lane; c < cols; c += 32) {
            const int k = k_first + c;
            const bool ok = row_ok && k >= 0 && k <= last;
            if constexpr (sizeof(T) == 4) copy4(d + staged_col(c), ok ? src + k : plane, ok);
            else d[staged_col(c)] = ok ? to_f32<T>(src[k]) : 0.0f;
        }
    }
}

template <typename T, int S>
__global__ void __launch_bounds__(THREADS, S == 15 ? 4 : 3)
conv2d_fma_kernel(const T* __restrict__ x, PlaneView xv, const void* __restrict__ w, int w_dtype, T* __restrict__ y, PlaneView yv, int C,
                  int H, int W, int R, int causal, int row_begin, int row_end, int write_upper, int tiles_n, int grad_input) {
    constexpr int NP = (S + 1) / 2;                         // tap pairs per row tap
    constexpr int WIN = 8 + S - 1;                          // inputs a thread needs per row
    constexpr int COLS = TN + S - 1, PITCH = (COLS + 15) & ~15;
    extern __shared__ __align__(16) float smem[];
    pdl_wait();
    const int th = TM + R - 1;
    float* xs = smem;                                       // th x PITCH
    float4* ws = reinterpret_cast<float4*>(smem + th * PITCH);   // R x NP: (even pair, odd pair)
    const int pad_h = grad_input ? 0 : R - 1, pad_w = grad_input ? S - 1 - (S - 1) / 2 : (S - 1) / 2;
    const long plane = blockIdx.y;
    const int tile_m = blockIdx.x / tiles_n, tile_n = blockIdx.x % tiles_n;
    const int m0 = row_begin + tile_m * TM, n0 = tile_n * TN;
    const int m_end = min(m0 + TM, row_end);
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    T* yp = y + plane * yv.plane_stride;
    const bool vec = sizeof(T) == 4 && yv.width % 4 == 0 && yv.plane_stride % 4 == 0 && reinterpret_cast<uintptr_t>(y) % 16 == 0;
    if (causal && n0 > m_end - 1) {                         // tile entirely above the diagonal: nothing to read
        if (write_upper)
            for (int r = ty; r < TM; r += 8) {
                const int q = m0 + r, k = n0 + tx * 8;
                if (q >= m_end) continue;
                T* row = yp + (long)(q - yv.row0) * yv.width + k;
                if (vec && k + 7 < W) {
                    reinterpret_cast<float4*>(row)[0] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    reinterpret_cast<float4*>(row)[1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                } else {
                    for (int e = 0; e < 8; ++e)
                        if (k + e < W) row[e] = from_f32<T>(0.0f);
                }
            }
        return;
    }
    // rows past m_end feed no output of the forward and need not be in its input view; the input gradient looks forward
    stage_tile<T>(xs, PITCH, x + plane * xv.plane_stride, xv, m0 - pad_h, th, 0, grad_input ? H : m_end, n0 - pad_w, COLS, W, causal, tid, THREADS);
    const long w0 = (plane % C) * (long)R * S;
    for (int e = tid; e < R * NP; e += THREADS) {
        const int i = e / NP, p = e % NP;
        auto tap = [&](int j) {
            if (j < 0 || j >= S) return 0.0f;
            return load_weight(w, w0 + (grad_input ? R * S - 1 - (i * S + j) : i * S + j), w_dtype);
        };
        ws[e] = make_float4(tap(2 * p), tap(2 * p + 1), tap(2 * p - 1), tap(2 * p));
    }
    copy_wait_all();
    __syncthreads();

    float2 acc[4][8];
#pragma unroll
    for (int o = 0; o < 4; ++o)
#pragma unroll
        for (int c = 0; c < 8; ++c) acc[o][c] = make_float2(0.0f, 0.0f);
#pragma unroll 1
    for (int m = 0; m < R + 3; ++m) {                       // input row m meets output row o through row tap m - o
        const float* row = xs + (ty * 4 + m) * PITCH;
        float2 xw[(WIN + 3) / 4 * 2];
#pragma unroll
        for (int c = 0; c < (WIN + 3) / 4; ++c) {
            const float4 v = *reinterpret_cast<const float4*>(row + staged_col(tx * 8 + 4 * c));
            xw[2 * c] = make_float2(v.x, v.y);
            xw[2 * c + 1] = make_float2(v.z, v.w);
        }
#pragma unroll
        for (int o = 0; o < 4; ++o) {
            const int i = m - o;
            if (i < 0 || i >= R) continue;
            const float4* wi = ws + i * NP;
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                const float4 wr = wi[p];
                const float2 we = make_float2(wr.x, wr.y), wo = make_float2(wr.z, wr.w);
#pragma unroll
                for (int c = 0; c < 8; c += 2) {
                    acc[o][c] = __ffma2_rn(xw[c / 2 + p], we, acc[o][c]);
                    acc[o][c + 1] = __ffma2_rn(xw[c / 2 + p], wo, acc[o][c + 1]);
                }
            }
        }
    }
#pragma unroll
    for (int o = 0; o < 4; ++o) {
        const int q = m0 + ty * 4 + o, k = n0 + tx * 8;
        if (q >= m_end) continue;
        T* row = yp + (long)(q - yv.row0) * yv.width + k;
        const int valid = (causal ? min(q, W - 1) : W - 1) - k + 1;          // of the 8 columns, those the conv defines
        float v[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) v[c] = c < valid ? acc[o][c].x + acc[o][c].y : 0.0f;
        const int stored = write_upper ? W - k : valid;
        if (vec && stored >= 8) {
            reinterpret_cast<float4*>(row)[0] = make_float4(v[0], v[1], v[2], v[3]);
            reinterpret_cast<float4*>(row)[1] = make_float4(v[4], v[5], v[6], v[7]);
        } else {
#pragma unroll
            for (int c = 0; c < 8; ++c)
                if (c < stored) row[c] = from_f32<T>(v[c]);
        }
    }
}

// ------------------------------------------------------------------------------------------------
// Weight gradient: a warp owns T consecutive row taps of a share of the rows and keeps their T * S sums in registers over all
// tiles of a work item; the only reduction is one warp sum per tap at the end of the item.  (Summing per tile cost a warp
// reduction per tap and 4096 positions.)  Lane = (column group of 8, half of the warp's rows).  A window of x is read once and
// meets the T rows of dy that its taps pair it with.  The taps of odd j pair the inputs with dy shifted by one column.
constexpr int DW_WARPS = 8;

// Tiles of row tile tm that hold a key <= query.
__host__ __device__ inline int dw_row_tiles(int tm, int H, int tiles_n, int causal) {
    if (!causal) return tiles_n;
    const int last = (tm + 1) * TM < H ? (tm + 1) * TM : H, n = (last + TN - 1) / TN;
    return n < tiles_n ? n : tiles_n;
}

template <typename T, int S, int TAPS>
__global__ void __launch_bounds__(DW_WARPS * 32, 2)
conv2d_dw_fma_kernel(const T* __restrict__ x, PlaneView xv, const T* __restrict__ dy, PlaneView dyv, float* __restrict__ partial, int H, int W,
                     int R, int causal, int tiles_m, int tiles_n, int parts, int row_groups) {
    constexpr int COLS = TN + S - 1, PITCH = (COLS + 15) & ~15;
    constexpr int WIN = 8 + S - 1;
    extern __shared__ __align__(16) float smem[];
    __shared__ float red[DW_WARPS][TAPS * S];
    pdl_wait();
    const int th = TM + R - 1, pad_w = (S - 1) / 2;
    float* xs = smem;                                       // (th + TAPS - 1) x PITCH
    float* gs = smem + (th + TAPS - 1) * PITCH;             // TM x TN
    const int part = blockIdx.x % parts;
    const long plane = blockIdx.x / parts;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = lane & 15, sub = lane >> 4;
    const T* xp = x + plane * xv.plane_stride;
    const T* gp = dy + plane * dyv.plane_stride;
    // warp -> taps [i0, i0 + TAPS) and rows [r0, r0 + chunk) of the tile
    const int i0 = warp / row_groups * TAPS;
    const int chunk = TM / (2 * row_groups), r0 = (warp % row_groups * 2 + sub) * chunk;
    float2 acc[TAPS][S];
#pragma unroll
    for (int t = 0; t < TAPS; ++t)
#pragma unroll
        for (int j = 0; j < S; ++j) acc[t][j] = make_float2(0.0f, 0.0f);
    for (int e = tid; e < (TAPS - 1) * PITCH; e += blockDim.x) xs[th * PITCH + e] = 0.0f;     // rows that taps past R would read
    // every parts-th of the plane's tiles that touch keys <= query
    int tm = 0, tn = part, here = dw_row_tiles(0, H, tiles_n, causal);
    for (;; tn += parts) {
        while (tn >= here && tm < tiles_m) {
            tn -= here;
            if (++tm < tiles_m) here = dw_row_tiles(tm, H, tiles_n, causal);
        }
        if (tm >= tiles_m) break;
        const int m0 = tm * TM, n0 = tn * TN;
        __syncthreads();                                    // the previous tile has been read
        stage_tile<T>(xs, PITCH, xp, xv, m0 - (R - 1), th, 0, H, n0 - pad_w, COLS, W, causal, tid, blockDim.x);
        stage_tile<T>(gs, TN, gp, dyv, m0, TM, 0, H, n0, TN, W, causal, tid, blockDim.x);
        copy_wait_all();
        __syncthreads();
#pragma unroll 1
        for (int m = 0; m < chunk + TAPS - 1; ++m) {        // x row r0 + i0 + m meets dy row r0 + m - u through tap i0 + u
            const float* row = xs + (r0 + i0 + m) * PITCH;
            float2 xw[(WIN + 3) / 4 * 2];
#pragma unroll
            for (int c = 0; c < (WIN + 3) / 4; ++c) {
                const float4 v = *reinterpret_cast<const float4*>(row + staged_col(tx * 8 + 4 * c));
                xw[2 * c] = make_float2(v.x, v.y);
                xw[2 * c + 1] = make_float2(v.z, v.w);
            }
#pragma unroll
            for (int u = 0; u < TAPS; ++u) {
                if (m - u < 0 || m - u >= chunk) continue;
                const float* grow = gs + (r0 + m - u) * TN;
                const float4 g0 = *reinterpret_cast<const float4*>(grow + staged_col(tx * 8)), g1 = *reinterpret_cast<const float4*>(grow + staged_col(tx * 8 + 4));
                const float2 ge[4] = {make_float2(g0.x, g0.y), make_float2(g0.z, g0.w), make_float2(g1.x, g1.y), make_float2(g1.z, g1.w)};
                const float2 go[5] = {make_float2(0.0f, g0.x), make_float2(g0.y, g0.z), make_float2(g0.w, g1.x), make_float2(g1.y, g1.z),
                                      make_float2(g1.w, 0.0f)};
#pragma unroll
                for (int j = 0; j < S; ++j) {
                    if (j % 2 == 0) {
#pragma unroll
                        for (int p = 0; p < 4; ++p) acc[u][j] = __ffma2_rn(xw[j / 2 + p], ge[p], acc[u][j]);
                    } else {                                // dy[c] meets x[c + j]: pairs (dy[-1], dy[0]), (dy[1], dy[2]), ...
#pragma unroll
                        for (int p = 0; p < 5; ++p) acc[u][j] = __ffma2_rn(xw[(j - 1) / 2 + p], go[p], acc[u][j]);
                    }
                }
            }
        }
    }
#pragma unroll
    for (int u = 0; u < TAPS; ++u)
#pragma unroll
        for (int j = 0; j < S; ++j) {
            float v = acc[u][j].x + acc[u][j].y;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) red[warp][u * S + j] = v;
        }
    __syncthreads();
    float* out = partial + (plane * parts + part) * (long)R * S;
    for (int e = tid; e < R * S; e += blockDim.x) {
        const int tg = e / S / TAPS, at = (e / S % TAPS) * S + e % S;
        float v = 0.0f;
        for (int gr = 0; gr < row_groups; ++gr) v += red[tg * row_groups + gr][at];
        out[e] = v;
    }
}

bool extent_ok(int S) { return S % 2 == 1 && S >= 3 && S <= 15; }

#define MTA_FMA_EXTENTS(CASE)                                                             \
    switch (S) {                                                                          \
        case 3: CASE(3); case 5: CASE(5); case 7: CASE(7); case 9: CASE(9);               \
        case 11: CASE(11); case 13: CASE(13); default: CASE(15);                          \
    }

template <typename T>
int launch_conv(const void* x, PlaneView xv, const void* w, int w_dtype, void* y, PlaneView yv, long planes, int C, int H, int W, int R, int S,
                int causal, int row_begin, int row_end, bool write_upper, bool grad_input, cudaStream_t st) {
    const int tiles_m = (row_end - row_begin + TM - 1) / TM, tiles_n = (W + TN - 1) / TN;
    const size_t smem = ((size_t)(TM + R - 1) * ((TN + S - 1 + 15) & ~15) + (size_t)R * ((S + 1) / 2) * 4) * sizeof(float);
    const dim3 grid((unsigned)(tiles_m * tiles_n), (unsigned)planes);
#define MTA_CONV_CASE(SV)                                                                                                                \
    return launch_kernel<conv2d_fma_kernel<T, SV>>("conv2d_fma_kernel", grid, THREADS, smem, st, static_cast<const T*>(x), xv, w, w_dtype, \
                                                   static_cast<T*>(y), yv, C, H, W, R, causal, row_begin, row_end, write_upper ? 1 : 0,  \
                                                   tiles_n, grad_input ? 1 : 0)
    MTA_FMA_EXTENTS(MTA_CONV_CASE)
#undef MTA_CONV_CASE
}

// Parts of a plane's tiles: equal CTAs that fill the chip's two CTAs per SM in whole waves as well as a few more parts can.
int dw_parts(long planes, int tiles, int sms) {
    const long slots = 2L * sms;
    const long least = std::max<long>(1, slots / planes);
    long best = 1;
    double best_fill = 0.0;
    for (long p = least; p <= least + 3 && p <= std::max(1, tiles / 2); ++p) {
        const double fill = (double)planes * p / (double)((planes * p + slots - 1) / slots * slots);
        if (fill > best_fill + 0.02) {
            best_fill = fill;
            best = p;
        }
    }
    if (best_fill == 0.0) best = std::max(1, tiles / 2);
    return (int)best;
}

// Row taps per warp: three, or two where three times S sums do not leave two CTAs' registers, or the taps come in pairs.
constexpr int dw_taps(int R, int S) { return S >= 13 || R == 2 || R == 4 ? 2 : 3; }

template <typename T, int S, int TAPS>
int launch_dw_taps(const void* x, PlaneView xv, const void* dy, PlaneView dyv, float* partial, long planes, int H, int W, int R, int causal,
                   int parts, cudaStream_t st) {
    const int tiles_m = (H + TM - 1) / TM, tiles_n = (W + TN - 1) / TN;
    const int tap_groups = (R + TAPS - 1) / TAPS;
    int row_groups = 1;
    while (2 * row_groups * tap_groups <= DW_WARPS) row_groups *= 2;
    const size_t smem = ((size_t)(TM + R - 1 + TAPS - 1) * ((TN + S - 1 + 15) & ~15) + (size_t)TM * TN) * sizeof(float);
    return launch_kernel<conv2d_dw_fma_kernel<T, S, TAPS>>("conv2d_dw_fma_kernel", (unsigned)(planes * parts), (unsigned)(tap_groups * row_groups * 32), smem,
                                                           st, static_cast<const T*>(x), xv, static_cast<const T*>(dy), dyv, partial, H, W, R, causal,
                                                           tiles_m, tiles_n, parts, row_groups);
}

template <typename T>
int launch_dw(const void* x, PlaneView xv, const void* dy, PlaneView dyv, float* partial, long planes, int H, int W, int R, int S, int causal,
              int parts, cudaStream_t st) {
#define MTA_DW_CASE(SV)                                                                                                        \
    if constexpr (SV < 13) {                                                                                                   \
        if (dw_taps(R, SV) == 3) return launch_dw_taps<T, SV, 3>(x, xv, dy, dyv, partial, planes, H, W, R, causal, parts, st); \
    }                                                                                                                          \
    return launch_dw_taps<T, SV, 2>(x, xv, dy, dyv, partial, planes, H, W, R, causal, parts, st)
    MTA_FMA_EXTENTS(MTA_DW_CASE)
#undef MTA_DW_CASE
}

}  // namespace

bool conv2d_fma_supported(int R, int S, long planes) { return extent_ok(S) && R <= 2 * DW_WARPS && planes <= 65535; }

int conv2d_fma_launch(const void* x, PlaneView xv, const void* w, int w_dtype, void* y, PlaneView yv, long planes, int C, int H, int W, int R,
                      int S, int causal, int row_begin, int row_end, bool write_upper, bool grad_input, int dtype, cudaStream_t st) {
#define MTA_T(TT) return launch_conv<TT>(x, xv, w, w_dtype, y, yv, planes, C, H, W, R, S, causal, row_begin, row_end, write_upper, grad_input, st)
    if (dtype == MTA_F32) MTA_T(float);
    if (dtype == MTA_BF16) MTA_T(__nv_bfloat16);
    MTA_T(__half);
#undef MTA_T
}

// Per-part sums [plane][part][R * S] in `partial`; *parts_out parts per plane, never more than `max_parts`.
int conv2d_dw_fma_launch(const void* x, PlaneView xv, const void* dy, PlaneView dyv, float* partial, int max_parts, int* parts_out, long planes,
                         int H, int W, int R, int S, int causal, int dtype, cudaStream_t st) {
    int sms = 0;
    if (int rc = sm_count(&sms)) return rc;
    int tiles = 0;
    for (int tm = 0; tm < (H + TM - 1) / TM; ++tm) tiles += dw_row_tiles(tm, H, (W + TN - 1) / TN, causal);
    const int parts = dw_parts(planes, tiles < max_parts ? tiles : max_parts, sms);
    *parts_out = parts;
#define MTA_T(TT) return launch_dw<TT>(x, xv, dy, dyv, partial, planes, H, W, R, S, causal, parts, st)
    if (dtype == MTA_F32) MTA_T(float);
    if (dtype == MTA_BF16) MTA_T(__nv_bfloat16);
    MTA_T(__half);
#undef MTA_T
}

}  // namespace mta
