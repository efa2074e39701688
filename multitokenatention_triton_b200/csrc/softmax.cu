// Row softmax of score planes over the keys that a query may see.
//
// Stands in for F.softmax(scores.float(), dim=-1).type_as(xq) in the reference's forward
// (mta_attention_triton.py:79): fp32 arithmetic, output in the input dtype, exactly 0 above the
// diagonal.  Only keys q <= p are read when causal, so the -inf fill the reference relies on need
// not exist in memory.  `pre_scale` multiplies the logits first (the conv-attention path scales after
// its conv, conv_attention_pytorch.py:63-64); in a 16-bit dtype the scaled logit is rounded to that
// dtype as the reference's tensor multiply does.
//
// One CTA per row.  The row is read once into shared memory as fp32 (rows of up to ROW_CACHE keys;
// longer rows are re-read from global memory), reduced for the maximum and the sum of exponentials,
// and written once.
#include "kernels.cuh"

namespace mta {
namespace {

constexpr int SM_THREADS = 256;
constexpr int ROW_CACHE = 16384;    // floats of shared memory used as the row cache (64 KB)

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

template <typename T>
__global__ void __launch_bounds__(SM_THREADS)
softmax_rows_kernel(const T* __restrict__ x, PlaneView xv, T* __restrict__ y, PlaneView yv, int Q, int causal,
                    int row_begin, int write_upper, int cache_elems, float pre_scale, int round_prescaled, DeadKeys dead, int heads) {
    extern __shared__ float row[];
    __shared__ float red[SM_THREADS / 32];
    pdl_wait();
    const int p = row_begin + blockIdx.x;
    const long plane = blockIdx.y;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n = causal ? min(p + 1, Q) : Q;
    const T* xr = x + xv.at(plane, p, 0);
    T* yr = y + yv.at(plane, p, 0);
    const bool cached = n <= cache_elems;

    const long batch = plane / heads;
    auto is_dead = [&](int k) { return dead.bits && (dead.word(batch, k) >> (k & 31) & 1u); };
    float mx = -INFINITY;
    for (int k = tid; k < n; k += SM_THREADS) {
        float v = to_f32<T>(xr[k]) * pre_scale;
        if (round_prescaled) v = round_to<T>(v);
        if (is_dead(k)) v = -INFINITY;
        if (cached) row[k] = v;
        mx = fmaxf(mx, v);
    }
    mx = warp_max(mx);
    if (lane == 0) red[warp] = mx;
    __syncthreads();
    mx = red[0];
#pragma unroll
    for (int i = 1; i < SM_THREADS / 32; ++i) mx = fmaxf(mx, red[i]);
    __syncthreads();

    float sum = 0.0f;
    for (int k = tid; k < n; k += SM_THREADS) {
        float v;
        if (cached) v = row[k];
        else { v = to_f32<T>(xr[k]) * pre_scale; if (round_prescaled) v = round_to<T>(v); if (is_dead(k)) v = -INFINITY; }
        const float e = (mx == -INFINITY) ? 0.0f : __expf(v - mx);
        if (cached) row[k] = e;
        sum += e;
    }
    sum = warp_sum(sum);
    if (lane == 0) red[warp] = sum;
    __syncthreads();
    sum = 0.0f;
#pragma unroll
    for (int i = 0; i < SM_THREADS / 32; ++i) sum += red[i];
    const float inv = dead.bits && sum == 0.0f ? 0.0f : 1.0f / sum;

    // x may alias y: every thread re-reads only the elements it writes.
    for (int k = tid; k < n; k += SM_THREADS) {
        float e;
        if (cached) e = row[k];
        else { float v = to_f32<T>(xr[k]) * pre_scale; if (round_prescaled) v = round_to<T>(v); e = is_dead(k) ? 0.0f : __expf(v - mx); }
        yr[k] = from_f32<T>(e * inv);
    }
    if (write_upper)
        for (int k = n + tid; k < Q; k += SM_THREADS) yr[k] = from_f32<T>(0.0f);
}

// Vector version for 16-byte aligned rows: a CTA of 128 threads owns one row and keeps it in registers as NCH 16-byte chunks
// (8 keys, or 4 of float32) per thread, so the row is read once with 16-byte loads and written once with 16-byte stores
// (B1 H16 S2048 float32: 67 us, 119 with the general kernel).
constexpr int VT = 128;

template <typename T> __device__ __forceinline__ void unpack8(const uint4& v, float (&f)[16 / sizeof(T)]);
template <> __device__ __forceinline__ void unpack8<float>(const uint4& v, float (&f)[4]) {
    f[0] = __uint_as_float(v.x); f[1] = __uint_as_float(v.y); f[2] = __uint_as_float(v.z); f[3] = __uint_as_float(v.w);
}
template <> __device__ __forceinline__ void unpack8<__nv_bfloat16>(const uint4& v, float (&f)[8]) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) { f[2 * i] = __uint_as_float(w[i] << 16); f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u); }
}
template <> __device__ __forceinline__ void unpack8<__half>(const uint4& v, float (&f)[8]) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 t = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
        f[2 * i] = t.x; f[2 * i + 1] = t.y;
    }
}
template <typename T, int NCH>
__global__ void __launch_bounds__(VT)
softmax_rows_vec_kernel(const T* __restrict__ x, PlaneView xv, T* __restrict__ y, PlaneView yv, int Q, int causal,
                        int row_begin, int write_upper, float pre_scale, int round_prescaled, DeadKeys dead, int heads) {
    __shared__ float red[2][VT / 32];
    pdl_wait();
    const int p = row_begin + blockIdx.x;
    const long plane = blockIdx.y;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n = causal ? min(p + 1, Q) : Q;
    constexpr int VEC = 16 / (int)sizeof(T);            // keys per chunk
    const int nch = (n + VEC - 1) / VEC;                // chunks that hold at least one valid key
    const uint4* xr = reinterpret_cast<const uint4*>(x + xv.at(plane, p, 0));
    uint4* yr = reinterpret_cast<uint4*>(y + yv.at(plane, p, 0));
    const long batch = plane / heads;
    float v[NCH][VEC];
    float mx = -INFINITY;
#pragma unroll
    for (int c = 0; c < NCH; ++c) {
        const int ch = tid + c * VT;
        if (ch < nch) {
            unpack8<T>(__ldg(xr + ch), v[c]);
            const uint32_t dw = dead.word(batch, ch * VEC) >> (ch * VEC & 31);
#pragma unroll
            for (int e = 0; e < VEC; ++e) {
                float t = v[c][e] * pre_scale;
                if (round_prescaled) t = round_to<T>(t);
                if (ch * VEC + e >= n || (dw >> e & 1u)) t = -INFINITY;     // keys past the diagonal inside the last chunk
                v[c][e] = t;
                mx = fmaxf(mx, t);
            }
        }
    }
    mx = warp_max(mx);
    if (lane == 0) red[0][warp] = mx;
    __syncthreads();
    mx = fmaxf(fmaxf(red[0][0], red[0][1]), fmaxf(red[0][2], red[0][3]));
    float sum = 0.0f;
#pragma unroll
    for (int c = 0; c < NCH; ++c) {
        if (tid + c * VT < nch) {
#pragma unroll
            for (int e = 0; e < VEC; ++e) {
                const float ex = dead.bits && mx == -INFINITY ? 0.0f : __expf(v[c][e] - mx);   // exp(-inf) = 0 for the masked tail
                v[c][e] = ex;
                sum += ex;
            }
        }
    }
    sum = warp_sum(sum);
    if (lane == 0) red[1][warp] = sum;
    __syncthreads();
    sum = red[1][0] + red[1][1] + red[1][2] + red[1][3];
    const float inv = dead.bits && sum == 0.0f ? 0.0f : 1.0f / sum;
#pragma unroll
    for (int c = 0; c < NCH; ++c) {
        const int ch = tid + c * VT;
        if (ch < nch) {
            uint4 o;
            if constexpr (sizeof(T) == 4) {
                o = make_uint4(__float_as_uint(v[c][0] * inv), __float_as_uint(v[c][1] * inv), __float_as_uint(v[c][2] * inv), __float_as_uint(v[c][3] * inv));
            } else {
                o.x = pack2<T>(v[c][0] * inv, v[c][1] * inv);
                o.y = pack2<T>(v[c][2] * inv, v[c][3] * inv);
                o.z = pack2<T>(v[c][4] * inv, v[c][5] * inv);
                o.w = pack2<T>(v[c][6] * inv, v[c][7] * inv);
            }
            if (!write_upper && ch * VEC + VEC > n) {       // last chunk: keys past the diagonal stay untouched
                T* dst = reinterpret_cast<T*>(yr + ch);
                const T* src = reinterpret_cast<const T*>(&o);
                for (int e = 0; e < VEC; ++e)
                    if (ch * VEC + e < n) dst[e] = src[e];
            } else {
                yr[ch] = o;
            }
        }
    }
    if (write_upper)
        for (int ch = nch + tid; ch < (Q + VEC - 1) / VEC; ch += VT) yr[ch] = make_uint4(0u, 0u, 0u, 0u);
}

template <typename T, int NCH>
int launch_vec(const void* x, PlaneView xv, void* y, PlaneView yv, long planes, int Q, int causal, int row_begin,
               int row_end, bool write_upper, float pre_scale, int round_prescaled, DeadKeys dead, int heads, cudaStream_t st) {
    dim3 grid((unsigned)(row_end - row_begin), (unsigned)planes);
    return launch_kernel<softmax_rows_vec_kernel<T, NCH>>("softmax_rows_vec_kernel", grid, VT, 0, st, static_cast<const T*>(x), xv,
                                                          static_cast<T*>(y), yv, Q, causal, row_begin, write_upper ? 1 : 0, pre_scale, round_prescaled, dead, heads);
}

template <typename T>
int launch(const void* x, PlaneView xv, void* y, PlaneView yv, long planes, int Q, int causal, int row_begin,
           int row_end, bool write_upper, float pre_scale, int round_prescaled, DeadKeys dead, int heads, cudaStream_t st) {
    constexpr int VEC = 16 / (int)sizeof(T);
    if (Q <= 16 * VEC * VT && xv.plane_stride % VEC == 0 && yv.plane_stride % VEC == 0 && xv.width % VEC == 0 && yv.width % VEC == 0 && aligned16(x) &&
        aligned16(y)) {
        const int longest = causal ? (row_end < Q ? row_end : Q) : Q;
        const int need = (longest + VEC * VT - 1) / (VEC * VT);
        if (need <= 1) return launch_vec<T, 1>(x, xv, y, yv, planes, Q, causal, row_begin, row_end, write_upper, pre_scale, round_prescaled, dead, heads, st);
        if (need <= 2) return launch_vec<T, 2>(x, xv, y, yv, planes, Q, causal, row_begin, row_end, write_upper, pre_scale, round_prescaled, dead, heads, st);
        if (need <= 4) return launch_vec<T, 4>(x, xv, y, yv, planes, Q, causal, row_begin, row_end, write_upper, pre_scale, round_prescaled, dead, heads, st);
        if (need <= 8) return launch_vec<T, 8>(x, xv, y, yv, planes, Q, causal, row_begin, row_end, write_upper, pre_scale, round_prescaled, dead, heads, st);
        return launch_vec<T, 16>(x, xv, y, yv, planes, Q, causal, row_begin, row_end, write_upper, pre_scale, round_prescaled, dead, heads, st);
    }
    const int cache = Q < ROW_CACHE ? Q : ROW_CACHE;
    const size_t smem = (size_t)cache * sizeof(float);
    const dim3 grid((unsigned)(row_end - row_begin), (unsigned)planes);
    return launch_kernel<softmax_rows_kernel<T>>("softmax_rows_kernel", grid, SM_THREADS, smem, st, static_cast<const T*>(x), xv, static_cast<T*>(y),
                                                 yv, Q, causal, row_begin, write_upper ? 1 : 0, cache, pre_scale, round_prescaled, dead, heads);
}

// Gradient of the causal row softmax: ds = p (g - sum_k g p) over keys k <= query, fp32 arithmetic; nothing is read or written
// above the diagonal.  ds may be g.  Bound by memory (two planes in, one out): one warp per row, 16-byte chunks.  HELD > 0: rows of up to
// 32 HELD chunks, which the warp loads at once and keeps in registers; otherwise the row is walked twice, and the second walk finds it
// in L1.  H16, walked twice -> held: bf16 B16 S256 22.8 -> 16.4 us, B8 S512 28.3 -> 21.7, B4 S1024 48.7 -> 43.0; float32 B4 S512
// 28.3 -> 21.3, B1 S1024 26.5 -> 20.4.
constexpr int SB_WARPS = 8;

template <typename T, int VEC, int HELD>
__global__ void __launch_bounds__(SB_WARPS * 32)
softmax_bwd_kernel(const T* __restrict__ p, PlaneView pv, const T* g, PlaneView gv, T* ds, PlaneView dv, int P, int Q, int causal) {
    struct alignas(sizeof(T) * VEC) V { T e[VEC]; };
    pdl_wait();
    const int row = P - 1 - ((int)blockIdx.x * SB_WARPS + (threadIdx.x >> 5));     // longest rows first
    if (row < 0) return;
    const long plane = blockIdx.y;
    const int lane = threadIdx.x & 31;
    const int n = causal ? min(row + 1, Q) : Q;
    const T* pr = p + pv.at(plane, row, 0);
    const T* gr = g + gv.at(plane, row, 0);
    T* dr = ds + dv.at(plane, row, 0);
    const int whole = n / VEC;
    float dot = 0.0f;
    auto add = [&](V a, V b) {            // by value: a chunk is one 16-byte load
#pragma unroll
        for (int e = 0; e < VEC; ++e) dot = fmaf(to_f32<T>(a.e[e]), to_f32<T>(b.e[e]), dot);
    };
    auto put = [&](V a, V b, int c) {
        V o;
#pragma unroll
        for (int e = 0; e < VEC; ++e) o.e[e] = from_f32<T>(to_f32<T>(a.e[e]) * (to_f32<T>(b.e[e]) - dot));
        reinterpret_cast<V*>(dr)[c] = o;
    };
    const int tail = whole * VEC + lane;
    float tp = 0.0f, tg = 0.0f;
    if (tail < n) {
        tp = to_f32<T>(pr[tail]);
        tg = to_f32<T>(gr[tail]);
    }
    V a[HELD > 0 ? HELD : 1], b[HELD > 0 ? HELD : 1];
    if constexpr (HELD > 0) {
#pragma unroll
        for (int j = 0; j < HELD; ++j)
            if (j * 32 + lane < whole) {
                a[j] = reinterpret_cast<const V*>(pr)[j * 32 + lane];
                b[j] = reinterpret_cast<const V*>(gr)[j * 32 + lane];
            }
#pragma unroll
        for (int j = 0; j < HELD; ++j)
            if (j * 32 + lane < whole) add(a[j], b[j]);
    } else {
#pragma unroll 4
        for (int c = lane; c < whole; c += 32) add(reinterpret_cast<const V*>(pr)[c], reinterpret_cast<const V*>(gr)[c]);
    }
    if (tail < n) dot = fmaf(tp, tg, dot);
    dot = warp_sum(dot);
    if constexpr (HELD > 0) {
#pragma unroll
        for (int j = 0; j < HELD; ++j)
            if (j * 32 + lane < whole) put(a[j], b[j], j * 32 + lane);
    } else {
#pragma unroll 4
        for (int c = lane; c < whole; c += 32) put(reinterpret_cast<const V*>(pr)[c], reinterpret_cast<const V*>(gr)[c], c);
    }
    if (tail < n) dr[tail] = from_f32<T>(tp * (tg - dot));
}

template <typename T>
int launch_bwd(const void* p, PlaneView pv, const void* g, PlaneView gv, void* ds, PlaneView dv, long planes, int P, int Q, int causal,
               cudaStream_t st) {
    constexpr int VEC = 16 / (int)sizeof(T);
    auto ok = [](const void* b, const PlaneView& v) { return aligned16(b) && v.width % VEC == 0 && v.plane_stride % VEC == 0; };
    const dim3 grid((unsigned)((P + SB_WARPS - 1) / SB_WARPS), (unsigned)planes);
    const T *pt = static_cast<const T*>(p), *gt = static_cast<const T*>(g);
    T* dt = static_cast<T*>(ds);
#define MTA_SB(VECV, HELD) \
    return launch_kernel<softmax_bwd_kernel<T, VECV, HELD>>("softmax_bwd_kernel", grid, SB_WARPS * 32, 0, st, pt, pv, gt, gv, dt, dv, P, Q, causal)
    if (!(ok(p, pv) && ok(g, gv) && ok(ds, dv))) MTA_SB(1, 0);
    const int chunks = Q / VEC;
    if (chunks <= 32) MTA_SB(VEC, 1);
    if (chunks <= 64) MTA_SB(VEC, 2);
    if (chunks <= 128) MTA_SB(VEC, 4);
    if constexpr (VEC == 4) {       // eight 16-bit chunks need 152 registers a thread: bf16 B1 H16 S1536 46 us against 28 walked twice, S2048 68 against 50
        if (chunks <= 256) MTA_SB(VEC, 8);
    }
    MTA_SB(VEC, 0);
#undef MTA_SB
}

}  // namespace

int softmax_bwd_launch(const void* p, PlaneView pv, const void* g, PlaneView gv, void* ds, PlaneView dv, long planes, int P, int Q,
                       int causal, int dtype, cudaStream_t st) {
    if (planes == 0 || P == 0 || Q == 0) return MTA_OK;
    MTA_REQUIRE(planes <= 65535, "softmax_bwd: N*C = %ld exceeds 65535", planes);
    if (dtype == MTA_F32) return launch_bwd<float>(p, pv, g, gv, ds, dv, planes, P, Q, causal, st);
    if (dtype == MTA_BF16) return launch_bwd<__nv_bfloat16>(p, pv, g, gv, ds, dv, planes, P, Q, causal, st);
    return launch_bwd<__half>(p, pv, g, gv, ds, dv, planes, P, Q, causal, st);
}

int softmax_launch(const void* x, PlaneView xv, void* y, PlaneView yv, long planes, int P, int Q, int causal,
                   int row_begin, int row_end, bool write_upper, float pre_scale, int dtype, cudaStream_t st, DeadKeys dead, int heads) {
    (void)P;
    if (planes == 0 || row_end <= row_begin || Q == 0) return MTA_OK;
    MTA_REQUIRE(planes <= 65535, "softmax: N*C = %ld exceeds 65535", planes);
    switch (dtype) {
        case MTA_F32: return launch<float>(x, xv, y, yv, planes, Q, causal, row_begin, row_end, write_upper, pre_scale, (dtype != MTA_F32 && pre_scale != 1.0f) ? 1 : 0, dead, heads, st);
        case MTA_BF16: return launch<__nv_bfloat16>(x, xv, y, yv, planes, Q, causal, row_begin, row_end, write_upper, pre_scale, (dtype != MTA_F32 && pre_scale != 1.0f) ? 1 : 0, dead, heads, st);
        default: return launch<__half>(x, xv, y, yv, planes, Q, causal, row_begin, row_end, write_upper, pre_scale, (dtype != MTA_F32 && pre_scale != 1.0f) ? 1 : 0, dead, heads, st);
    }
}

}  // namespace mta
