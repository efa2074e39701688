// Weight gradient of the depthwise conv on tcgen05 (16-bit dtypes, key extent <= 17):
//   dw[c,i,j] = sum_{n,q,k} xh[n,c,q+i-(R-1),k+j-(S-1)/2] * dyh[n,c,q,k]
// (conv_bwd_weight_kernel, convolution_2d_trit.py:226-295; xh / dyh are x / dy inside the plane and, when causal, where key <=
// query, 0 elsewhere).
//
// As a contraction over query rows: for a row tap i and a block of 48 keys of dy,
//   D_i[kk][n] = sum_q x[q + i - (R-1)][key0 - 8 + kk] * dy[q][key0 + n],   kk < 64, n < 48,
// and dw[i][j] is the sum of D_i along the diagonal kk - n = 8 - (S-1)/2 + j.  D_i does not depend on where the block lies, so
// all blocks of a plane accumulate into the same TMEM columns and the diagonals are summed once per flush.  Both operands are
// read as they lie in memory (rows = contraction index, keys contiguous: MN-major).  One MMA (M128 N48 K16) serves two row
// taps: a row tap is the x operand's start address advanced by one row, so with "64 M elements further on" declared to be one
// row further on, the two halves of M are the same 64 keys at taps i and i + 1.
// Bound: shared-memory operand reads, 5.5 KB per MMA = 43 cycles, 8 MMAs per pair of taps and 128 x 48 positions.  (One tap per
// MMA, a 128-key window and N = 64 needed 6 KB for half of that and took 248 us where this takes 140, B4 H16 S2048 6x11 bf16; the
// CUDA-core kernel takes 1010.)
//
// A CTA owns a contiguous range of all planes' steps; what it sums up for a plane goes to a slot of the workspace and a second
// kernel adds a plane's slots in a fixed order in double.  The accumulators are flushed every DW_FLUSH steps into double
// registers, so an fp32 sum in tensor memory is never longer than 128 * DW_FLUSH products.
// Alternating accumulators from one MMA to the next (contraction steps outside, pairs inside) is slower: 163 against 148 us
// with one issuer.  Warps: 0 TMA producer, 1-2 MMA issuers (alternate pairs of taps), 4-7 zero what lies
// above the causal diagonal in the staged tiles, 8-11 flush.
#include <algorithm>

#include "kernels.cuh"
#include "tc05.cuh"

namespace mta {
namespace {
using namespace tc05;

constexpr int DW_ROWS = 128;                     // query rows per step = contraction length
constexpr int DW_KEYS = 48;                      // keys of dy per step = MMA N
constexpr int DW_THREADS = 384;
constexpr int DW_MAX_PAIRS = 10;                 // pairs of row taps: 10 x 48 TMEM columns
constexpr int DW_MAX_STAGES = 6;
constexpr int DW_DY_BYTES = DW_ROWS * 128;       // a 64-key box, of which 48 are used
constexpr int DW_FLUSH = 32;

template <typename T> struct AbFmtD;
template <> struct AbFmtD<__nv_bfloat16> { static constexpr int value = 1; };
template <> struct AbFmtD<__half> { static constexpr int value = 0; };

struct DwGeom {
    int H, W, R, S, causal;
    int pairs, nstage, slots;                    // slots of the workspace per plane
    int row_blocks, key_blocks;
    int steps;                                   // steps of a plane
    long total;                                  // of all planes
};

// Key blocks of row block tm.
__host__ __device__ inline int dw_blocks(const DwGeom& g, int tm) {
    if (!g.causal) return g.key_blocks;
    const int last = (tm + 1) * DW_ROWS < g.H ? (tm + 1) * DW_ROWS : g.H;        // one past the block's last query
    const int n = (last + DW_KEYS - 1) / DW_KEYS;
    return n < g.key_blocks ? n : g.key_blocks;
}

// CTA b of `ctas` owns steps [dw_begin(b), dw_begin(b + 1)).
__host__ __device__ inline long dw_begin(const DwGeom& g, long b, int ctas) { return b * g.total / ctas; }
// The CTA that owns a step.
__host__ __device__ inline int dw_owner(long total, long step, int ctas) { return (int)(((step + 1) * ctas - 1) / total); }

// Walks the steps of a CTA; a segment is what it owns of one plane.
struct DwIter {
    long left;                                   // steps left, the current one included
    int plane, tm, kb, nb;
    int seg_left;                                // of them in this plane
    __device__ void init(const DwGeom& g) {
        const long begin = dw_begin(g, blockIdx.x, gridDim.x);
        left = dw_begin(g, blockIdx.x + 1, gridDim.x) - begin;
        plane = (int)(begin / g.steps);
        int r = (int)(begin - (long)plane * g.steps);
        seg_left = (int)min((long)(g.steps - r), left);
        for (tm = 0;; ++tm) {
            nb = dw_blocks(g, tm);
            if (r < nb) break;
            r -= nb;
        }
        kb = r;
    }
    __device__ void next(const DwGeom& g) {
        --left;
        if (--seg_left == 0) seg_left = (int)min((long)g.steps, left);
        if (++kb == nb) {
            kb = 0;
            if (++tm == g.row_blocks) { tm = 0; ++plane; }
            nb = dw_blocks(g, tm);
        }
    }
};

// Zeroes a staged line of 64 keys (128 bytes, 128-byte swizzle, line index `line`) from key `first` on.
__device__ __forceinline__ void zero_line(uint8_t* lp, int line, int first) {
    if (first < 0) first = 0;
    for (int ch = first >> 3; ch < 8; ++ch) {
        uint4* chunk = reinterpret_cast<uint4*>(lp + ((ch ^ (line & 7)) << 4));
        if (ch * 8 >= first) {
            *chunk = make_uint4(0u, 0u, 0u, 0u);
        } else {
            uint16_t* e16 = reinterpret_cast<uint16_t*>(chunk);
            for (int e = first & 7; e < 8; ++e) e16[e] = 0;
        }
    }
}

// A segment's last step, or the last before a flush.  `s`: step within the segment.
__device__ __forceinline__ bool dw_flushes(int s, int seg_left) { return s % DW_FLUSH == DW_FLUSH - 1 || seg_left == 1; }

template <typename T>
__global__ void __launch_bounds__(DW_THREADS, 1)
conv2d_dw_tc05_kernel(const __grid_constant__ CUtensorMap mx, const __grid_constant__ CUtensorMap mdy, float* __restrict__ partial,
                      const DwGeom g, int* err_flag) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ __align__(8) uint64_t full_bar[DW_MAX_STAGES], ready_bar[DW_MAX_STAGES], empty_bar[DW_MAX_STAGES], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;
    __shared__ double red[2][2 * DW_MAX_PAIRS * 17];          // [half of the 64 keys][tap]
    const int tid = threadIdx.x, lane = tid & 31, warp = warp_index();
    const int th = DW_ROWS + 2 * g.pairs - 1;                 // staged rows of x
    const int xbox = (th * 128 + 1023) & ~1023;
    const int stage_bytes = xbox + DW_DY_BYTES;
    const int nacc = 2 * g.pairs * DW_KEYS <= 512 ? 2 : 1;    // sets of accumulators
    const uint32_t acc_cols = (uint32_t)(g.pairs * DW_KEYS);

    if (gave_up_before(err_flag, &abort_flag)) return;
    if (warp == 0) {
        if (lane == 0) {
            for (int i = 0; i < DW_MAX_STAGES; ++i) {
                mbar_init(&full_bar[i], 1);
                mbar_init(&ready_bar[i], 4);
                mbar_init(&empty_bar[i], 2);
            }
            for (int i = 0; i < 2; ++i) {
                mbar_init(&acc_full[i], 2);
                mbar_init(&acc_empty[i], 4);
            }
            fence_mbar_init();
            prefetch_tensormap(&mx);
            prefetch_tensormap(&mdy);
        }
        __syncwarp();
        tmem_alloc(&tmem_slot, 512);
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = tmem_slot;
    pdl_wait();

    // Every role walks the same steps; st / use = the step's stage and how often the stage was used before.
    DwIter it;
    it.init(g);
    int st = 0, use = 0;
    auto advance = [&] {
        if (++st == g.nstage) { st = 0; ++use; }
    };
    if (warp == 0) {
        if (lane == 0) {
            for (; it.left > 0; it.next(g), advance()) {
                mbar_wait(&empty_bar[st], (use & 1) ^ 1, err_flag);
                uint8_t* xs = smem + st * stage_bytes;
                const int key0 = it.kb * DW_KEYS, m0 = it.tm * DW_ROWS;
                mbar_expect_tx(&full_bar[st], (uint32_t)(th * 128 + DW_DY_BYTES));
                tma_load_3d(xs, &mx, &full_bar[st], key0 - 8, m0 - (g.R - 1), it.plane);
                tma_load_3d(xs + xbox, &mdy, &full_bar[st], key0, m0, it.plane);
            }
        }
    } else if (warp == 1 || warp == 2) {
        constexpr uint32_t idesc = instr_desc_f16(AbFmtD<T>::value, 1, 1, 128, DW_KEYS);
        const uint32_t el = elect_one();
        int f = 0, s = 0;                                     // flushes so far, step within the segment
        for (; it.left > 0; it.next(g), advance()) {
            const int ab = f % nacc;
            const bool fresh = s % DW_FLUSH == 0, last = dw_flushes(s, it.seg_left);
            if (fresh) mbar_wait(&acc_empty[ab], ((f / nacc) & 1) ^ 1, err_flag);
            mbar_wait(&ready_bar[st], use & 1, err_flag);
            __syncwarp();
            fence_after_sync();
            const uint32_t xa = smem_u32(smem + st * stage_bytes), ya = xa + (uint32_t)xbox;
            // x: the 64 M elements of the second tap lie one row (128 bytes) after those of the first
            const uint64_t da0 = smem_desc_sw128(xa, 128, 1024), db0 = smem_desc_sw128(ya, 16, 1024);
            for (int p = warp - 1; p < g.pairs; p += 2) {
                const uint32_t d = tmem + (uint32_t)ab * acc_cols + (uint32_t)(p * DW_KEYS);
#pragma unroll
                for (int kk = 0; kk < DW_ROWS / 16; ++kk)
                    mma_f16_ss(d, da0 + (uint64_t)(((2 * p + 16 * kk) * 128) >> 4), db0 + (uint64_t)((16 * kk * 128) >> 4), idesc,
                               (fresh && kk == 0) ? 0u : 1u, el);
            }
            mma_commit(&empty_bar[st], el);
            if (last) mma_commit(&acc_full[ab], el);
            f += last ? 1 : 0;
            s = it.seg_left == 1 ? 0 : s + 1;
        }
    } else if (warp >= 4 && warp < 8) {
        // ---- what lies above the diagonal of the staged tiles becomes zero ----
        const int mt = tid - 128;
        for (; it.left > 0; it.next(g), advance()) {
            mbar_wait(&full_bar[st], use & 1, err_flag);
            const int key0 = it.kb * DW_KEYS, m0 = it.tm * DW_ROWS, xrow = m0 - (g.R - 1);
            if (g.causal && key0 + 55 > xrow) {
                uint8_t* xs = smem + st * stage_bytes;
                for (int r = mt; r < th; r += 128) {
                    const int first = xrow + r + 1 - (key0 - 8);
                    if (first < 64) zero_line(xs + r * 128, r, first);
                }
                const int first = m0 + mt + 1 - key0;
                if (first < DW_KEYS) zero_line(xs + xbox + mt * 128, mt, first);
                fence_proxy_async();
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&ready_bar[st]);
        }
    } else if (warp >= 8) {
        // ---- flush: sums along the diagonals.  TMEM lane 32 quarter + lane = (tap quarter / 2 of the pair, kk = 32 half + lane);
        // lane j of the warp collects key tap j, which column n holds in the warp's lane n + j + 8 - pad - 32 half ----
        const int quarter = warp & 3, half = quarter & 1;
        const int from = lane + 8 - (g.S - 1) / 2 - 32 * half;
        const int n_out = flag_down(err_flag) ? g.R * g.S : 0;
        int f = 0;
        long done = 0;                                        // steps of this CTA before the segment
        const long all = it.left;
        while (done < all) {
            const int plane = it.plane, seg = it.seg_left;
            double acc[DW_MAX_PAIRS];
#pragma unroll
            for (int p = 0; p < DW_MAX_PAIRS; ++p) acc[p] = 0.0;
            for (int s0 = 0; s0 < seg; s0 += DW_FLUSH, ++f) {
                const int ab = f % nacc;
                mbar_wait(&acc_full[ab], (f / nacc) & 1, err_flag);
                fence_after_sync();
                const uint32_t t0 = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)ab * acc_cols;
#pragma unroll
                for (int p = 0; p < DW_MAX_PAIRS; ++p) {
                    if (p < g.pairs) {
                        float sum = 0.0f;
#pragma unroll 1
                        for (int c = 0; c < 3; ++c) {
                            uint32_t r[16];
                            tmem_ld_32x16(t0 + (uint32_t)(p * DW_KEYS + c * 16), r);
                            tmem_ld_wait();
#pragma unroll
                            for (int e = 0; e < 16; ++e) {
                                const int src = from + c * 16 + e;
                                const float v = __shfl_sync(0xffffffffu, __uint_as_float(r[e]), src & 31);
                                if (src >= 0 && src < 32) sum += v;
                            }
                        }
                        acc[p] += (double)sum;
                    }
                }
                fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[ab]);
            }
            if (lane < g.S) {
#pragma unroll
                for (int p = 0; p < DW_MAX_PAIRS; ++p)
                    if (p < g.pairs) red[half][(2 * p + (quarter >> 1)) * g.S + lane] = acc[p];
            }
            named_barrier(1, 128);
            const int slot = (int)blockIdx.x - dw_owner(g.total, (long)plane * g.steps, gridDim.x);
            float* out = partial + ((long)plane * g.slots + slot) * g.R * g.S;
            for (int i = tid - 256; i < n_out; i += 128) out[i] = (float)(red[0][i] + red[1][i]);
            named_barrier(1, 128);                            // nobody overwrites red while another thread still reads it
            done += seg;
            it.left -= seg;
            it.seg_left = (int)min((long)g.steps, it.left);
            ++it.plane;
        }
    }
    fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 512);
}

// dw[c, tap] = sum over the planes of channel c and the slots of each, in a fixed order, in double.
__global__ void conv2d_dw_reduce_kernel(const float* __restrict__ partial, void* __restrict__ dw, int dw_dtype, int N, int C, int taps, int slots,
                                        int steps, long total, int ctas) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    pdl_wait();
    if (i >= C * taps) return;
    const int c = i / taps, tap = i % taps;
    double acc = 0.0;
    for (int n = 0; n < N; ++n) {
        const long plane = (long)n * C + c;
        const int used = dw_owner(total, (plane + 1) * steps - 1, ctas) - dw_owner(total, plane * steps, ctas) + 1;
        for (int s = 0; s < used; ++s) acc += (double)partial[(plane * slots + s) * taps + tap];
    }
    store_weight(dw, i, dw_dtype, (float)acc);
}

DwGeom dw_geom(long planes, int H, int W, int R, int S, int causal, int sms, int* ctas) {
    DwGeom g{};
    g.H = H; g.W = W; g.R = R; g.S = S; g.causal = causal;
    g.pairs = (R + 1) / 2;
    g.row_blocks = (H + DW_ROWS - 1) / DW_ROWS;
    g.key_blocks = (W + DW_KEYS - 1) / DW_KEYS;
    for (int tm = 0; tm < g.row_blocks; ++tm) g.steps += dw_blocks(g, tm);
    g.total = planes * g.steps;
    *ctas = (int)(g.total < sms ? g.total : sms);
    const long per = g.total / *ctas;                         // the fewest steps a CTA owns
    g.slots = (int)((g.steps + per - 1) / per) + 1;
    return g;
}

template <typename T>
int launch_dw(const void* x, PlaneView xv, const void* dy, PlaneView dyv, float* partial, void* dw, int dw_dtype, int N, int C, DwGeom g, int ctas,
              cudaStream_t st) {
    CUtensorMap mx, mdy;
    int rc;
    const int th = DW_ROWS + 2 * g.pairs - 1;
    const uint64_t planes = (uint64_t)N * C;
    if ((rc = make_tensor_map_3d(&mx, x, planes, (uint64_t)g.H, (uint64_t)g.W, (uint64_t)xv.width, (uint64_t)xv.plane_stride, 64, (uint32_t)th, true))) return rc;
    if ((rc = make_tensor_map_3d(&mdy, dy, planes, (uint64_t)g.H, (uint64_t)g.W, (uint64_t)dyv.width, (uint64_t)dyv.plane_stride, 64, DW_ROWS, true))) return rc;
    int* flag = nullptr;
    if ((rc = wait_flag_ptr(&flag))) return rc;
    const size_t stage = (size_t)((th * 128 + 1023) & ~1023) + DW_DY_BYTES;
    g.nstage = (int)std::min<size_t>(DW_MAX_STAGES, (218 * 1024) / stage);
    const size_t smem = 1024 + g.nstage * stage;
    if ((rc = launch_kernel<conv2d_dw_tc05_kernel<T>>("conv2d_dw_tc05_kernel", (unsigned)ctas, DW_THREADS, smem, st, mx, mdy, partial, g, flag))) return rc;
    const int taps = g.R * g.S;
    return launch_kernel<conv2d_dw_reduce_kernel>("conv2d_dw_reduce_kernel", (unsigned)((C * taps + 63) / 64), 64, 0, st, partial, dw, dw_dtype, N, C, taps,
                                                  g.slots, g.steps, g.total, ctas);
}

}  // namespace

bool conv2d_dw_tc05_supported(const void* x, PlaneView xv, const void* dy, PlaneView dyv, int R, int S, int dtype) {
    return dtype != MTA_F32 && S <= 17 && R <= 2 * DW_MAX_PAIRS && xv.row0 == 0 && dyv.row0 == 0 && xv.width % 8 == 0 && dyv.width % 8 == 0 &&
           xv.plane_stride % 8 == 0 && dyv.plane_stride % 8 == 0 && aligned16(x) && aligned16(dy);
}

size_t conv2d_dw_tc05_workspace(int N, int C, int H, int W, int R, int S) {
    int sms = 148, ctas = 1;
    if (sm_count(&sms) != MTA_OK) sms = 148;
    size_t most = 0;
    for (int causal = 0; causal < 2; ++causal) {
        const DwGeom g = dw_geom((long)N * C, H, W, R, S, causal, sms, &ctas);
        most = std::max(most, (size_t)N * C * g.slots * R * S * sizeof(float));
    }
    return most;
}

int conv2d_dw_tc05_launch(const void* x, PlaneView xv, const void* dy, PlaneView dyv, void* dw, int dw_dtype, void* workspace, int N, int C, int H,
                          int W, int R, int S, int causal, int dtype, cudaStream_t st) {
    int sms = 0, ctas = 0;
    if (int rc = sm_count(&sms)) return rc;
    const DwGeom g = dw_geom((long)N * C, H, W, R, S, causal, sms, &ctas);
    float* partial = static_cast<float*>(workspace);
    if (dtype == MTA_BF16) return launch_dw<__nv_bfloat16>(x, xv, dy, dyv, partial, dw, dw_dtype, N, C, g, ctas, st);
    return launch_dw<__half>(x, xv, dy, dyv, partial, dw, dw_dtype, N, C, g, ctas, st);
}

}  // namespace mta
