// Weight gradient of the head mix on tcgen05 (16-bit dtypes, up to 128 heads):
//   dW[o,h] = sum_{n,p,q<=p} dy[n,o,p,q] * x[n,h,p,q]
// (linear_head_kernel_backward_weight, triton_linear_head.py:210-278).
//
// One TMA box holds 64 keys of R consecutive query rows of all C planes: C * R <= 128 lines, line h * R + r = row r of head h.
// With the dy box as the M operand and the x box as the N operand (both K-major, keys are the contraction),
//   D[(o,r)][(h,r')] += sum over 64 keys of dy * x;   dW[o,h] = sum_r D[(o,r)][(h,r)].
// The entries with r != r' are wasted: R - 1 of R multiplications, which the tensor pipe has to spare - 256 cycles per step
// where the step's 32 KB take 1400 at the SM's share of HBM.  Bound: HBM, two triangles read once.  D stays in tensor memory
// over all steps of a segment, so nothing is reduced inside the loop.
// A CTA owns a contiguous range of steps and cuts it into HD_SEGMENTS segments, each summed into a slot of its own: the fp32 sums
// stay short, and a second kernel adds the slots in a fixed order in double.
// Warps: 0 TMA producer, 1 MMA issuer, 2-5 zero what lies above the diagonal in both staged boxes (it may hold anything), 6-9
// read the accumulator out.
#include <algorithm>

#include "kernels.cuh"
#include "tc05.cuh"

namespace mta {
namespace {
using namespace tc05;

constexpr int HD_KEYS = 64;
constexpr int HD_BOX_BYTES = 128 * 128;
constexpr int HD_STAGE_BYTES = 2 * HD_BOX_BYTES;      // dy, x
constexpr int HD_MAX_STAGES = 6;
constexpr int HD_THREADS = 320;
constexpr int HD_SEGMENTS = 4;                        // the workspace holds four slots per SM

template <typename T> struct AbFmtW;
template <> struct AbFmtW<__nv_bfloat16> { static constexpr int value = 1; };
template <> struct AbFmtW<__half> { static constexpr int value = 0; };

struct HdGeom {
    int C, R, r_log, P, Q, causal, groups, nstage;
    int steps;               // of one batch element
    long total;              // of all
};

__host__ __device__ inline int hd_steps(const HdGeom& g, int group) {
    int keys = g.Q;
    if (g.causal) {
        const int last = (group + 1) * g.R < g.P ? (group + 1) * g.R : g.P;      // one past the group's last row
        if (last < keys) keys = last;
    }
    return (keys + HD_KEYS - 1) / HD_KEYS;
}

struct HdIter {
    long left;
    int n, group, step, count;
    __device__ void next(const HdGeom& g) {
        --left;
        if (++step == count) {
            step = 0;
            if (++group == g.groups) { group = 0; ++n; }
            count = hd_steps(g, group);
        }
    }
};

template <typename T>
__global__ void __launch_bounds__(HD_THREADS, 1)
head_dw_tc05_kernel(const __grid_constant__ CUtensorMap mdy, const __grid_constant__ CUtensorMap mx, float* __restrict__ partial,
                    const HdGeom g, uint32_t idesc, int* err_flag) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    float* picked = reinterpret_cast<float*>(smem + g.nstage * HD_STAGE_BYTES);        // [128 lines][C]
    __shared__ __align__(8) uint64_t full_bar[HD_MAX_STAGES], ready_bar[HD_MAX_STAGES], empty_bar[HD_MAX_STAGES], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;
    __shared__ HdIter first;
    const int tid = threadIdx.x, lane = tid & 31, warp = warp_index();
    const int C = g.C, R = g.R;
    if (tid == 32) {
        const long begin = blockIdx.x * g.total / gridDim.x;
        first.left = (blockIdx.x + 1) * g.total / gridDim.x - begin;
        first.n = (int)(begin / g.steps);
        int r = (int)(begin - (long)first.n * g.steps), grp = 0, cnt;
        while (r >= (cnt = hd_steps(g, grp))) { r -= cnt; ++grp; }
        first.group = grp;
        first.step = r;
        first.count = cnt;
    }
    if (gave_up_before(err_flag, &abort_flag)) return;
    if (warp == 0) {
        if (lane == 0) {
            for (int i = 0; i < HD_MAX_STAGES; ++i) {
                mbar_init(&full_bar[i], 1);
                mbar_init(&ready_bar[i], 4);
                mbar_init(&empty_bar[i], 1);
            }
            for (int i = 0; i < 2; ++i) {
                mbar_init(&acc_full[i], 1);
                mbar_init(&acc_empty[i], 4);
            }
            fence_mbar_init();
            prefetch_tensormap(&mdy);
            prefetch_tensormap(&mx);
        }
        __syncwarp();
        tmem_alloc(&tmem_slot, 256);
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = tmem_slot;
    pdl_wait();

    HdIter it = first;
    const long all = it.left;
    int st = 0, use = 0;                                  // stage of the step and how often it was used before
    auto advance = [&] {
        if (++st == g.nstage) { st = 0; ++use; }
    };
    if (warp == 0) {
        if (lane == 0) {
            for (; it.left > 0; it.next(g), advance()) {
                mbar_wait(&empty_bar[st], (use & 1) ^ 1, err_flag);
                uint8_t* sb = smem + st * HD_STAGE_BYTES;
                mbar_expect_tx(&full_bar[st], (uint32_t)(2 * C * R * 128));
                tma_load_3d(sb, &mdy, &full_bar[st], it.step * HD_KEYS, it.group * R, it.n * C);
                tma_load_3d(sb + HD_BOX_BYTES, &mx, &full_bar[st], it.step * HD_KEYS, it.group * R, it.n * C);
            }
        }
    } else if (warp == 1) {
        const uint32_t el = elect_one();
        int seg = 0, filled = 0;                          // segments begun, accumulators handed over so far
        long end = 0;
        for (long i = 0; i < all; ++i, advance()) {
            bool fresh = false;
            while (i == end) end = all * ++seg / HD_SEGMENTS, fresh = true;      // (segments without steps are skipped)
            const int ab = filled & 1;
            if (fresh) mbar_wait(&acc_empty[ab], ((filled >> 1) & 1) ^ 1, err_flag);
            mbar_wait(&ready_bar[st], use & 1, err_flag);
            __syncwarp();
            fence_after_sync();
            const uint32_t a = smem_u32(smem + st * HD_STAGE_BYTES), b = a + HD_BOX_BYTES;
#pragma unroll
            for (int kk = 0; kk < HD_KEYS / 16; ++kk)
                mma_f16_ss(tmem + (uint32_t)(ab * 128), smem_desc_sw128(a + kk * 32, 16, 1024), smem_desc_sw128(b + kk * 32, 16, 1024), idesc,
                           (fresh && kk == 0) ? 0u : 1u, el);
            mma_commit(&empty_bar[st], el);
            if (i + 1 == end) {
                mma_commit(&acc_full[ab], el);
                ++filled;
            }
        }
    } else if (warp < 6) {
        const int l = tid - 64, r = l & (R - 1);          // this thread's line
        for (; it.left > 0; it.next(g), advance()) {
            mbar_wait(&full_bar[st], use & 1, err_flag);
            const int p0 = it.group * R, k0 = it.step * HD_KEYS;
            if (g.causal && k0 + HD_KEYS - 1 > p0) {
                int zero_from = p0 + r + 1 - k0;          // first key of the line above the diagonal
                if (zero_from < 0) zero_from = 0;
                if (l < C * R) {
#pragma unroll
                    for (int box = 0; box < 2; ++box) {
                        uint8_t* lp = smem + st * HD_STAGE_BYTES + box * HD_BOX_BYTES + l * 128;
                        for (int ch = zero_from >> 3; ch < 8; ++ch) {
                            uint4* chunk = reinterpret_cast<uint4*>(lp + ((ch ^ (l & 7)) << 4));
                            if (ch * 8 >= zero_from) {
                                *chunk = make_uint4(0u, 0u, 0u, 0u);
                            } else {
                                uint16_t* e16 = reinterpret_cast<uint16_t*>(chunk);
                                for (int e = zero_from & 7; e < 8; ++e) e16[e] = 0;
                            }
                        }
                    }
                }
                fence_proxy_async();
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&ready_bar[st]);
        }
    } else {
        const int quarter = warp & 3, et = tid - 192;     // TMEM lanes this warp may read; thread index 0..127
        const int l = quarter * 32 + lane, r = l & (R - 1);
        const int n_out = flag_down(err_flag) ? C * C : 0;
        int filled = 0;
        for (int seg = 0; seg < HD_SEGMENTS; ++seg) {
            float* out = partial + ((long)blockIdx.x * HD_SEGMENTS + seg) * C * C;
            if (all * seg / HD_SEGMENTS == all * (seg + 1) / HD_SEGMENTS) {
                for (int i = et; i < n_out; i += 128) out[i] = 0.0f;
                continue;
            }
            const int ab = filled & 1;
            mbar_wait(&acc_full[ab], (filled >> 1) & 1, err_flag);
            __syncwarp();
            fence_after_sync();
#pragma unroll 1
            for (int c0 = 0; c0 < C * R; c0 += 32) {
                uint32_t v[32];
                tmem_ld_32x32(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(ab * 128 + c0), v);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 32; ++e) {
                    const int c = c0 + e;
                    if ((c & (R - 1)) == r && c < C * R) picked[l * C + (c >> g.r_log)] = __uint_as_float(v[e]);
                }
            }
            fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[ab]);
            ++filled;
            named_barrier(1, 128);
            for (int i = et; i < n_out; i += 128) {
                const int o = i / C, h = i - o * C;
                float sum = 0.0f;
                for (int rr = 0; rr < R; ++rr) sum += picked[(o * R + rr) * C + h];
                out[i] = sum;
            }
            named_barrier(1, 128);
        }
    }
    fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 256);
}

}  // namespace

bool head_dw_tc05_supported(const void* x, PlaneView xv, const void* dy, PlaneView dyv, int C, int dtype) {
    return dtype != MTA_F32 && C >= 1 && C <= 128 && xv.row0 == 0 && dyv.row0 == 0 && xv.width % 8 == 0 && dyv.width % 8 == 0 &&
           xv.plane_stride % 8 == 0 && dyv.plane_stride % 8 == 0 && aligned16(x) && aligned16(dy);
}

// Writes *slots_out sums of C * C floats to `partial` (at most four per SM).
int head_dw_tc05_launch(const void* x, PlaneView xv, const void* dy, PlaneView dyv, float* partial, int* slots_out, int N, int C, int P, int Q,
                        int causal, int dtype, cudaStream_t st) {
    HdGeom g{};
    g.C = C; g.P = P; g.Q = Q; g.causal = causal;
    g.R = 1;
    while (2 * g.R * C <= 128) { g.R *= 2; ++g.r_log; }
    g.groups = (P + g.R - 1) / g.R;
    for (int i = 0; i < g.groups; ++i) g.steps += hd_steps(g, i);
    g.total = (long)N * g.steps;
    int sms = 0, rc;
    if ((rc = sm_count(&sms))) return rc;
    CUtensorMap mdy, mx;
    if ((rc = make_tensor_map_3d_mode(&mdy, dy, (uint64_t)N * C, (uint64_t)P, (uint64_t)Q, (uint64_t)dyv.width, (uint64_t)dyv.plane_stride, 64,
                                      (uint32_t)g.R, 128, (uint32_t)C)))
        return rc;
    if ((rc = make_tensor_map_3d_mode(&mx, x, (uint64_t)N * C, (uint64_t)P, (uint64_t)Q, (uint64_t)xv.width, (uint64_t)xv.plane_stride, 64,
                                      (uint32_t)g.R, 128, (uint32_t)C)))
        return rc;
    int* flag = nullptr;
    if ((rc = wait_flag_ptr(&flag))) return rc;
    const size_t picked = (size_t)128 * C * sizeof(float);
    g.nstage = (int)std::min<size_t>(HD_MAX_STAGES, (220 * 1024 - picked) / HD_STAGE_BYTES);
    const size_t smem = 1024 + g.nstage * (size_t)HD_STAGE_BYTES + picked;
    const unsigned ctas = (unsigned)std::min<long>(g.total, sms);
    *slots_out = (int)ctas * HD_SEGMENTS;
    const int n_mma = (C * g.R + 15) / 16 * 16;
    if (dtype == MTA_BF16)
        return launch_kernel<head_dw_tc05_kernel<__nv_bfloat16>>("head_dw_tc05_kernel", ctas, HD_THREADS, smem, st, mdy, mx, partial, g,
                                                                 instr_desc_f16(AbFmtW<__nv_bfloat16>::value, 0, 0, 128, n_mma), flag);
    return launch_kernel<head_dw_tc05_kernel<__half>>("head_dw_tc05_kernel", ctas, HD_THREADS, smem, st, mdy, mx, partial, g,
                                                      instr_desc_f16(AbFmtW<__half>::value, 0, 0, 128, n_mma), flag);
}

}  // namespace mta
