// The products with a causal score plane in float32, 16-byte aligned rows (any other case: gemm_simt.cu):
//   QK  s[q,k] = scale * sum_d Q[q,d] K[k,d]      PV  o[q,d] = scale * sum_{k<=q} P[q,k] V[k,d]      PT  o[k,d] = scale * sum_{q>=k} P[q,k] V[q,d]
// Stand in for the torch.matmul calls at mta_attention_triton.py:68-71 and :89 and for their gradients.
//
// Bound: the FP32 pipe.  A CTA is four groups of 64 threads; a group multiplies a 64 x 64 output tile (8 x 8 outputs a
// thread) and has its own ring of staged blocks of 16 contraction indices, filled by cp.async two blocks ahead, and its own
// barrier, so nothing waits on a load in the steady state and the groups drift apart.  cp.async zero-fills what lies past
// its source bytes, which is how the causal edge and the ends of the tensors become zeros.  For QK the groups are a 2 x 2
// block of output tiles.  For PV and PT, whose contraction is as long as the sequence while the output is D wide, they share
// one output tile and take every fourth block: four times the parallelism for the few heavy tiles; the partial tiles are
// added in group order, so a row's sum depends only on which index lies in which block.
// The accumulators are packed pairs of columns: the packed FMA needs half the issue slots, which the operand loads then use.
// Measured at B1 H16 S2048 D64: P V 115 us (the general kernel: 532), Q K^T 131 us (183); the FMAs alone would take 64.
// Few tiles leave SMs idle and an SM with four groups needs 10 000 cycles for 64 x 64 x 256: there the groups of QK are CTAs of their own
// and the others take half as many columns.  B2 H8 S256 D64 inside the forward: Q K^T 18.7 -> 14.4 us, P V 16.4 -> 10.2.
#include "kernels.cuh"

namespace mta {
namespace {

constexpr int BT = 64;               // output tile edge of a group
constexpr int BK = 16;               // contraction indices per staged block
constexpr int GROUPS = 4;
constexpr int GTHREADS = 64;
constexpr int THREADS = GROUPS * GTHREADS;
constexpr int NST = 3;               // ring depth
constexpr int PLANE_GROUP = 16;
constexpr int KPITCH = BK + 4;       // row pitch of an operand staged [row][index]: four rows of a warp land in different banks
constexpr int OPER_K = BT * KPITCH;  // floats of an operand staged [row][index]
constexpr int OPER_N = BK * BT;      // floats of an operand staged [index][row]

enum Kind { QK, PV, PT };
constexpr int a_floats(Kind kind) { return kind == PT ? OPER_N : OPER_K; }
// bn: columns of an output tile, 64 or 32
constexpr int stage_floats(Kind kind, int bn) { return a_floats(kind) + BK * bn; }
constexpr int smem_bytes(Kind kind, int bn) { return GROUPS * NST * stage_floats(kind, bn) * (int)sizeof(float); }
static_assert(NST * stage_floats(PV, 64) >= BT * 64 && NST * stage_floats(PT, 64) >= BT * 64 && NST * stage_floats(PV, 32) >= BT * 32 &&
                  NST * stage_floats(PT, 32) >= BT * 32,
              "the partial tiles reuse the rings");

__device__ __forceinline__ void group_barrier(int group) { asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(GTHREADS) : "memory"); }
// 16 bytes to shared memory, of which only the first n floats come from src (none: src is not touched), the rest become 0.
__device__ __forceinline__ void copy16(float* dst, const float* src, int n) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int bytes = n >= 4 ? 16 : (n > 0 ? 4 * n : 0);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Rows of a thread: ty + 8 i (PT: ty * 4 + {0..3} and 32 + ty * 4 + {0..3}).  Columns of its pairs: tx * 4 + {0,1}, {2,3} and
// 32 + tx * 4 + {0,1}, {2,3}.
__device__ __forceinline__ int pair_col(int tx, int j) { return (j < 2 ? tx * 4 + 2 * j : 32 + tx * 4 + 2 * (j - 2)); }

// G groups a CTA: four, a 2 x 2 block of tiles that share their operands in L1, or one, when there are fewer blocks than SMs.
template <int G>
__global__ void __launch_bounds__(G * GTHREADS, 8 / G)
qk_f32_kernel(const float* __restrict__ q, const float* __restrict__ k, float* __restrict__ s, PlaneView sv, int S, int D, float scale,
              int causal, int row_begin, int row_end, int tiles_k) {
    extern __shared__ __align__(16) float smem[];
    pdl_wait();
    const long bh = blockIdx.x;
    constexpr int EDGE = G == 1 ? BT : 2 * BT;           // of a CTA's block
    const int tq = blockIdx.y / tiles_k, tk = blockIdx.y % tiles_k;
    if (causal && tk * EDGE > min(row_begin + (tq + 1) * EDGE, row_end) - 1) return;
    const int group = threadIdx.x / GTHREADS, gt = threadIdx.x % GTHREADS;
    const int q0 = row_begin + tq * EDGE + (group >> 1) * BT, k0 = tk * EDGE + (group & 1) * BT;
    const int q_end = min(q0 + BT, row_end);
    if (q0 >= row_end || k0 >= S || (causal && k0 > q_end - 1)) return;      // a whole group: its barrier has no other members
    const float* qp = q + (bh * S + q0) * D;
    const float* kp = k + (bh * S + k0) * D;
    float* ring = smem + group * NST * stage_floats(QK, BT);
    const int ty = gt >> 3, tx = gt & 7;
    const int blocks = (D + BK - 1) / BK;
    const int lm = gt >> 2, lq = gt & 3;          // loader: rows lm + 16 r, index quad lq of the block
    auto issue_q = [&](int b) {
        if (b < blocks) {
            float* as = ring + (b % NST) * stage_floats(QK, BT);
            const int d = b * BK + lq * 4;
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int m = lm + 16 * r, n = q0 + m < q_end ? D - d : 0;
                copy16(as + m * KPITCH + lq * 4, n > 0 ? qp + (long)m * D + d : q, n);
            }
        }
        copy_commit();
    };
    // K goes through registers into [index][key] order: keys are then pairs for the packed FMA.  Element (index c, key m) sits
    // at column (m + 8 (c / 4)) % 64: a warp's 8 keys x 4 quads store to 32 different banks.
    float4 kr[4];
    auto load_k = [&](int b) {
        const int d = b * BK + lq * 4;
#pragma unroll
        for (int r = 0; r < 4; ++r)
            kr[r] = b < blocks && k0 + lm + 16 * r < S && d < D ? __ldg(reinterpret_cast<const float4*>(kp + (long)(lm + 16 * r) * D + d))
                                                                : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    };
    float2 acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int b = 0; b < NST - 1; ++b) issue_q(b);
    load_k(0);
#pragma unroll 1
    for (int b = 0; b < blocks; ++b) {
        const float* as = ring + (b % NST) * stage_floats(QK, BT);
        float* bs = ring + (b % NST) * stage_floats(QK, BT) + OPER_K;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int col = (lm + 16 * r + 8 * lq) & (BT - 1);
#pragma unroll
            for (int e = 0; e < 4; ++e) bs[(lq * 4 + e) * BT + col] = (&kr[r].x)[e];
        }
        copy_wait<NST - 2>();
        group_barrier(group);                 // block b has landed for everyone, and everyone is done with block b - 1
        issue_q(b + NST - 1);
        load_k(b + 1);
#pragma unroll
        for (int k2 = 0; k2 < BK / 2; ++k2) {
            float2 av[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) av[i] = *reinterpret_cast<const float2*>(as + (ty + 8 * i) * KPITCH + k2 * 2);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int c = k2 * 2 + e, rot = 8 * (c >> 2);
                const float4 b0 = *reinterpret_cast<const float4*>(bs + c * BT + ((tx * 4 + rot) & (BT - 1)));
                const float4 b1 = *reinterpret_cast<const float4*>(bs + c * BT + ((32 + tx * 4 + rot) & (BT - 1)));
                const float2 bv[4] = {make_float2(b0.x, b0.y), make_float2(b0.z, b0.w), make_float2(b1.x, b1.y), make_float2(b1.z, b1.w)};
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float2 a2 = e ? make_float2(av[i].y, av[i].y) : make_float2(av[i].x, av[i].x);
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[i][j] = __ffma2_rn(a2, bv[j], acc[i][j]);
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int qq = q0 + ty + 8 * i;
        if (qq >= q_end) continue;
        const int last = causal ? min(qq, S - 1) : S - 1;
        float* row = s + sv.at(bh, qq, 0);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int kk = k0 + 32 * h + tx * 4;
            const float4 r = make_float4(acc[i][2 * h].x * scale, acc[i][2 * h].y * scale, acc[i][2 * h + 1].x * scale, acc[i][2 * h + 1].y * scale);
            if (kk + 3 <= last) *reinterpret_cast<float4*>(row + kk) = r;
            else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (kk + e <= last) row[kk + e] = (&r.x)[e];
            }
        }
    }
}

// BN: 64 columns of the output, or 32 (half of a thread's accumulators), when there are fewer tiles than SMs.
template <Kind KIND, int BN>
__global__ void __launch_bounds__(THREADS, 2)
pv_f32_kernel(const float* __restrict__ p, PlaneView pv, const float* __restrict__ v, float* __restrict__ o, int planes, int S, int D,
              int causal, int row_begin, int row_end, int tiles_d, float scale) {
    extern __shared__ __align__(16) float smem[];
    pdl_wait();
    // heaviest tiles first over groups of planes (as in gemm_tc05.cu: few enough for their V to stay in L2)
    const int n_q = (row_end - row_begin + BT - 1) / BT;
    const int per_group = n_q * tiles_d * PLANE_GROUP, in_group = (int)(blockIdx.x % per_group), p0 = (int)(blockIdx.x / per_group) * PLANE_GROUP;
    const int width = min(PLANE_GROUP, planes - p0);
    const long bh = p0 + in_group % width;
    const int t = in_group / width / tiles_d, td = in_group / width % tiles_d, tq = KIND == PT ? t : n_q - 1 - t;
    const int q0 = row_begin + tq * BT, d0 = td * BN;
    const int q_end = min(q0 + BT, row_end);
    // contraction indices [c_lo, c_hi), c_lo a multiple of BK
    const int c_lo = KIND == PT && causal ? q0 / BK * BK : 0, c_hi = KIND == PV && causal ? min(q_end, S) : S;
    const int group = threadIdx.x / GTHREADS, gt = threadIdx.x % GTHREADS;
    const float* vp = v + bh * (long)S * D + d0;
    const float* pp = p + bh * pv.plane_stride;
    float* ring = smem + group * NST * stage_floats(KIND, BN);
    const int ty = gt >> 3, tx = gt & 7;
    // blocks of this group: the absolute block index modulo 4 says whose it is, so a row range changes no sum
    const int first = c_lo / BK + ((group - c_lo / BK) & (GROUPS - 1));
    const int n_all = (c_hi + BK - 1) / BK;
    const int blocks = n_all > first ? (n_all - first + GROUPS - 1) / GROUPS : 0;
    auto issue = [&](int b) {
        if (b < blocks) {
            float* as = ring + (b % NST) * stage_floats(KIND, BN);
            float* bs = as + a_floats(KIND);
            const int c0 = (first + b * GROUPS) * BK;
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                if (KIND == PV) {
                    const int m = (gt >> 2) + 16 * r, qq = q0 + m, kk = c0 + (gt & 3) * 4;
                    const int n = qq < q_end ? min(c_hi, causal ? qq + 1 : c_hi) - kk : 0;
                    copy16(as + m * KPITCH + (gt & 3) * 4, n > 0 ? pp + (long)(qq - pv.row0) * pv.width + kk : p, n);
                } else {
                    const int c = (gt >> 4) + 4 * r, qq = c0 + c, kk = q0 + (gt & 15) * 4;
                    const int n = qq < c_hi ? min(q_end, causal ? qq + 1 : q_end) - kk : 0;
                    copy16(as + c * BT + (gt & 15) * 4, n > 0 ? pp + (long)(qq - pv.row0) * pv.width + kk : p, n);
                }
                if (r < BN / 16) {
                    const int c = gt / (BN / 4) + 256 / BN * r, d = gt % (BN / 4) * 4;
                    const int n = c0 + c < c_hi ? D - d0 - d : 0;
                    copy16(bs + c * BN + d, n > 0 ? vp + (long)(c0 + c) * D + d : v, n);
                }
            }
        }
        copy_commit();
    };
    float2 acc[8][BN / 16];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < BN / 16; ++j) acc[i][j] = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int b = 0; b < NST - 1; ++b) issue(b);
    for (int b = 0; b < blocks; ++b) {
        copy_wait<NST - 2>();
        group_barrier(group);
        issue(b + NST - 1);
        const float* as = ring + (b % NST) * stage_floats(KIND, BN);
        const float* bs = as + a_floats(KIND);
#pragma unroll
        for (int k4 = 0; k4 < BK / 4; ++k4) {
            float4 av[8];                      // PV: four indices of row ty + 8 i
            if (KIND == PV) {
#pragma unroll
                for (int i = 0; i < 8; ++i) av[i] = *reinterpret_cast<const float4*>(as + (ty + 8 * i) * KPITCH + k4 * 4);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int kk = k4 * 4 + e;
                float2 bv[BN / 16];
#pragma unroll
                for (int h = 0; h < BN / 32; ++h) {
                    const float4 b0 = *reinterpret_cast<const float4*>(bs + kk * BN + 32 * h + tx * 4);
                    bv[2 * h] = make_float2(b0.x, b0.y);
                    bv[2 * h + 1] = make_float2(b0.z, b0.w);
                }
                float a[8];
                if (KIND == PV) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) a[i] = (&av[i].x)[e];
                } else {                       // PT: rows ty * 4 .. + 3 and 32 + ty * 4 .. + 3
                    const float4 a0 = *reinterpret_cast<const float4*>(as + kk * BT + ty * 4);
                    const float4 a1 = *reinterpret_cast<const float4*>(as + kk * BT + 32 + ty * 4);
                    a[0] = a0.x; a[1] = a0.y; a[2] = a0.z; a[3] = a0.w;
                    a[4] = a1.x; a[5] = a1.y; a[6] = a1.z; a[7] = a1.w;
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float2 a2 = make_float2(a[i], a[i]);
#pragma unroll
                    for (int j = 0; j < BN / 16; ++j) acc[i][j] = __ffma2_rn(a2, bv[j], acc[i][j]);
                }
            }
        }
    }
    // the groups' partial tiles through shared memory, added in group order
    __syncthreads();
    float* part = smem + group * BT * BN;
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < BN / 16; ++j) {
            const int r = KIND == PV ? ty + 8 * i : (i < 4 ? ty * 4 + i : 32 + ty * 4 + i - 4);
            *reinterpret_cast<float2*>(part + r * BN + pair_col(tx, j)) = acc[i][j];
        }
    __syncthreads();
    float* op = o + bh * (long)S * D;
    for (int e = threadIdx.x; e < BT * BN; e += THREADS) {
        const int r = e / BN, d = d0 + e % BN;
        if (q0 + r >= q_end || d >= D) continue;
        op[(long)(q0 + r) * D + d] = (smem[e] + smem[BT * BN + e] + smem[2 * BT * BN + e] + smem[3 * BT * BN + e]) * scale;
    }
}

template <Kind KIND>
int launch_pv(const float* p, PlaneView pview, const float* v, float* o, int B, int H, int S, int D, int causal, int row_begin, int row_end,
              float scale, cudaStream_t st) {
    int sms = 0;
    if (int bad = sm_count(&sms)) return bad;
    const int tiles_q = (row_end - row_begin + BT - 1) / BT, tiles_d = (D + BT - 1) / BT, fine_d = (D + 31) / 32;
    if ((long)B * H * tiles_q * tiles_d < sms)                // a sum does not depend on the choice
        return launch_kernel<pv_f32_kernel<KIND, 32>>("pv_f32_kernel", (unsigned)(B * H * tiles_q * fine_d), THREADS, smem_bytes(KIND, 32), st, p, pview, v,
                                                      o, B * H, S, D, causal, row_begin, row_end, fine_d, scale);
    return launch_kernel<pv_f32_kernel<KIND, BT>>("pv_f32_kernel", (unsigned)(B * H * tiles_q * tiles_d), THREADS, smem_bytes(KIND, BT), st, p, pview, v, o,
                                                  B * H, S, D, causal, row_begin, row_end, tiles_d, scale);
}

}  // namespace

bool gemm_f32_supported(const void* a, const void* b, const void* c, PlaneView plane, int S, int D, int dtype) {
    // grid y holds the tiles of a plane: 128 x 128 tiles for QK, 64-row tiles times 64-column tiles for the others
    const long qk_tiles = (long)((S + 127) / 128) * ((S + 127) / 128);
    return dtype == MTA_F32 && D % 4 == 0 && plane.width % 4 == 0 && plane.plane_stride % 4 == 0 && qk_tiles <= 65535 && aligned16(a) &&
           aligned16(b) && aligned16(c);
}

int qk_f32_launch(const void* q, const void* k, void* s, PlaneView sv, int B, int H, int S, int D, float scale, int causal, int row_begin,
                  int row_end, cudaStream_t st) {
    int sms = 0;
    if (int bad = sm_count(&sms)) return bad;
    const float *qf = static_cast<const float*>(q), *kf = static_cast<const float*>(k);
    float* sf = static_cast<float*>(s);
    const int edge = 2 * BT, tiles_q = (row_end - row_begin + edge - 1) / edge, tiles_k = (S + edge - 1) / edge;
    // About half of the blocks lie above the diagonal.  A sum does not depend on the choice.
    if ((long)B * H * tiles_q * tiles_k < (causal ? 2l : 1l) * sms) {
        const int fine_q = (row_end - row_begin + BT - 1) / BT, fine_k = (S + BT - 1) / BT;
        return launch_kernel<qk_f32_kernel<1>>("qk_f32_kernel", dim3((unsigned)(B * H), (unsigned)(fine_q * fine_k)), GTHREADS, smem_bytes(QK, BT) / GROUPS, st,
                                               qf, kf, sf, sv, S, D, scale, causal, row_begin, row_end, fine_k);
    }
    return launch_kernel<qk_f32_kernel<GROUPS>>("qk_f32_kernel", dim3((unsigned)(B * H), (unsigned)(tiles_q * tiles_k)), THREADS, smem_bytes(QK, BT), st, qf, kf,
                                                sf, sv, S, D, scale, causal, row_begin, row_end, tiles_k);
}

int pv_f32_launch(const void* p, PlaneView pview, const void* v, void* o, int B, int H, int S, int D, int causal, int row_begin, int row_end,
                  bool trans, float scale, cudaStream_t st) {
    const float *pf = static_cast<const float*>(p), *vf = static_cast<const float*>(v);
    float* of = static_cast<float*>(o);
    if (trans) return launch_pv<PT>(pf, pview, vf, of, B, H, S, D, causal, row_begin, row_end, scale, st);
    return launch_pv<PV>(pf, pview, vf, of, B, H, S, D, causal, row_begin, row_end, scale, st);
}

}  // namespace mta
