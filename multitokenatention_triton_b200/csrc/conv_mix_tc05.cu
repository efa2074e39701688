// A small causal depthwise conv and the head mix that follows it as one kernel (16-bit dtypes, C = 8, 16, 32 or 64 heads):
//   y[n,o,p,k] = round16( sum_h Wm[o,h] * round16( sum_ij w[h,i,j] * x[n,h,p-(CQ-1)+i,k-(CK-1)/2+j] ) ),   0 above the diagonal
// (mta_attention_triton.py:83-86: convolution_2d_trit.py:52-135 followed by triton_linear_head.py:76-139).
//
// Every stage of the forward that touches whole score planes is bound by HBM, and the two stages after the softmax used to write a
// plane set between them.  Here a tile of all heads' rows comes in by TMA, CUDA cores compute the conv, and its 16-bit output is in
// shared memory, as the operand of the mix's MMAs, when it is complete: one plane set read, one written.
//
// A unit = (batch element n, group of R = 128 / C rows, segment of its keys), walked in tiles of 128 keys:
//   input     one TMA box of 144 keys x (R + CQ - 1) rows x C planes (the rows before the group and 8 keys on each side come with it;
//             what lies outside the plane is filled with zeros)
//   conv      8 warps; an item = 8 keys of RI consecutive rows of a head.  Packed FMAs along the keys: the 16-bit inputs are unpacked
//             twice, into pairs that begin at even and at odd keys (another unpacking costs less than moving halves of pairs, or than
//             tap pairs with a zero in them).  Input rows are read once and feed the CQ output rows that they reach.  Entries above the diagonal are
//             replaced by zeros on the way in and out.  The output goes to a tile of 128 lines (line h R + r = row r of head h) of 128
//             keys, in the layout the MMA reads with keys as the N index (two boxes of 64 keys, 128-byte swizzle).
//   mix       eight MMAs of M128 N128 K16: the weight spread over diagonal blocks (as in head_mix_tc05.cu), kept in tensor memory,
//             times the conv's tile, into accumulator tile % 2
//   epilogue  4 warps: rounded, staged, one TMA store per 32 keys x 128 rows
// Warps: 0 TMA producer, 1 MMAs, 4-11 conv, 12-15 epilogue.  The conv is the longest of the roles (3 x 3: 288 packed
// FMAs and as many other instructions for 64 results, at 2.5 cycles each), which is why larger convs stay on the tensor cores and apart.
// Measured: B8 H16 S4096 3x3 1.09 to 1.18 ms as a stage of the forward (0.93 in a first run alone), 1.67 as two kernels (HBM alone: 0.66); B4 S1024
// 49 us, 66.  On the way there: tap pairs with
// zeros in them instead of the second unpacking 1.75 ms, rows in a loop 1.21; sixteen conv warps of four rows instead of eight of
// eight are level; neighbours' pairs by shuffles instead of 4-byte reads 1.04.
#include <algorithm>

#include "kernels.cuh"
#include "tc05.cuh"

namespace mta {
namespace {
using namespace tc05;

constexpr int CM_KEYS = 128;                         // keys per tile = MMA N
constexpr int CM_COLS = CM_KEYS + 16;                // keys of the input box
constexpr int CM_PITCH = CM_COLS * 2;                // bytes of a line of it
constexpr int CM_TILE_BYTES = 128 * 256;             // the conv's output: 128 lines x 128 keys
constexpr int CM_BOX_BYTES = 128 * 128;
constexpr int CM_OUT_BYTES = 128 * 64, CM_OUT_BUFS = 3;      // output staging: 128 rows x 32 keys
constexpr int CM_CONV_THREADS = 256;
constexpr int CM_EPI_WARP = 4 + CM_CONV_THREADS / 32;          // the first of four
constexpr int CM_THREADS = (CM_EPI_WARP + 4) * 32;
constexpr int CM_MAX_STAGES = 3;
constexpr uint32_t CM_A_COL = 256;                   // the weight operand; accumulators at columns 0 and 128

template <typename T> struct AbFmtC;
template <> struct AbFmtC<__nv_bfloat16> { static constexpr int value = 1; };
template <> struct AbFmtC<__half> { static constexpr int value = 0; };

template <typename T> __device__ __forceinline__ float2 cm_unpack2(uint32_t w);
template <> __device__ __forceinline__ float2 cm_unpack2<__nv_bfloat16>(uint32_t w) {
    return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}
template <> __device__ __forceinline__ float2 cm_unpack2<__half>(uint32_t w) { return __half22float2(*reinterpret_cast<const __half2*>(&w)); }

template <typename T> __device__ __forceinline__ float cm_lo(uint32_t w) { return cm_unpack2<T>(w).x; }
template <typename T> __device__ __forceinline__ float cm_hi(uint32_t w) { return cm_unpack2<T>(w).y; }

// Keeps the first n of the two 16-bit values at positions 2 i and 2 i + 1.
__device__ __forceinline__ uint32_t cm_keep(uint32_t w, int i, int n) { return w & ((2 * i < n ? 0x0000ffffu : 0u) | (2 * i + 1 < n ? 0xffff0000u : 0u)); }

struct CmGeom {
    int N, C, R, r_log, Q, row_begin, row_end, groups, x_row0, y_row0;
    int nstage, ntile;                               // input stages, conv output tiles
    int stage_bytes, lines;                          // of an input stage
    int seg;                                         // key tiles of a unit
    long units;
};

// How many row groups reach segment s of their keys (they are the last ones).
__host__ __device__ __forceinline__ int cm_reach(const CmGeom& g, int s) {
    const int key = s * g.seg * CM_KEYS;             // a group reaches it when its last row lies beyond
    if (key >= g.row_end) return 0;
    return g.groups - (key <= g.row_begin ? 0 : (key - g.row_begin) >> g.r_log);
}
__device__ __forceinline__ int cm_tiles(const CmGeom& g, int p0) {
    const int p_last = min(p0 + g.R, g.row_end) - 1;
    return (min(p_last + 1, g.Q) + CM_KEYS - 1) / CM_KEYS;
}

// The conv of one item.  `src`: the 8 keys of staged row 0 of the item; `l0` and `strip`: the item's first line in the output tile and its
// 16-byte piece there.  `live0`: how many of the item's keys and the two before them lie on or below the diagonal in staged row 0 (one
// more with every row).  DIAG: some of them do not (a copy of its own: made into selects the comparisons would run for every tile).
template <typename T, int CQ, int CK, int RI, bool DIAG>
__device__ __forceinline__ void conv_item(const uint8_t* src, uint8_t* tile, int l0, int strip, const float* w, int live0) {
    constexpr int H = (CK - 1) / 2;
    float2 ww[CQ][CK];
#pragma unroll
    for (int i = 0; i < CQ; ++i)
#pragma unroll
        for (int j = 0; j < CK; ++j) ww[i][j] = make_float2(w[i * CK + j], w[i * CK + j]);
    float2 acc[CQ][4];                               // of the output rows in work, by row modulo CQ
    auto load = [&](int rp, uint32_t (&in)[6]) {
        const uint8_t* p = src + rp * CM_PITCH;
        const uint4 v = *reinterpret_cast<const uint4*>(p);
        in[0] = *reinterpret_cast<const uint32_t*>(p - 4);
        in[1] = v.x; in[2] = v.y; in[3] = v.z; in[4] = v.w;
        in[5] = *reinterpret_cast<const uint32_t*>(p + 16);
    };
    uint32_t next[6];
    load(0, next);
#pragma unroll
    for (int rp = 0; rp < RI + CQ - 1; ++rp) {
        uint32_t in[6];
#pragma unroll
        for (int j = 0; j < 6; ++j) in[j] = DIAG ? cm_keep(next[j], j, live0 + rp) : next[j];
        if (rp + 1 < RI + CQ - 1) load(rp + 1, next);
        // pairs of neighbouring keys that begin at an even key (even[j]: 2 j - 2, 2 j - 1) and at an odd one (odd[j]: 2 j - 1, 2 j)
        float2 even[6], odd[5];
#pragma unroll
        for (int j = 0; j < 6; ++j) even[j] = cm_unpack2<T>(in[j]);
#pragma unroll
        for (int j = 0; j < 5; ++j) odd[j] = make_float2(cm_hi<T>(in[j]), cm_lo<T>(in[j + 1]));
        // independent sums, one tap of each after the other
#pragma unroll
        for (int j = 0; j < CK; ++j)
#pragma unroll
            for (int i = 0; i < CQ; ++i) {
                if (rp - i < 0 || rp - i >= RI) continue;        // output row rp - i
                float2(&a)[4] = acc[(rp - i + CQ) % CQ];
#pragma unroll
                for (int m = 0; m < 4; ++m) {                    // keys 2 m, 2 m + 1 from the pair that begins at 2 m + j - H
                    const float2 x = (j - H) % 2 == 0 ? even[m + 1 + (j - H) / 2] : odd[m + (j - H + 1) / 2];
                    a[m] = i == 0 && j == 0 ? __fmul2_rn(x, ww[i][j]) : __ffma2_rn(x, ww[i][j], a[m]);
                }
            }
        if (rp >= CQ - 1) {                                      // output row rp - (CQ - 1) is complete
            const float2(&a)[4] = acc[(rp + 1) % CQ];
            uint32_t o[4];
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                o[m] = pack2<T>(a[m].x, a[m].y);
                if (DIAG) o[m] = cm_keep(o[m], m, live0 + rp - 2);
            }
            const int l = l0 + rp - (CQ - 1);
            *reinterpret_cast<uint4*>(tile + l * 128 + (((strip & 7) ^ (l & 7)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
        }
    }
}

template <typename T, int CQ, int CK, int RI>
__global__ void __launch_bounds__(CM_THREADS, 1)
conv_mix_tc05_kernel(const __grid_constant__ CUtensorMap mx, const __grid_constant__ CUtensorMap my, const T* __restrict__ w, const T* __restrict__ Wm,
                     const CmGeom g, int* err_flag) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ __align__(8) uint64_t full_bar[CM_MAX_STAGES], empty_bar[CM_MAX_STAGES], tile_full[2], tile_empty[2], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;
    __shared__ float wsm[64 * CQ * CK];
    uint8_t* tile_base = smem;                                       // g.ntile conv output tiles
    uint8_t* out_base = tile_base + g.ntile * CM_TILE_BYTES;         // CM_OUT_BUFS staging buffers
    uint8_t* stage_base = out_base + CM_OUT_BUFS * CM_OUT_BYTES;
    const int tid = threadIdx.x, lane = tid & 31, warp = warp_index();
    const int C = g.C, R = g.R;

    if (gave_up_before(err_flag, &abort_flag)) return;
    if (warp == 0) {
        if (lane == 0) {
            for (int i = 0; i < CM_MAX_STAGES; ++i) {
                mbar_init(&full_bar[i], 1);
                mbar_init(&empty_bar[i], CM_CONV_THREADS / 32);
            }
            for (int i = 0; i < 2; ++i) {
                mbar_init(&tile_full[i], CM_CONV_THREADS / 32);
                mbar_init(&tile_empty[i], 1);
                mbar_init(&acc_full[i], 1);
                mbar_init(&acc_empty[i], 4);
            }
            fence_mbar_init();
            prefetch_tensormap(&mx);
            prefetch_tensormap(&my);
        }
        __syncwarp();
        tmem_alloc(&tmem_slot, 512);
    }
    for (int i = tid; i < C * CQ * CK; i += CM_THREADS) wsm[i] = to_f32<T>(w[i]);
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = 0;                                         // the allocation is all of tensor memory
    if (warp >= CM_EPI_WARP) {
        // The weight operand: lane m = o R + r, contraction index k = h R + r' two to a column; Wm[o,h] where r = r', else 0.
        const int m = (warp & 3) * 32 + lane, r = m & (R - 1), o = m >> g.r_log;
#pragma unroll 1
        for (int c0 = 0; c0 < 64; c0 += 32) {
            uint32_t pk[32];
#pragma unroll
            for (int c = 0; c < 32; ++c) {
                const int k = 2 * (c0 + c);
                const float lo = (k & (R - 1)) == r ? to_f32<T>(Wm[o * C + (k >> g.r_log)]) : 0.0f;
                const float hi = ((k + 1) & (R - 1)) == r ? to_f32<T>(Wm[o * C + ((k + 1) >> g.r_log)]) : 0.0f;
                pk[c] = pack2<T>(lo, hi);
            }
            tmem_st_32x32(tmem + ((uint32_t)((warp & 3) * 32) << 16) + CM_A_COL + (uint32_t)c0, pk);
        }
        tmem_st_wait();
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    pdl_wait();

    // Units are dealt to the CTAs in rounds of alternating direction: every group's first segment, the last groups first, then the second
    // segments, and so on, so that all but a group's last are equally long.  Neighbouring row groups, which share CQ - 1 input rows,
    // are in work at the same time.
#define CM_FOR_UNITS                                                                                   \
    for (long rnd = 0;; ++rnd) {                                                                       \
        const long u = rnd * gridDim.x + ((rnd & 1) ? gridDim.x - 1 - blockIdx.x : blockIdx.x);        \
        if (u >= g.units) break;                                                                       \
        const int n = (int)(u % g.N);                                                                  \
        int v = (int)(u / g.N), s = 0;                                                                 \
        for (int c; v >= (c = cm_reach(g, s)); ++s) v -= c;                                            \
        const int p0 = g.row_begin + (g.groups - 1 - v) * R;                                           \
        const int kt0 = s * g.seg, kt1 = min(kt0 + g.seg, cm_tiles(g, p0));                            \
        (void)n;

    if (warp == 0) {
        if (lane == 0) {
            int st = 0, use = 0;
            CM_FOR_UNITS
                for (int kt = kt0; kt < kt1; ++kt) {
                    mbar_wait(&empty_bar[st], (use & 1) ^ 1, err_flag);
                    mbar_expect_tx(&full_bar[st], (uint32_t)(g.lines * CM_PITCH));
                    tma_load_3d(stage_base + st * g.stage_bytes, &mx, &full_bar[st], kt * CM_KEYS - 8, p0 - (CQ - 1) - g.x_row0, n * C);
                    if (++st == g.nstage) { st = 0; ++use; }
                }
            }
        }
    } else if (warp == 1) {
        constexpr uint32_t idesc = instr_desc_f16(AbFmtC<T>::value, 0, 1, 128, CM_KEYS);
        const uint32_t el = elect_one();
        int tb = 0, tuse = 0, it = 0;
        CM_FOR_UNITS
            const int count = uniform(kt1 - kt0);
            for (int i = 0; i < count; ++i, ++it) {
                const int ab = it & 1;
                mbar_wait_spin(&acc_empty[ab], ((it >> 1) & 1) ^ 1, err_flag);
                mbar_wait_spin(&tile_full[tb], tuse & 1, err_flag);
                __syncwarp();
                fence_after_sync();
                const uint64_t db = smem_desc_sw128(smem_u32(tile_base + tb * CM_TILE_BYTES), CM_BOX_BYTES, 1024);
#pragma unroll
                for (int kk = 0; kk < 8; ++kk)
                    mma_f16_ts(tmem + (uint32_t)(ab * CM_KEYS), tmem + CM_A_COL + (uint32_t)(kk * 8), db + (uint64_t)(kk * 128), idesc, kk > 0 ? 1u : 0u, el);
                mma_commit(&tile_empty[tb], el);
                mma_commit(&acc_full[ab], el);
                if (++tb == g.ntile) { tb = 0; ++tuse; }
            }
        }
    } else if (warp >= 4 && warp < CM_EPI_WARP) {
        const int ct = tid - 128;
        const int parts = R / RI, items = C * 16 * parts, in_rows = R + CQ - 1;
        int st = 0, use = 0, tb = 0, tuse = 0;
        CM_FOR_UNITS
            for (int kt = kt0; kt < kt1; ++kt) {
                const int key0 = kt * CM_KEYS;
                mbar_wait(&tile_empty[tb], (tuse & 1) ^ 1, err_flag);            // the MMAs have read what was there
                mbar_wait(&full_bar[st], use & 1, err_flag);
                const uint8_t* stage = stage_base + st * g.stage_bytes;
                uint8_t* tile = tile_base + tb * CM_TILE_BYTES;
                const bool diag = key0 + CM_KEYS + 1 > p0 - (CQ - 1);            // some staged key above some staged row
#pragma unroll 1
                for (int i = ct; i < items; i += CM_CONV_THREADS) {
                    const int strip = i & 15, hp = i >> 4, part = hp % parts, h = hp / parts;
                    const int r0 = part * RI;
                    const uint8_t* src = stage + (h * in_rows + r0) * CM_PITCH + 16 + strip * 16;
                    uint8_t* box = tile + (strip >> 3) * CM_BOX_BYTES;
                    const int live0 = p0 - (CQ - 1) + r0 - (key0 + strip * 8 - 2) + 1;
                    if (diag) conv_item<T, CQ, CK, RI, true>(src, box, h * R + r0, strip, wsm + h * CQ * CK, live0);
                    else conv_item<T, CQ, CK, RI, false>(src, box, h * R + r0, strip, wsm + h * CQ * CK, live0);
                }
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&empty_bar[st]);
                    mbar_arrive(&tile_full[tb]);
                }
                if (++st == g.nstage) { st = 0; ++use; }
                if (++tb == g.ntile) { tb = 0; ++tuse; }
            }
        }
    } else if (warp >= CM_EPI_WARP) {
        const int quarter = warp & 3, m = quarter * 32 + lane;
        const bool issuer = warp == CM_EPI_WARP && lane == 0 && flag_down(err_flag);
        int it = 0, ob = 0;
        CM_FOR_UNITS
            const int unit_keys = min(min(p0 + R, g.row_end), g.Q);              // keys that some row of the unit may see
            for (int kt = kt0; kt < kt1; ++kt, ++it) {
                const int ab = it & 1, key0 = kt * CM_KEYS;
                mbar_wait(&acc_full[ab], (it >> 1) & 1, err_flag);
                __syncwarp();
                fence_after_sync();
                const uint32_t tacc = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(ab * CM_KEYS);
                // the same count for all four warps, which meet at a barrier per 32 keys
                const int chunks = min(4, (unit_keys - key0 + 31) / 32);
                uint32_t r[32];
                tmem_ld_32x32(tacc, r);
#pragma unroll 1
                for (int c = 0; c < chunks; ++c) {
                    uint32_t pk[16];
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 16; ++e) pk[e] = pack2<T>(__uint_as_float(r[2 * e]), __uint_as_float(r[2 * e + 1]));
                    if (c + 1 < chunks) {
                        tmem_ld_32x32(tacc + (uint32_t)(c * 32 + 32), r);        // on its way while this one is stored
                    } else {
                        fence_before_sync();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&acc_empty[ab]);
                    }
                    uint8_t* obuf = out_base + ob * CM_OUT_BYTES;
#pragma unroll
                    for (int q4 = 0; q4 < 4; ++q4)
                        *reinterpret_cast<uint4*>(obuf + m * 64 + ((q4 ^ ((m >> 1) & 3)) << 4)) =
                            make_uint4(pk[4 * q4], pk[4 * q4 + 1], pk[4 * q4 + 2], pk[4 * q4 + 3]);
                    fence_proxy_async();
                    // three buffers: the one that is written next was read by the store before the last
                    if (issuer) bulk_wait_read_1();
                    named_barrier(1, 128);
                    if (issuer) {
                        tma_store_3d(&my, obuf, key0 + c * 32, p0 - g.y_row0, n * C);
                        bulk_commit();
                    }
                    if (++ob == CM_OUT_BUFS) ob = 0;
                }
            }
        }
        if (issuer) bulk_wait_all();
    }
#undef CM_FOR_UNITS
    fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 512);
}

size_t cm_smem_limit(int taps) { return 227 * 1024 - 64 * (size_t)taps * 4 - 384; }       // what the static arrays leave

struct CmPlan {
    int nstage, ntile, stage_bytes, lines;
    size_t smem;
};
CmPlan cm_plan(int C, int CQ, int CK) {
    CmPlan p{};
    p.lines = C * (128 / C + CQ - 1);
    p.stage_bytes = (p.lines * CM_PITCH + 127) & ~127;
    for (p.nstage = CM_MAX_STAGES; p.nstage >= 2; --p.nstage)
        for (p.ntile = 2; p.ntile >= 1; --p.ntile) {
            p.smem = 1024 + (size_t)p.ntile * CM_TILE_BYTES + CM_OUT_BUFS * CM_OUT_BYTES + (size_t)p.nstage * p.stage_bytes;
            if (p.smem <= cm_smem_limit(CQ * CK)) return p;
        }
    p.smem = 0;
    return p;
}

template <typename T, int CQ, int CK, int RI>
int launch_cm(const void* x, PlaneView xv, const void* w, const void* Wm, void* y, PlaneView yv, int N, int C, int Q, int row_begin, int row_end,
              cudaStream_t st) {
    CmGeom g{};
    const CmPlan p = cm_plan(C, CQ, CK);
    g.N = N; g.C = C; g.R = 128 / C; g.Q = Q;
    while ((1 << g.r_log) < g.R) ++g.r_log;
    g.row_begin = row_begin; g.row_end = row_end;
    g.x_row0 = xv.row0; g.y_row0 = yv.row0;
    g.groups = (row_end - row_begin + g.R - 1) / g.R;
    g.nstage = p.nstage; g.ntile = p.ntile; g.stage_bytes = p.stage_bytes; g.lines = p.lines;
    CUtensorMap mx, my;
    int rc;
    if ((rc = make_tensor_map_3d_mode(&mx, x, (uint64_t)N * C, (uint64_t)(row_end - xv.row0), (uint64_t)Q, (uint64_t)xv.width, (uint64_t)xv.plane_stride,
                                      CM_COLS, (uint32_t)(g.R + CQ - 1), 0, (uint32_t)C)))
        return rc;
    if ((rc = make_tensor_map_3d_mode(&my, y, (uint64_t)N * C, (uint64_t)(row_end - yv.row0), (uint64_t)Q, (uint64_t)yv.width, (uint64_t)yv.plane_stride, 32,
                                      (uint32_t)g.R, 64, (uint32_t)C)))
        return rc;
    int* flag = nullptr;
    if ((rc = wait_flag_ptr(&flag))) return rc;
    int sms = 0;
    if ((rc = sm_count(&sms))) return rc;
    // Whole rows where they make a unit a CTA or more, else four units a CTA, as long as the keys allow (B1 H8 S2048 45 -> 33 us; but a
    // short unit costs its start: B1 H16 S2048, 256 whole units, 45 -> 53 us).
    g.seg = (Q + CM_KEYS - 1) / CM_KEYS;
    if ((long)N * g.groups < sms) {
        long tiles = 0;
        for (int i = 0; i < g.groups; ++i) tiles += (std::min(row_begin + (i + 1) * g.R, std::min(row_end, Q)) + CM_KEYS - 1) / CM_KEYS;
        g.seg = (int)std::max<long>(1, (tiles * N + 4l * sms - 1) / (4l * sms));
    }
    for (int i = 0; cm_reach(g, i) > 0; ++i) g.units += (long)N * cm_reach(g, i);
    return launch_kernel<conv_mix_tc05_kernel<T, CQ, CK, RI>>("conv_mix_tc05_kernel", (unsigned)std::min<long>(g.units, sms), CM_THREADS, p.smem, st, mx, my,
                                                              static_cast<const T*>(w), static_cast<const T*>(Wm), g, flag);
}

}  // namespace

bool conv_mix_supported(const void* x, PlaneView xv, const void* y, PlaneView yv, int C, int CQ, int CK, int causal, int dtype, int w_dtype) {
    return causal && dtype != MTA_F32 && w_dtype == dtype && (C == 8 || C == 16 || C == 32 || C == 64) && (CQ == 2 || CQ == 3) && CK == 3 &&
           cm_plan(C, CQ, CK).smem > 0 && x != y && aligned16(x) && aligned16(y) && xv.width % 8 == 0 && xv.plane_stride % 8 == 0 && yv.width % 8 == 0 &&
           yv.plane_stride % 8 == 0;
}

int conv_mix_launch(const void* x, PlaneView xv, const void* w, const void* Wm, void* y, PlaneView yv, int N, int C, int Q, int CQ, int CK, int row_begin,
                    int row_end, int dtype, cudaStream_t st) {
    if (N == 0 || row_end <= row_begin || Q == 0) return MTA_OK;
#define MTA_CM_RI(T, CQV, CKV)                                                                                                       \
    do {                                                                                                                             \
        if (C <= 16) return launch_cm<T, CQV, CKV, 8>(x, xv, w, Wm, y, yv, N, C, Q, row_begin, row_end, st);                         \
        if (C == 32) return launch_cm<T, CQV, CKV, 4>(x, xv, w, Wm, y, yv, N, C, Q, row_begin, row_end, st);                         \
        return launch_cm<T, CQV, CKV, 2>(x, xv, w, Wm, y, yv, N, C, Q, row_begin, row_end, st);                                      \
    } while (0)
#define MTA_CM(T)                                                                                                                    \
    do {                                                                                                                             \
        if (CQ == 2) MTA_CM_RI(T, 2, 3);                                                                                             \
        MTA_CM_RI(T, 3, 3);                                                                                                          \
    } while (0)
    if (dtype == MTA_BF16) MTA_CM(__nv_bfloat16);
    MTA_CM(__half);
#undef MTA_CM
#undef MTA_CM_RI
}

}  // namespace mta
