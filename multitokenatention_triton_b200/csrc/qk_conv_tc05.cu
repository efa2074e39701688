// Scaled scores Q K^T and the first causal depthwise conv in one kernel: the score tile a conv tile needs is computed
// into tensor memory, rounded there and read there by the conv's MMAs, so the score planes are never written to or read from
// HBM (mta_attention_triton.py:68-73 as one pass).
//
// Per output tile (4 (33 - R) query rows x 112 keys) of the conv:
//   scores             four groups of 32 rows, R - 1 of each shared with the next group, keys n0-8 .. n0+119:
//                      S = Q[rows] . K[keys]^T, 8 (D = 128) tcgen05.mma of M128 N128 K16 into score buffer n % 2
//   drain (8 warps)    S -> round(round(S) * scale) as the reference's 16-bit matmul and multiply do -> 0 where key > query ->
//                      back into the buffer.  Rows and keys outside the plane come out 0 because TMA
//                      zero-fills Q / K there: that is the conv's zero padding.
//   conv               the MMAs of toeplitz_ts.cuh, A from the score buffer, into accumulator n % 2
//   epilogue (4 warps) TMEM -> 16-bit -> staging tiles -> TMA stores
// Warps: 0 TMA producer (K tile per tile, Q tile per row of tiles), 1 and 2 MMAs (of the even and the odd tiles), 4-11 drain (64 columns
// each), 12-15 epilogue.  TMEM: score buffers at columns 0 and 128, conv accumulators at 256 and 368.
// Bound: the tensor pipe (per tile 512 cycles of score MMAs, 120 per row tap of conv MMAs: 1232 of the 1850 that a tile takes for 6 x 11)
// and the hand-overs from MMA to drain to MMA.  Before, with the conv's operand in shared memory (a tile of 123 x 128 took 4700 cycles,
// 3000 of them the conv MMAs' operand reads): B8 H16 S4096 6x11 1.27 -> 0.80 ms, B1 H16 S2048 7x7 72 -> 51 us, B2 H16 S1021 44 -> 29 us.
// 16-bit dtypes, D in {64, 128}, odd key extent <= 17, causal.
#include "toeplitz_ts.cuh"

namespace mta {
namespace {
using namespace tc05;
using namespace qc;

// K of the planes that are worked on at a time stays in L2 (B8 H16 S4096: with one group 148 planes were in work, 155 MB of K; the kernel
// 0.93 ms, 0.84 with groups).
constexpr long GROUP_BYTES = 32 << 20;
constexpr int DRAIN_WARPS = 8;
constexpr int THREADS = 512;
constexpr uint32_t C_COL = 2 * SN;                // TMEM column of the first conv accumulator
// What the MMAs of a tile depend on besides its operands; the producer writes it next to the K tile, which spares the issuing warps
// the walk over the tiles.
enum : int { ODD_TILE = 1, SECOND_SET = 2 };

struct QcGeom : TileGeom {
    int S, R, KS, split_w, y_row0;
    float scale;
};

template <typename T, int D>
__global__ void __launch_bounds__(THREADS, 1)
qk_conv_tc05_kernel(const __grid_constant__ CUtensorMap mq, const __grid_constant__ CUtensorMap mk,
                    const __grid_constant__ CUtensorMap my, const void* __restrict__ w, int w_dtype, QcGeom g, int* err_flag) {
    constexpr int DBOX = D / 64;                               // 64-element boxes along the head dimension
    constexpr int QK_BYTES = DBOX * BOX_BYTES;                 // a Q or K tile: 128 rows x D
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ __align__(8) uint64_t full_bar[2], free_bar[2], s_full[2], ready_bar[2], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int ctl[2];                // a control word per chain
    __shared__ int abort_flag;
    __shared__ float wsm[TAP_FLOATS];               // the current head's conv weights on their way into the Toeplitz slices
    const int R = g.R, KS = g.KS;
    const int tb_bytes = toeplitz_bytes(R, g.split_w), stage = out_bytes(R);
    uint8_t* q_base = smem;
    uint8_t* k_base = q_base + 2 * QK_BYTES;
    uint8_t* tb_base = k_base + 2 * QK_BYTES;                   // two sets of Toeplitz slices: successive heads alternate
    uint8_t* out_base = tb_base + 2 * tb_bytes;                // two staging tiles
    const int tid = threadIdx.x, lane = tid & 31, warp = warp_index();
    const int pad_w = (KS - 1) / 2;
    const int a_off = 8 - pad_w;
    const int lead = R - 1, gr = group_rows(R);

    TileIter it;
    const int my_tiles = uniform(it.total(g));

    if (gave_up_before(err_flag, &abort_flag) || my_tiles == 0) return;

    if (warp == 0) {
        if (lane == 0) {
            for (int i = 0; i < 2; ++i) {
                mbar_init(&full_bar[i], 1);
                mbar_init(&free_bar[i], 1);
                mbar_init(&s_full[i], 1);
                mbar_init(&ready_bar[i], DRAIN_WARPS);
                mbar_init(&acc_full[i], 1);
                mbar_init(&acc_empty[i], 4);
            }
            fence_mbar_init();
            prefetch_tensormap(&mq);
            prefetch_tensormap(&mk);
            prefetch_tensormap(&my);
        }
        __syncwarp();
        tmem_alloc(&tmem_slot, 512);
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = 0;                       // the allocation is all of tensor memory
    pdl_wait();

    if (warp == 0) {
        // ---------------- producer: K tile per tile, Q tile per row of tiles, for each of the two chains ----------------
        if (lane == 0) {
            it.init(g);
            int head = it.head, set = 0, row = 0, in0 = -1, in1 = -1;        // row of tiles, and the one whose Q tile each chain has
            for (int n = 0; n < my_tiles; ++n) {
                const int b = n & 1;
                mbar_wait_spin(&free_bar[b], ((n >> 1) & 1) ^ 1, err_flag);      // the score MMAs of tile n - 2 have read the K tile
                if (it.head != head) { head = it.head; set ^= SECOND_SET; }
                ctl[b] = (it.tn & ODD_TILE) | set;
                const bool new_q = (b ? in1 : in0) != row;
                mbar_expect_tx(&full_bar[b], (uint32_t)((new_q ? 2 : 1) * QK_BYTES));
#pragma unroll
                for (int j = 0; j < DBOX; ++j)
                    tma_load_3d(k_base + b * QK_BYTES + j * BOX_BYTES, &mk, &full_bar[b], 64 * j, it.n0() - 8, it.plane);
                if (new_q) {
#pragma unroll
                    for (int j = 0; j < DBOX; ++j)
#pragma unroll 1
                        for (int gq = 0; gq < 4; ++gq)
                            tma_load_3d(q_base + b * QK_BYTES + j * BOX_BYTES + gq * QBOX_BYTES, &mq, &full_bar[b], 64 * j, it.m0(g) - lead + gq * gr,
                                        it.plane);
                    if (b) in1 = row;
                    else in0 = row;
                }
                if (it.next(g)) ++row;
            }
        }
    } else if (warp <= 2) {
        // ---------------- MMAs: two chains of score -> drain -> conv, one for the even tiles, one for the odd ones ----------------
        // Each chain has its Q and K tile, its score buffer and its accumulator, and a warp that issues its MMAs, so while one chain waits
        // for its drain (or its warp for an instruction) the other has the tensor pipe.  One warp for all MMAs left the pipe idle
        // for half of the time, and a warp for the scores and one for the convs hold each other up MMA by MMA.
        // The scores of tile n + 2 overwrite the A operand of the conv of tile n: MMAs of one thread execute in the order of issue. (PTX
        // promises that for MMAs of one shape on one accumulator.  Across shapes and accumulators, as here and between the row taps, whose shift each MMA
        // leaves in A for the next, it is what the hardware was seen to do: results are the same bits in every run.)
        constexpr uint32_t idesc = instr_desc_f16(AbFmtQ<T>::value, 0, 0, TM, SN);
        const uint32_t el = elect_one();
        const int b = warp - 1;
        const uint32_t t_s = tmem + (uint32_t)(b * SN), t_c = tmem + C_COL + (uint32_t)(b * TN), tb_addr = smem_u32(tb_base);
        const uint64_t q0 = smem_desc_sw128(smem_u32(q_base + b * QK_BYTES), 16, 1024), k0 = smem_desc_sw128(smem_u32(k_base + b * QK_BYTES), 16, 1024);
        uint32_t phase = 0;
        for (int n = b; n < my_tiles; n += 2, phase ^= 1) {
            mbar_wait_spin(&full_bar[b], phase, err_flag);
            const int c = uniform(ctl[b]);
            __syncwarp();
            fence_after_sync();
#pragma unroll
            for (int kk = 0; kk < D / 16; ++kk) {
                const uint64_t off = (uint64_t)(((kk / 4) * BOX_BYTES + (kk % 4) * 32) >> 4);
                mma_f16_ss(t_s, q0 + off, k0 + off, idesc, kk > 0 ? 1u : 0u, el);
            }
            mma_commit(&s_full[b], el);
            mma_commit(&free_bar[b], el);
            mbar_wait_spin(&acc_empty[b], phase ^ 1, err_flag);
            mbar_wait_spin(&ready_bar[b], phase, err_flag);
            __syncwarp();
            fence_after_sync();
            issue_conv<T>(t_s, tb_addr + (uint32_t)((c & SECOND_SET) ? tb_bytes : 0), t_c, c & ODD_TILE, R, g.split_w, el);
            mma_commit(&acc_full[b], el);
        }
    } else if (warp >= 4 && warp < 12) {
        // ---------------- drain: fp32 scores -> rounded, scaled, masked, in place; Toeplitz slices ----------------
        const int quarter = warp & 3;
        const int row = quarter * gr + lane - lead;          // staged row of this thread's lane, relative to the tile's first output row
        const int half = warp >= 8 ? 1 : 0;                  // of the staged columns
        const int ft = tid - 128;                            // 0..127 in the warps that build the slices
        const uint32_t sc = pack2<T>(g.scale, g.scale);
        if (half == 0) clear_taps(wsm, ft, 2);
        it.init(g);
        int cur_head = -1, hn = -1;
        for (int n = 0; n < my_tiles; ++n, it.next(g)) {
            const int b = n & 1;
            const int m0 = it.m0(g), kbase = it.n0() - 8 + 64 * half;
            const int head = it.head;
            if (half == 0 && head != cur_head) {
                cur_head = head;
                ++hn;
                // this set of slices was read last by the conv MMAs of the head before the previous one: tiles <= n - 2
                // (that of tile n - 3 is over: the scores of tile n - 1, seen above, followed it)
                if (n >= 2) mbar_wait_spin(&acc_full[b], ((n - 2) >> 1) & 1, err_flag);
                float taps[TAPS_PER_THREAD];
                fetch_taps(taps, w, w_dtype, head, R, KS, ft);
                build_from_taps<T>(tb_base + (hn & 1) * tb_bytes, wsm, taps, R, KS, a_off, g.split_w, ft, 2);
            }
            mbar_wait_spin(&s_full[b], (n >> 1) & 1, err_flag);
            __syncwarp();
            fence_after_sync();
            drain_half<T>(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(b * SN + 64 * half), sc, m0 + row - kbase + 1, kbase + 63 > m0 - lead);
            fence_before_sync();
            fence_proxy_async();          // the slices, written through the generic proxy, must be visible to the MMAs (async proxy)
            __syncwarp();
            if (lane == 0) mbar_arrive(&ready_bar[b]);
        }
    } else if (warp >= 12) {
        // ---------------- epilogue ----------------
        const int quarter = warp & 3;
        const bool issuer = warp == 12 && lane == 0 && flag_down(err_flag);
        const int row = quarter * gr + lane;                 // row of the tile
        const bool inside = lane < gr;
        it.init(g);
        for (int n = 0; n < my_tiles; ++n, it.next(g)) {
            const int b = n & 1;
            const int plane = it.plane, m0 = it.m0(g), n0 = it.n0();
            uint8_t* obuf = out_base + b * stage;
            uint8_t* orow = obuf + row * OUT_PITCH;
            if (issuer) bulk_wait_read_1();                  // the store of tile n - 2 has finished reading this staging tile
            mbar_wait_spin(&acc_full[b], (n >> 1) & 1, err_flag);
            named_barrier(1, 128);
            fence_after_sync();
            const uint32_t tacc = tmem + ((uint32_t)(quarter * 32) << 16) + C_COL + (uint32_t)(b * TN);
            const int live = m0 + row - n0 + 1;              // columns on or below the diagonal
            const bool diag = n0 + TN - 1 > m0;
            stage_row<T>(tacc, orow, live, diag, inside);
            fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[b]);
            fence_proxy_async();
            named_barrier(1, 128);
            if (issuer) {
                // the box has the tile's rows; rows past row_end and columns past S are clipped by the tensor map
                tma_store_3d(&my, obuf, n0, m0 - g.y_row0, plane);
                bulk_commit();
            }
        }
        if (issuer) bulk_wait_all();
    }
    fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 512);
}

constexpr size_t QC_SMEM_LIMIT = 225 * 1024;

size_t qk_conv_smem_bytes(int D, int R, bool split_w) {
    return 1024 + 2 * (size_t)out_bytes(R) + 4 * (size_t)(D / 64) * BOX_BYTES + 2 * (size_t)toeplitz_bytes(R, split_w ? 1 : 0);
}

template <typename T, int D>
int launch_qc(const void* q, const void* k, const void* w, int w_dtype, void* y, PlaneView yv, int B, int H, int S, int R, int KS,
              float scale, int row_begin, int row_end, cudaStream_t st) {
    const long planes = (long)B * H;
    QcGeom g{};
    set_tiles(g, planes, H, S, R, 1, row_begin, row_end);
    set_groups(g, (planes * S * D * 2 + GROUP_BYTES - 1) / GROUP_BYTES);
    g.S = S; g.R = R; g.KS = KS; g.scale = scale;
    g.split_w = w_dtype == MTA_F32 ? 1 : 0;
    g.y_row0 = yv.row0;
    CUtensorMap mq, mk, my;
    int rc;
    if ((rc = make_tensor_map_3d(&mq, q, (uint64_t)planes, S, D, D, (uint64_t)S * D, 64, 32, true))) return rc;
    if ((rc = make_tensor_map_3d(&mk, k, (uint64_t)planes, S, D, D, (uint64_t)S * D, 64, SN, true))) return rc;
    if ((rc = make_tensor_map_3d(&my, y, (uint64_t)planes, (uint64_t)(row_end - yv.row0), S, (uint64_t)yv.width,
                                 (uint64_t)yv.plane_stride, TN, (uint32_t)g.tmo, false)))
        return rc;
    int* flag = nullptr;
    if ((rc = wait_flag_ptr(&flag))) return rc;
    int sms = 0;
    if (int bad = sm_count(&sms)) return bad;
    MTA_REQUIRE(tiles_countable(g, sms), "qk_conv: planes of %d x %d are too large", row_end - row_begin, S);
    const unsigned grid = (unsigned)std::min<long>((long)g.tiles_per_plane * planes, sms);
    return launch_kernel<qk_conv_tc05_kernel<T, D>>("qk_conv_tc05_kernel", grid, THREADS, qk_conv_smem_bytes(D, R, g.split_w != 0), st, mq, mk, my, w,
                                                    w_dtype, g, flag);
}

}  // namespace

bool qk_conv_supported(const void* q, const void* k, const void* y, PlaneView yv, int S, int D, int R, int KS, int causal, int dtype,
                       int w_dtype) {
    return causal && dtype != MTA_F32 && (D == 64 || D == 128) && KS % 2 == 1 && KS <= 17 && R >= 1 && R <= 16 &&
           qk_conv_smem_bytes(D, R, w_dtype == MTA_F32) <= QC_SMEM_LIMIT && yv.width >= S && yv.width % 8 == 0 && yv.plane_stride % 8 == 0 && aligned16(q) &&
           aligned16(k) && aligned16(y);
}

int qk_conv_launch(const void* q, const void* k, const void* w, int w_dtype, void* y, PlaneView yv, int B, int H, int S, int D,
                   int R, int KS, float scale, int row_begin, int row_end, int dtype, cudaStream_t st) {
    if ((long)B * H == 0 || row_end <= row_begin) return MTA_OK;
#define MTA_QC(TT, DD) return launch_qc<TT, DD>(q, k, w, w_dtype, y, yv, B, H, S, R, KS, scale, row_begin, row_end, st)
    if (dtype == MTA_BF16) { if (D == 64) MTA_QC(__nv_bfloat16, 64); MTA_QC(__nv_bfloat16, 128); }
    if (D == 64) MTA_QC(__half, 64);
    MTA_QC(__half, 128);
#undef MTA_QC
}

}  // namespace mta
