// Depthwise causal conv over score planes on the tcgen05 tensor cores, 16-bit dtypes, key extent S <= 17, up to 16 row taps.
//
// Toeplitz formulation: for a fixed row tap i the key-direction taps form a banded matrix,
//   out[q, k] += sum_kk X[q + i - (R-1), kk] * T_i[kk, k],   T_i[kk, k] = w[i, kk - k + pad_w]  (0 outside the band)
// so every row tap and every 16 staged columns are one MMA of the staged tile, rows shifted by i, against a 16 x 32 slice of T_i.  The
// staged tile is the MMA's A operand in tensor memory, where the shift costs nothing (toeplitz_ts.cuh).
//
// Persistent, warp-specialised kernel; per output tile (4 (33 - R) rows x 112 keys; only tiles that touch keys <= query when causal):
//   warp 0      TMA producer: two boxes of 64 columns (128-byte swizzle) of the tile's 4 (33 - R) + R - 1 rows, a ring of tiles
//               (out-of-range rows / columns arrive as zero = the conv's zero padding)
//   warps 4-11  shared memory -> registers -> tensor memory, one row and 64 columns a thread (the four groups of 32 rows share R - 1
//               rows with the next, which are read twice here and not loaded twice), keys above the causal diagonal replaced by zeros
//               on the way; the Toeplitz slices when the head changes
//   warps 1, 2  the MMAs of the even and of the odd tiles, each with an accumulator and two A buffers
//   warps 12-15 epilogue: accumulator -> 16-bit -> staging tiles -> TMA stores
//   warp 3      stores zero tiles above the diagonal when the whole output is wanted
// Against the form with the staged tile as an operand in shared memory (tiles of 128 x 128), the zeros above the diagonal written, us, that form / this:
//   S1024 B2: 3x3 23 / 22, 6x11 28 / 21, 11x15 38 / 25;  B4 S1024: 3x3 49 / 49, 6x11 47 / 45, 11x15 61 / 47;  B1 S3000: 3x3 110 / 104, 6x11 112 / 101;
//   B4 S2048: 1x1 163 / 172, 3x3 173 / 178, 6x11 174 / 173, 7x9 168 / 171, 11x15 208 / 166;  B1 S4096: 3x3 172 / 174, 6x11 171 / 173, 7x9 168 / 177
// (H16).  So it is up to 5 % behind where rows are 4 or 8 KB, a power of two, and taps are few, level or ahead everywhere else: not worth a second kernel.
// Bound: 120 cycles of MMAs a row tap and tile for large kernels, HBM for small ones.  With the staged tile as an operand in shared
// memory an MMA took 40 cycles instead of 16.  6 x 11, lower triangles only: B4 H16 S1024 41 -> 31 us; 7 x 7 B1 H16 S2048 fp16 42 -> 30;
// with the zeros above the diagonal written (B4 H16 S2048, 805 MB) 171 us before and after: HBM, three quarters of it writes.
#include <algorithm>

#include "toeplitz_ts.cuh"

namespace mta {

namespace {
using namespace tc05;
using namespace qc;

constexpr int STAGE_BYTES = 2 * BOX_BYTES;        // a tile: two boxes of 64 columns x up to 128 rows
// Rows of input that a tile's output rows reach.
__host__ __device__ constexpr int staged_rows(int R) { return 4 * (33 - R) + R - 1; }
constexpr int MAX_STAGES = 4;
constexpr int ABUFS = 4;                          // A operands in tensor memory; buffer b in columns 128 (b / 2) + 32 (b % 2) .. + 31 and 64 more on
constexpr uint32_t C_COL = 256;                   // accumulators
constexpr int ZERO_COLS = 64;                     // columns of a zero tile
constexpr int THREADS = 512;

struct ConvGeom : TileGeom {
    int W, R, S, x_row0, y_row0, write_upper, split_w;
    int nstage;
    int early_weights; // see pdl_wait()
    int lead;          // staged rows start `lead` rows before the tile: R-1 for the conv (row taps look back), 0 for its
                       // input gradient (taps reversed, looking forward)
    int flip;          // input gradient: tap (i, j) uses w[R-1-i][S-1-j]
    long zero_per_plane, zero_total;     // tiles wholly above the diagonal that must be written as zero (write_upper)
};

// Zero tiles to the right of row of tiles tm.  The first begins where the compute tiles end, the others at multiples of ZERO_COLS, so that they
// store whole lines; what the first two have in common is stored twice.
__host__ __device__ __forceinline__ int zero_tiles(const ConvGeom& g, int tm) {
    const int c0 = key_tiles(g, tm) * TN;
    return c0 < g.W ? (g.W + ZERO_COLS - 1) / ZERO_COLS - c0 / ZERO_COLS : 0;
}

__device__ __forceinline__ int zero_tile_col(const ConvGeom& g, int tm, int tn) {
    const int c0 = key_tiles(g, tm) * TN;
    return tn == 0 ? c0 : (c0 / ZERO_COLS + tn) * ZERO_COLS;
}

template <typename T>
__global__ void __launch_bounds__(THREADS, 1)
conv2d_tc05_kernel(const __grid_constant__ CUtensorMap mx, const __grid_constant__ CUtensorMap my, const __grid_constant__ CUtensorMap mz,
                   const void* __restrict__ w, int w_dtype, ConvGeom g, int* err_flag) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ __align__(8) uint64_t full_bar[MAX_STAGES], empty_bar[MAX_STAGES], ready_bar[ABUFS], a_empty[ABUFS], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int ctl[ABUFS];        // bit 0: an odd key tile, bit 1: the second set of slices
    __shared__ int abort_flag;
    __shared__ float wsm[TAP_FLOATS];          // the current head's weights on their way into the Toeplitz slices
    __shared__ int tiles_loaded;               // compute tiles whose loads the producer has issued (paces the zero tiles)
    const int R = g.R, S = g.S;
    const int tb_bytes = toeplitz_bytes(R, g.split_w), stage = out_bytes(R);
    uint8_t* stage_base = smem;
    uint8_t* tb_base = stage_base + g.nstage * STAGE_BYTES;        // two sets of Toeplitz slices: successive heads alternate
    uint8_t* out_base = tb_base + 2 * tb_bytes;                    // two staging tiles
    uint8_t* zero_box = out_base + 2 * stage;                      // zeros, with write_upper
    const int tid = threadIdx.x, lane = tid & 31, warp = warp_index();
    const int a_off = 8 - (S - 1) / 2;
    const int gr = group_rows(R);

    TileIter it;
    const int my_tiles = uniform(it.total(g));

    if (tid == 0) tiles_loaded = 0;
    if (gave_up_before(err_flag, &abort_flag) || my_tiles == 0) return;

    if (warp == 0) {
        if (lane == 0) {
            for (int i = 0; i < MAX_STAGES; ++i) {
                mbar_init(&full_bar[i], 1);
                mbar_init(&empty_bar[i], 8);
            }
            for (int i = 0; i < ABUFS; ++i) {
                mbar_init(&ready_bar[i], 8);
                mbar_init(&a_empty[i], 1);
            }
            for (int i = 0; i < 2; ++i) {
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
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = 0;                       // the allocation is all of tensor memory
    // the copying warps and the MMA warps touch no other kernel's memory but the weights
    if (!g.early_weights || !(warp == 1 || warp == 2 || (warp >= 4 && warp < 12))) pdl_wait();

    if (warp == 0) {
        // ---------------- producer ----------------
        if (lane == 0) {
            it.init(g);
            int st = 0, use = 0;
            for (int n = 0; n < my_tiles; ++n, it.next(g)) {
                mbar_wait_spin(&empty_bar[st], (use & 1) ^ 1, err_flag);
                uint8_t* xa = stage_base + st * STAGE_BYTES;
                mbar_expect_tx(&full_bar[st], (uint32_t)(2 * staged_rows(R) * 128));
#pragma unroll
                for (int j = 0; j < 2; ++j)
                    tma_load_3d(xa + j * BOX_BYTES, &mx, &full_bar[st], it.n0() - 8 + 64 * j, it.m0(g) - g.lead - g.x_row0, it.plane);
                *reinterpret_cast<volatile int*>(&tiles_loaded) = n + 1;
                if (++st == g.nstage) { st = 0; ++use; }
            }
        }
    } else if (warp == 3) {
        // ---------------- zero tiles ----------------
        // The tiles wholly above the diagonal are part of the output the API returns: this warp writes its share of
        // them as TMA stores of a zero box, in step with the producer's progress through the compute tiles, so the two
        // kinds of traffic overlap for the whole run instead of the zero stores flooding the memory system first.
        const long zper = (g.zero_total + gridDim.x - 1) / gridDim.x;
        const long z_begin = min((long)blockIdx.x * zper, g.zero_total), z_end = min(z_begin + zper, g.zero_total);
        const int my_zero = (int)(z_end - z_begin);
        if (my_zero > 0) {
            for (int i = lane; i < g.tmo * ZERO_COLS / 8; i += 32) reinterpret_cast<uint4*>(zero_box)[i] = make_uint4(0u, 0u, 0u, 0u);
            fence_proxy_async();
        }
        __syncwarp();
        if (lane == 0 && my_zero > 0 && flag_down(err_flag)) {
            // walker over (plane, row of tiles, zero tile)
            int zp = (int)(z_begin / g.zero_per_plane), ztm = 0, ztn = (int)(z_begin - (long)zp * g.zero_per_plane), nz;
            while (ztn >= (nz = zero_tiles(g, ztm))) { ztn -= nz; ++ztm; }
            for (int zi = 0; zi < my_zero; ++zi) {
                // zero tile zi is due once the producer has loaded compute tile zi * my_tiles / my_zero (bounded wait:
                // the producer always reaches its last tile, and giving up early only changes the pacing)
                const int due = (int)((long)zi * my_tiles / my_zero);
                for (int spin = 0; *reinterpret_cast<volatile int*>(&tiles_loaded) < due && spin < (1 << 20); ++spin) __nanosleep(256);
                tma_store_3d(&mz, zero_box, zero_tile_col(g, ztm, ztn), g.row_begin + ztm * g.tmo - g.y_row0, zp);
                bulk_commit();
                bulk_wait_read_1();
                if (++ztn == nz && zi + 1 < my_zero) {
                    ztn = 0;
                    do {
                        if (++ztm == g.tiles_m) { ztm = 0; ++zp; }
                    } while ((nz = zero_tiles(g, ztm)) == 0);
                }
            }
            bulk_wait_all();
        }
    } else if (warp <= 2) {
        // ---------------- MMAs of the even (warp 1) and the odd tiles ----------------
        const uint32_t el = elect_one();
        const int b = warp - 1;
        const uint32_t t_c = tmem + C_COL + (uint32_t)(b * TN), tb_addr = smem_u32(tb_base);
        for (int n = b; n < my_tiles; n += 2) {
            const int ab = n & (ABUFS - 1);
            mbar_wait_spin(&acc_empty[b], ((n >> 1) & 1) ^ 1, err_flag);
            mbar_wait_spin(&ready_bar[ab], (n / ABUFS) & 1, err_flag);
            const int c = uniform(ctl[ab]);
            __syncwarp();
            fence_after_sync();
            issue_conv<T>(tmem + (uint32_t)((ab >> 1) * 128 + (ab & 1) * 32), tb_addr + (uint32_t)((c & 2) ? tb_bytes : 0), t_c, c & 1, R, g.split_w, el);
            mma_commit(&a_empty[ab], el);
            mma_commit(&acc_full[b], el);
        }
    } else if (warp < 12) {
        // ---------------- staged tile -> tensor memory; Toeplitz slices ----------------
        const int quarter = warp & 3, half = warp >= 8 ? 1 : 0;
        const int sr = quarter * gr + lane;                  // staged row that becomes TMEM lane 32 quarter + lane
        const int row = quarter * gr + lane - g.lead;        // its row relative to the tile's first output row
        const int ft = tid - 128;                            // 0..127 in the warps that build the slices
        if (half == 0) clear_taps(wsm, ft, 2);
        it.init(g);
        int cur_head = -1, set = 2, st = 0, use = 0;
        for (int n = 0; n < my_tiles; ++n, it.next(g)) {
            const int ab = n & (ABUFS - 1);
            const int m0 = it.m0(g), kbase = it.n0() - 8 + 64 * half;
            if (it.head != cur_head) {
                cur_head = it.head;
                set ^= 2;
                if (half == 0) {
                    // this set of slices was read last by the conv MMAs of the head before the previous one: tiles <= n - 2, of both warps
                    for (int p = n - 3; p < n - 1; ++p)
                        if (p >= 0) mbar_wait_spin(&a_empty[p & (ABUFS - 1)], (p / ABUFS) & 1, err_flag);
                    float taps[TAPS_PER_THREAD];
                    fetch_taps(taps, w, w_dtype, it.head, R, S, ft, g.flip != 0);
                    build_from_taps<T>(tb_base + (set ? tb_bytes : 0), wsm, taps, R, S, a_off, g.split_w, ft, 2);
                }
            }
            mbar_wait_spin(&full_bar[st], use & 1, err_flag);
            // row sr of the box: eight 16-byte pieces, piece c at position c xor sr % 8
            const uint8_t* src = stage_base + st * STAGE_BYTES + half * BOX_BYTES + sr * 128;
            uint32_t pk[32];
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const uint4 v = *reinterpret_cast<const uint4*>(src + ((c ^ (sr & 7)) << 4));
                pk[4 * c] = v.x; pk[4 * c + 1] = v.y; pk[4 * c + 2] = v.z; pk[4 * c + 3] = v.w;
            }
            if (g.causal && kbase + 63 > m0 - g.lead) {      // some staged key above some staged row
                const int live = m0 + row - kbase + 1;
#pragma unroll
                for (int i = 0; i < 32; ++i) pk[i] &= (2 * i < live ? 0x0000ffffu : 0u) | (2 * i + 1 < live ? 0xffff0000u : 0u);
            }
            mbar_wait_spin(&a_empty[ab], ((n / ABUFS) & 1) ^ 1, err_flag);       // the MMAs of tile n - ABUFS have read the buffer
            __syncwarp();
            fence_after_sync();
            tmem_st_32x32(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)((ab >> 1) * 128 + (ab & 1) * 32 + half * 64), pk);
            if (tid == 128) ctl[ab] = (it.tn & 1) | set;
            tmem_st_wait();
            fence_before_sync();
            fence_proxy_async();          // the slices, written through the generic proxy, must be visible to the MMAs (async proxy)
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&empty_bar[st]);
                mbar_arrive(&ready_bar[ab]);
            }
            if (++st == g.nstage) { st = 0; ++use; }
        }
    } else {
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
            if (issuer) bulk_wait_read_1();                  // the store of tile n - 2 has finished reading this staging tile
            mbar_wait_spin(&acc_full[b], (n >> 1) & 1, err_flag);
            named_barrier(1, 128);
            fence_after_sync();
            stage_row<T>(tmem + ((uint32_t)(quarter * 32) << 16) + C_COL + (uint32_t)(b * TN), obuf + row * OUT_PITCH, m0 + row - n0 + 1,
                         g.causal && n0 + TN - 1 > m0, inside);
            fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[b]);
            fence_proxy_async();                             // staging tile written through the generic proxy, read by TMA
            named_barrier(1, 128);
            if (issuer) {
                // rows past row_end and columns past W are clipped by the tensor map
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

constexpr size_t CONV_SMEM_LIMIT = 222 * 1024;         // what the static arrays leave

size_t conv2d_tc05_smem_bytes(int R, bool split_w, bool zeros, int nstage) {
    return 1024 + (size_t)nstage * STAGE_BYTES + 2 * (size_t)toeplitz_bytes(R, split_w ? 1 : 0) + 2 * (size_t)out_bytes(R) +
           (zeros ? (size_t)tile_rows(R) * ZERO_COLS * 2 : 0);
}

// Of one group's tiles a CTA gets this many or more.  The fewer planes are in work at a time, the more of the rows that neighbouring tiles
// share come from L2, but a CTA changes its head with every group and then builds R slices.  Where the zeros above the diagonal are stored and the
// planes do not all fit into L2, HBM is the bound and small groups pay, up to 9 row taps.  Forward, us, with 2 / 8 / 16 tiles:
//   B4 H16 S2048: 3x3 175 / 181 / 184, 6x11 175 / 178 / 180, 7x9 174 / 183 / 186, 11x15 176 (input gradient 195) / 190 (185) / 189, 16x17 339 / 257 / 248
//   B4 H16 S1024: 3x3 49 / 50 / 50, 6x11 45 / 48 / 47, 11x15 59 / 51 / 47, 16x17 96 / 78 / 72;  B8 H16 S1024: 6x11 87 / 97 / 97
//   B1 H8 S2048 (67 MB of output): 3x3 22 / 20 / 20, 6x11 22 / 20 / 21, 16x17 50 / 35 / 34
// Without the zeros the head changes show at once: 158 against 153 us (forward B1 H16 S2048 with two 7x7 convs), 674 against 650 (training step
// B4 H16 S1024).
constexpr int GROUP_TILES = 8, GROUP_TILES_ZEROS = 2, GROUP_ZEROS_TAPS = 9;
constexpr long GROUP_ZEROS_BYTES = 80 << 20;       // of output: with the lower triangles of the input what L2 holds

int group_tiles(int R, bool zeros, long out_bytes) {
    return zeros && R <= GROUP_ZEROS_TAPS && out_bytes > GROUP_ZEROS_BYTES ? GROUP_TILES_ZEROS : std::max(GROUP_TILES, R);
}

template <typename T>
int launch_tc05(const void* x, PlaneView xv, long x_rows_stored, const void* w, int w_dtype, void* y, PlaneView yv,
                long planes, int C, int W, int R, int S, int causal, int row_begin, int row_end, bool write_upper,
                bool grad_input, bool early_weights, cudaStream_t st) {
    int rc, sms = 0;
    if ((rc = sm_count(&sms))) return rc;
    ConvGeom g{};
    set_tiles(g, planes, C, W, R, causal, row_begin, row_end);
    g.write_upper = causal && write_upper ? 1 : 0;
    set_groups(g, (long)g.tiles_per_plane * planes / ((long)group_tiles(R, g.write_upper != 0, planes * (row_end - row_begin) * W * (long)sizeof(T)) * sms));
    g.W = W; g.R = R; g.S = S; g.x_row0 = xv.row0; g.y_row0 = yv.row0;
    g.split_w = w_dtype == MTA_F32 ? 1 : 0;
    g.lead = grad_input ? 0 : R - 1;
    g.flip = grad_input ? 1 : 0;
    g.early_weights = early_weights ? 1 : 0;
    if (g.write_upper)
        for (int tm = 0; tm < g.tiles_m; ++tm) g.zero_per_plane += zero_tiles(g, tm);
    g.zero_total = g.zero_per_plane * planes;
    CUtensorMap mx, my, mz;
    if ((rc = make_tensor_map_3d(&mx, x, (uint64_t)planes, (uint64_t)x_rows_stored, (uint64_t)W, (uint64_t)xv.width,
                                 (uint64_t)xv.plane_stride, 64, (uint32_t)staged_rows(R), true)))
        return rc;
    // rows past row_end are outside these maps, so a tile's store never touches them
    if ((rc = make_tensor_map_3d(&my, y, (uint64_t)planes, (uint64_t)(row_end - yv.row0), (uint64_t)W, (uint64_t)yv.width,
                                 (uint64_t)yv.plane_stride, TN, (uint32_t)g.tmo, false)))
        return rc;
    mz = my;
    if (g.write_upper && (rc = make_tensor_map_3d(&mz, y, (uint64_t)planes, (uint64_t)(row_end - yv.row0), (uint64_t)W, (uint64_t)yv.width,
                                                  (uint64_t)yv.plane_stride, ZERO_COLS, (uint32_t)g.tmo, false)))
        return rc;
    int* flag = nullptr;
    if ((rc = wait_flag_ptr(&flag))) return rc;
    for (g.nstage = MAX_STAGES; g.nstage > 2 && conv2d_tc05_smem_bytes(R, g.split_w != 0, g.write_upper != 0, g.nstage) > CONV_SMEM_LIMIT; --g.nstage) {}
    const size_t smem = conv2d_tc05_smem_bytes(R, g.split_w != 0, g.write_upper != 0, g.nstage);
    MTA_REQUIRE(smem <= CONV_SMEM_LIMIT, "conv2d (tcgen05): kernel with %d row taps needs %zu bytes of shared memory", R, smem);
    MTA_REQUIRE(tiles_countable(g, sms), "conv2d (tcgen05): planes of %d x %d are too large", row_end - row_begin, W);
    const unsigned grid = (unsigned)std::min<long>((long)g.tiles_per_plane * planes, sms);
    return launch_kernel<conv2d_tc05_kernel<T>>("conv2d_tc05_kernel", grid, THREADS, smem, st, mx, my, mz, w, w_dtype, g, flag);
}

}  // namespace

bool conv2d_tc05_supported(const void* x, PlaneView xv, const void* y, PlaneView yv, int W, int R, int S, int dtype,
                           int w_dtype) {
    return dtype != MTA_F32 && S <= 17 && R <= 16 && conv2d_tc05_smem_bytes(R, w_dtype == MTA_F32, true, 2) <= CONV_SMEM_LIMIT && xv.width % 8 == 0 && yv.width % 8 == 0 &&
           xv.plane_stride % 8 == 0 && yv.plane_stride % 8 == 0 && aligned16(x) && aligned16(y);
}

int conv2d_tc05_launch(const void* x, PlaneView xv, long x_rows_stored, const void* w, int w_dtype, void* y, PlaneView yv,
                       long planes, int C, int H, int W, int R, int S, int causal, int row_begin, int row_end,
                       bool write_upper, int dtype, cudaStream_t st, bool grad_input, bool early_weights) {
    (void)H;
    MTA_REQUIRE(!grad_input || S % 2 == 1, "conv2d (tcgen05): the input gradient needs an odd key extent");
    if (dtype == MTA_BF16)
        return launch_tc05<__nv_bfloat16>(x, xv, x_rows_stored, w, w_dtype, y, yv, planes, C, W, R, S, causal, row_begin,
                                          row_end, write_upper, grad_input, early_weights, st);
    return launch_tc05<__half>(x, xv, x_rows_stored, w, w_dtype, y, yv, planes, C, W, R, S, causal, row_begin, row_end,
                               write_upper, grad_input, early_weights, st);
}

}  // namespace mta
