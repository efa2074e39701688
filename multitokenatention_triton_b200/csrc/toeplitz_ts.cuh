// Pieces shared by the kernels that run the conv as Toeplitz MMAs with its input in tensor memory (TMEM): conv2d_tc05.cu, and with the
// scores Q K^T computed on the spot qk_conv_tc05.cu and conv_attn_tc05.cu.  Tile geometry, the drain of the score
// + conv kernel (the conv attention, whose tiles are narrower, has its own), the conv MMA schedule and the Toeplitz slices.
//
// The score tile never leaves TMEM.  S[128 x 128] comes out of the score MMAs as fp32, the drain warps round it to 16 bits in place
// (64 columns of fp32 become 32 of the same columns), and the conv's MMAs read it there as their A operand.  A row tap is the A operand moved up by one
// lane, which the MMA of the tap before does on its way (mma_f16_ts_shift).  Lanes only move within their group of 32, so the four
// groups hold overlapping row blocks: lane 32 w + l holds staged row (33 - R) w + l (R row taps), and the first 33 - R lanes of a
// group carry output rows, 4 (33 - R) of the tile's 128 lanes (108 for 6 row taps, 88 for 11, 68 for 16).
//   With the staged tile in shared memory (128 + R - 1 rows, all 128 lanes of use for R = 1, 123 for R = 6) an MMA cost 40 cycles for
//   the 4 KB of A that every tap fetches again; from TMEM it costs 16, so 108 of 128 lanes are still 2.2 times the rate, and the
//   tile's trip through shared memory (36 KB written, 240 KB read) is gone.
// Staged columns: 8 (left halo) + 112 + 8 keys = the 128 columns of a score MMA; an output tile is 112 keys wide.
#pragma once

#include "kernels.cuh"
#include "tc05.cuh"

namespace mta {
namespace qc {
using namespace tc05;

constexpr int TM = 128;            // TMEM lanes = MMA M
constexpr int TN = 112;            // output columns per tile
constexpr int SN = 128;            // staged columns = N of the score MMA
constexpr int BOX_BYTES = TM * 128;               // 64 elements of 128 rows of Q, K or V: 128 bytes a row
constexpr int QBOX_BYTES = 32 * 128;              // the part of it that belongs to one group of lanes

// Output rows per group of lanes and per tile.
__host__ __device__ inline int group_rows(int R) { return 33 - R; }
__host__ __device__ inline int tile_rows(int R) { return 4 * (33 - R); }

template <typename T> struct AbFmtQ;
template <> struct AbFmtQ<__nv_bfloat16> { static constexpr int value = 1; };
template <> struct AbFmtQ<__half> { static constexpr int value = 0; };

// Two products in T, each rounded once (the exact product of two 16-bit values fits in fp32, so this is what fp32 and a
// conversion would give).
template <typename T> __device__ __forceinline__ uint32_t mul2q(uint32_t a, uint32_t b);
template <> __device__ __forceinline__ uint32_t mul2q<__nv_bfloat16>(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
template <> __device__ __forceinline__ uint32_t mul2q<__half>(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}

// Matrix descriptor without swizzle: lbo = bytes between the two 8-element k chunks of one MMA, sbo = bytes between
// groups of 8 rows.
__device__ __forceinline__ uint64_t desc_plain(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3ffffu) >> 4);
    d |= (uint64_t)((lbo_bytes >> 4) & 0x3fffu) << 16;
    d |= (uint64_t)((sbo_bytes >> 4) & 0x3fffu) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}

// Shared-memory bytes of one head's Toeplitz slices.
__host__ __device__ inline int toeplitz_bytes(int R, int split_w) { return (R * 1024 * (split_w ? 2 : 1) + 1023) & ~1023; }

// The conv MMAs of one row tap (or of the high or low part of its weights): A in a buffer of 16 NK columns at a0, k-step s = staged
// columns 16 s .. 16 s + 15, which reach the 16-column output blocks s - 1 and s of the accumulator at d0 (the first and the last
// k-step reach one block only: N = 16, half of the slice).  Every other k-step comes first: those touch each block once, so the first
// batch of a tile (ACC false) needs no cleared accumulator.  All from one thread, in this order, so the result does not depend on
// timing.  FIRST (0 or 1): the k-steps s with s % 2 = FIRST come first, 1 for even tiles and 0 for odd ones: a tile is seven blocks
// wide, and like this the k-steps of a block are added in the order in which conv2d_tc05.cu adds them, bit for bit the same sums.
// SHIFT: A is left one row up, for the next tap.
// An MMA takes 16 cycles on the tensor pipe and only so many instructions may come with it: with the accumulate flag or the order of
// the k-steps as run-time values it was 22 to 28 cycles an MMA.
template <typename T, int NK, int FIRST, bool SHIFT, bool ACC>
__device__ __forceinline__ void issue_tap(uint32_t a0, uint64_t db, uint32_t d0, uint32_t el) {
    constexpr uint32_t idesc32 = instr_desc_f16(AbFmtQ<T>::value, 0, 0, TM, 32);
    constexpr uint32_t idesc16 = instr_desc_f16(AbFmtQ<T>::value, 0, 0, TM, 16);
#pragma unroll
    for (int pass = 0; pass < 2; ++pass)
#pragma unroll
        for (int s = pass ^ FIRST; s < NK; s += 2) {
            const bool upper = s == 0, lower = s == NK - 1;
            const uint64_t b = db + (upper ? 16u : 0u);
            const uint32_t a = a0 + 8u * (uint32_t)s + (s >= NK / 2 ? 4u * NK : 0u);     // in the buffer's second half
            const uint32_t d = d0 + (upper ? 0u : 16u * (uint32_t)(s - 1)), idesc = (upper || lower) ? idesc16 : idesc32;
            if (SHIFT) mma_f16_ts_shift(d, a, b, idesc, (pass > 0 || ACC) ? 1u : 0u, el);
            else mma_f16_ts(d, a, b, idesc, (pass > 0 || ACC) ? 1u : 0u, el);
        }
}
template <typename T, int NK, int FIRST>
__device__ __forceinline__ void issue_taps(uint32_t a0, uint64_t db, uint32_t d0, int R, int split_w, uint32_t el) {
    // (the shift after the last tap is of no use to anybody and costs nothing)
    if (split_w) {                                                        // float32 weights: every tap in two parts
        const uint64_t low = (uint64_t)(R * 64);
        issue_tap<T, NK, FIRST, false, false>(a0, db, d0, el);
        issue_tap<T, NK, FIRST, true, true>(a0, db + low, d0, el);
#pragma unroll 1
        for (int i = 1; i < R; ++i) {
            db += 64;
            issue_tap<T, NK, FIRST, false, true>(a0, db, d0, el);
            issue_tap<T, NK, FIRST, true, true>(a0, db + low, d0, el);
        }
    } else {
        issue_tap<T, NK, FIRST, true, false>(a0, db, d0, el);
#pragma unroll 1
        for (int i = 1; i < R; ++i) {
            db += 64;
            issue_tap<T, NK, FIRST, true, true>(a0, db, d0, el);
        }
    }
}
// The conv MMAs of a tile; `odd`: of an odd key tile.
template <typename T>
__device__ __forceinline__ void issue_conv(uint32_t a0, uint32_t tb_addr, uint32_t d0, int odd, int R, int split_w, uint32_t el) {
    const uint64_t db = desc_plain(tb_addr, 512, 128);
    if (odd) issue_taps<T, SN / 16, 0>(a0, db, d0, R, split_w, el);
    else issue_taps<T, SN / 16, 1>(a0, db, d0, R, split_w, el);
}

// The Toeplitz slices of a head (row tap i, element (n', kk) = w[i][kk + 16 - n' - a_off]; with `split_w` a second set holding what
// the 16-bit rounding of a float32 weight lost) in the no-swizzle K-major layout the conv MMAs read: 8 rows x 16 bytes per core
// matrix, the two k chunks 512 bytes apart, row groups 128 bytes apart.  The weights pass through `wsm` (TAP_FLOATS floats of shared
// memory), tap row i at i * TAP_PITCH with zeros around its KS taps, so a thread writes 16 bytes at a time without a comparison.
constexpr int MAX_TAPS = 16 * 17;
constexpr int TAP_PITCH = 57, TAP_ZERO = 24, TAP_FLOATS = 16 * TAP_PITCH;     // taps -23 .. 31 of a row are looked at
constexpr int TAPS_PER_THREAD = (MAX_TAPS + 127) / 128;

// All by the 128 threads (whole warps, ft = 0 .. 127) that own hardware barrier `bar_id`.  clear_taps once, before the first build.
__device__ __forceinline__ void clear_taps(float* wsm, int ft, int bar_id) {
    for (int i = ft; i < TAP_FLOATS; i += 128) wsm[i] = 0.0f;
    named_barrier(bar_id, 128);
}
// A caller that knows its next head ahead of time fetches its weights (thread ft holds taps ft, ft + 128, ...) before it needs them,
// which hides the latency of global memory behind whatever it does next.  `flip`: taps in reverse order.
__device__ __forceinline__ void fetch_taps(float (&reg)[TAPS_PER_THREAD], const void* w, int w_dtype, int head, int R, int KS, int ft, bool flip = false) {
#pragma unroll
    for (int i = 0; i < TAPS_PER_THREAD; ++i) {
        const int idx = ft + 128 * i;
        reg[i] = idx < R * KS ? load_weight(w, (long)head * R * KS + (flip ? R * KS - 1 - idx : idx), w_dtype) : 0.0f;
    }
}
template <typename T>
__device__ __forceinline__ void build_from_taps(uint8_t* tb, float* wsm, const float (&reg)[TAPS_PER_THREAD], int R, int KS, int a_off,
                                                int split_w, int ft, int bar_id) {
#pragma unroll
    for (int i = 0; i < TAPS_PER_THREAD; ++i) {
        const int idx = ft + 128 * i;
        if (idx < R * KS) wsm[idx / KS * TAP_PITCH + TAP_ZERO + idx % KS] = reg[i];
    }
    named_barrier(bar_id, 128);
    for (int idx = ft; idx < R * 64; idx += 128) {
        const int i = idx >> 6, half = (idx >> 5) & 1, nn = idx & 31;
        const float* src = wsm + i * TAP_PITCH + TAP_ZERO + half * 8 + 16 - nn - a_off;
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float a = src[2 * e], b = src[2 * e + 1];
            hi[e] = pack2<T>(a, b);
            lo[e] = pack2<T>(a - round_to<T>(a), b - round_to<T>(b));
        }
        uint8_t* dst = tb + i * 1024 + half * 512 + (nn >> 3) * 128 + (nn & 7) * 16;
        *reinterpret_cast<uint4*>(dst) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        if (split_w) *reinterpret_cast<uint4*>(dst + R * 1024) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    }
    named_barrier(bar_id, 128);             // nobody refills wsm while another warp still reads it
}

// One thread's share of the score + conv kernel's drain: 64 of its lane's fp32 scores, at `tcol`, become 16-bit values, two per column, in the
// first 32 of the same columns: round(round(S) * scale), the reference's 16-bit matmul followed by its 16-bit multiply (`sc2`: the scale
// twice).  `live`: how many of the columns lie on or below the diagonal, the others become 0; `diag`
// (warp-uniform): some lane has fewer than 64.  Whole-warp call; the stores are complete when it returns.
template <typename T>
__device__ __forceinline__ void drain_half(uint32_t tcol, uint32_t sc2, int live, bool diag) {
    uint32_t r[64], pk[32];
    tmem_ld_32x32(tcol, *reinterpret_cast<uint32_t(*)[32]>(&r[0]));
    tmem_ld_32x32(tcol + 32, *reinterpret_cast<uint32_t(*)[32]>(&r[32]));
    tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 32; ++i) {
        pk[i] = mul2q<T>(pack2<T>(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1])), sc2);
    }
    if (diag) {
#pragma unroll
        for (int i = 0; i < 32; ++i) pk[i] &= (2 * i < live ? 0x0000ffffu : 0u) | (2 * i + 1 < live ? 0xffff0000u : 0u);
    }
    tmem_st_32x32(tcol, pk);
    tmem_st_wait();
}

// The output tiles of a launch: `planes` planes, rows [row_begin,row_end) in tiles_m rows of tiles of tmo rows, tiles_n tiles of TN keys
// (causal: only those that reach a key <= query).
struct TileGeom {
    int C, row_begin, row_end, tiles_n, tiles_m, tmo, causal;
    int planes, tiles_per_plane;
    int groups, group_planes;                     // planes are worked through in groups
};
__host__ __device__ __forceinline__ int key_tiles(const TileGeom& g, int tm) {
    if (!g.causal) return g.tiles_n;
    const int q_last = g.row_begin + (tm + 1) * g.tmo < g.row_end ? g.row_begin + (tm + 1) * g.tmo : g.row_end;
    const int n = (q_last + TN - 1) / TN;
    return n < g.tiles_n ? n : g.tiles_n;
}
// All but the groups, which are up to the kernel (set_groups).
inline void set_tiles(TileGeom& g, long planes, int C, int W, int R, int causal, int row_begin, int row_end) {
    g.C = C; g.row_begin = row_begin; g.row_end = row_end; g.causal = causal ? 1 : 0;
    g.tmo = tile_rows(R);
    g.tiles_n = (W + TN - 1) / TN;
    g.tiles_m = (row_end - row_begin + g.tmo - 1) / g.tmo;
    g.planes = (int)planes;
    g.tiles_per_plane = 0;
    for (int tm = 0; tm < g.tiles_m; ++tm) g.tiles_per_plane += key_tiles(g, tm);
}
inline void set_groups(TileGeom& g, long groups) {
    g.groups = (int)(groups < 1 ? 1 : (groups > g.planes ? g.planes : groups));
    g.group_planes = (g.planes + g.groups - 1) / g.groups;
    g.groups = (g.planes + g.group_planes - 1) / g.group_planes;
}
// The walk below counts the tiles of a group times the CTAs in 32 bits.
inline bool tiles_countable(const TileGeom& g, int sms) { return (double)g.tiles_per_plane * g.group_planes * (sms + 1) < 4294967296.0; }

// A CTA's tiles: of every group of planes a contiguous range, so that all CTAs work on the same few planes at a time.
struct TileIter {
    int plane, head, tm, tn, nk, left, group;
    // The range of this CTA in group gr: returns its length.
    __device__ int range(const TileGeom& g, int gr, unsigned* first) const {
        const int p0 = gr * g.group_planes, np = min(g.group_planes, g.planes - p0);
        const unsigned tiles = (unsigned)np * (unsigned)g.tiles_per_plane;
        const unsigned c = (blockIdx.x + (unsigned)gr * (gridDim.x / 2 + 1)) % gridDim.x;      // who gets one tile more changes
        const unsigned t0 = tiles * c / gridDim.x;
        *first = t0;
        return (int)(tiles * (c + 1) / gridDim.x - t0);
    }
    __device__ int total(const TileGeom& g) const {
        int n = 0;
        unsigned t;
        for (int gr = 0; gr < g.groups; ++gr) n += range(g, gr, &t);
        return n;
    }
    __device__ void enter(const TileGeom& g) {
        unsigned t = 0;
        do left = group < g.groups ? range(g, group++, &t) : 1 << 30;
        while (left == 0);
        const unsigned p = t / (unsigned)g.tiles_per_plane;
        int r = (int)(t - p * (unsigned)g.tiles_per_plane);
        plane = (group - 1) * g.group_planes + (int)p;
        head = plane % g.C;
        for (tm = 0;; ++tm) {
            nk = key_tiles(g, tm);
            if (r < nk) break;
            r -= nk;
        }
        tn = r;
    }
    __device__ void init(const TileGeom& g) {
        group = 0;
        enter(g);
    }
    // returns true when the walk moved on to another row of tiles (another Q tile)
    __device__ bool next(const TileGeom& g) {
        if (--left == 0) {
            enter(g);
            return true;
        }
        if (++tn == nk) {
            tn = 0;
            if (++tm == g.tiles_m) {
                tm = 0;
                ++plane;
                if (++head == g.C) head = 0;
            }
            nk = key_tiles(g, tm);
            return true;
        }
        return false;
    }
    __device__ int m0(const TileGeom& g) const { return g.row_begin + tm * g.tmo; }
    __device__ int n0() const { return tn * TN; }
};

// ---- output ------------------------------------------------------------------------------------------
// Bytes between rows of a staging tile: one box of 112 columns, whole 32-byte sectors in memory.  (Two boxes of 56, without the two-way
// bank conflict of this pitch: score + conv kernel at B8 H16 S4096 845 us, 805 like this.)
constexpr int OUT_PITCH = TN * 2;
__host__ __device__ inline int out_bytes(int R) { return (tile_rows(R) * OUT_PITCH + 127) & ~127; }

// A thread's row of a finished accumulator at `tacc` -> 16 bits -> its row of a staging tile at `orow`.  `live`:
// columns on or below the diagonal, the others become 0 (`diag`: there are others, for some thread of the warp); `inside`: the lane
// carries an output row.  Whole-warp call; on return the accumulator has been read.
template <typename T>
__device__ __forceinline__ void stage_row(uint32_t tacc, uint8_t* orow, int live, bool diag, bool inside) {
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
        constexpr int OUT_COLS = TN / 2;
        uint32_t r[OUT_COLS], pk[OUT_COLS / 2];
        tmem_ld_32x32(tacc + (uint32_t)(h * OUT_COLS), *reinterpret_cast<uint32_t(*)[32]>(&r[0]));
        tmem_ld_32x16(tacc + (uint32_t)(h * OUT_COLS + 32), *reinterpret_cast<uint32_t(*)[16]>(&r[32]));
        tmem_ld_32x8(tacc + (uint32_t)(h * OUT_COLS + 48), *reinterpret_cast<uint32_t(*)[8]>(&r[48]));
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < OUT_COLS / 2; ++e) pk[e] = pack2<T>(__uint_as_float(r[2 * e]), __uint_as_float(r[2 * e + 1]));
        if (diag) {
            const int nl = live - h * OUT_COLS;
#pragma unroll
            for (int e = 0; e < OUT_COLS / 2; ++e) pk[e] &= (2 * e < nl ? 0x0000ffffu : 0u) | (2 * e + 1 < nl ? 0xffff0000u : 0u);
        }
        if (inside) {
#pragma unroll
            for (int c = 0; c < OUT_COLS / 8; ++c)
                *reinterpret_cast<uint4*>(orow + h * OUT_COLS * 2 + c * 16) = make_uint4(pk[4 * c], pk[4 * c + 1], pk[4 * c + 2], pk[4 * c + 3]);
        }
    }
}

}  // namespace qc
}  // namespace mta
