// Products of a causal score plane with (rows x D) matrices on the 5th-generation tensor cores (tcgen05), 16-bit dtypes:
//   O[128 q x D] = scale * sum over keys <= q     P[q x k] V[k x D]     (A K-major, B MN-major): P V, and dS K of a backward
//   O[128 k x D] = scale * sum over queries >= k  P[q x k] X[q x D]     (A and B MN-major): P^T dO and dS^T Q of a backward
// Operand tiles arrive by TMA (128-byte swizzle, out-of-range rows and columns read as zero), the
// accumulator lives in tensor memory, and only tiles that touch keys k <= q are visited when causal.
// They stand in for the torch.matmul calls at mta_attention_triton.py:68-71 and :89.
#include <atomic>
#include <cstddef>
#include <cstring>
#include <mutex>

#include "kernels.cuh"
#include "tc05.cuh"

namespace mta {

// ---- host helpers ----------------------------------------------------------------------------------
namespace {
// What a bounded wait raises when it gives up: the flag the kernels test on entry, and the address of its mirror in
// page-locked host memory, which lets the entry points see a timeout without synchronising with the device.
struct WaitFlag {
    int flag;
    int pad;
    int* host_mirror;
};
__device__ WaitFlag g_wait_timeout = {0, 0, nullptr};
std::mutex g_flag_mutex;
std::atomic<int*> g_flag_dev[64];  // per device: address of g_wait_timeout.flag
int* g_flag_host[64] = {};         // per device: the host mirror (mapped page-locked memory)

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn g_encode = nullptr;
std::once_flag g_encode_once;

EncodeTiledFn encode_fn() {
    std::call_once(g_encode_once, [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            g_encode = reinterpret_cast<EncodeTiledFn>(fn);
    });
    return g_encode;
}
}  // namespace

int wait_flag_ptr(int** out) {
    int dev = 0;
    MTA_CUDA_OK(cudaGetDevice(&dev));
    MTA_REQUIRE(dev >= 0 && dev < 64, "device index %d out of range", dev);
    if ((*out = g_flag_dev[dev].load(std::memory_order_acquire))) return MTA_OK;
    std::lock_guard<std::mutex> lock(g_flag_mutex);
    if (!g_flag_dev[dev].load(std::memory_order_relaxed)) {
        // first tcgen05 launch on this device: look up the flag and give it a host-visible mirror (4 bytes of mapped
        // page-locked memory, kept until the process ends)
        void* p = nullptr;
        MTA_CUDA_OK(cudaGetSymbolAddress(&p, g_wait_timeout));
        int* host = nullptr;
        int* host_dev = nullptr;
        MTA_CUDA_OK(cudaHostAlloc(reinterpret_cast<void**>(&host), sizeof(int), cudaHostAllocMapped));
        *host = 0;
        MTA_CUDA_OK(cudaHostGetDevicePointer(reinterpret_cast<void**>(&host_dev), host, 0));
        MTA_CUDA_OK(cudaMemcpy(static_cast<char*>(p) + offsetof(WaitFlag, host_mirror), &host_dev, sizeof(host_dev), cudaMemcpyHostToDevice));
        g_flag_host[dev] = host;
        g_flag_dev[dev].store(static_cast<int*>(p), std::memory_order_release);
    }
    *out = g_flag_dev[dev].load(std::memory_order_relaxed);
    return MTA_OK;
}

// True when a bounded wait has given up on the current device since the last mta_device_status (no synchronisation:
// reads the host mirror the kernel wrote).
bool wait_flag_raised() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
    const int* host = g_flag_host[dev];
    return host && *reinterpret_cast<const volatile int*>(host) != 0;
}

// Raises the flag from the host as a kernel's timed-out wait would (fault injection without a fault on the device).
int wait_flag_inject(cudaStream_t st) {
    int* flag = nullptr;
    if (int rc = wait_flag_ptr(&flag)) return rc;
    int dev = 0;
    MTA_CUDA_OK(cudaGetDevice(&dev));
    const int one = 1;
    MTA_CUDA_OK(cudaMemcpyAsync(flag, &one, sizeof(int), cudaMemcpyHostToDevice, st));
    MTA_CUDA_OK(cudaStreamSynchronize(st));
    *reinterpret_cast<volatile int*>(g_flag_host[dev]) = 1;
    return MTA_OK;
}

// A kernel whose bounded wait runs out, with a limit of a few milliseconds: nothing arrives on its barrier.  It lets its
// successor start first, as every kernel does.
__global__ void wait_runs_out_kernel(int* err_flag) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) {
        tc05::mbar_init(&bar, 1);
        tc05::fence_mbar_init();
    }
    __syncwarp();
    pdl_wait();
    if (threadIdx.x == 0) tc05::mbar_wait(&bar, 0, err_flag, 2048);
}

int wait_flag_inject_late(cudaStream_t st) {
    int* flag = nullptr;
    if (int rc = wait_flag_ptr(&flag)) return rc;
    return launch_kernel<wait_runs_out_kernel>("wait_runs_out_kernel", dim3(1), 32, 0, st, flag);
}

int make_tensor_map_3d(CUtensorMap* out, const void* base, uint64_t planes, uint64_t rows, uint64_t cols,
                       uint64_t row_pitch_elems, uint64_t plane_pitch_elems, uint32_t box_cols, uint32_t box_rows,
                       bool swizzle128) {
    return make_tensor_map_3d_mode(out, base, planes, rows, cols, row_pitch_elems, plane_pitch_elems, box_cols, box_rows,
                                   swizzle128 ? 128 : 0);
}

int make_tensor_map_3d_mode(CUtensorMap* out, const void* base, uint64_t planes, uint64_t rows, uint64_t cols,
                            uint64_t row_pitch_elems, uint64_t plane_pitch_elems, uint32_t box_cols, uint32_t box_rows,
                            int swizzle_bytes, uint32_t box_planes) {
    // A map is a pure function of its description, and a program calls with the same few descriptions again and again: each
    // thread keeps the last maps it encoded (direct-mapped by a hash of the description, 24 KB).
    struct Key {
        const void* base;
        uint64_t planes, rows, cols, row_pitch, plane_pitch;
        uint32_t box_cols, box_rows, box_planes;
        int swizzle;
    };
    struct Entry {
        Key key;
        CUtensorMap map;
    };
    constexpr int ENTRIES = 128;
    static thread_local Entry cache[ENTRIES] = {};
    const Key key{base, planes, rows, cols, row_pitch_elems, plane_pitch_elems, box_cols, box_rows, box_planes, swizzle_bytes};
    static_assert(sizeof(Key) == 64, "compared and hashed as bytes: no padding");
    uint64_t words[8], hash = 0;
    memcpy(words, &key, sizeof(key));
    for (uint64_t w : words) hash = (hash ^ w) * 0x9E3779B97F4A7C15ull ^ (hash >> 29);
    Entry& entry = cache[(hash >> 40) % ENTRIES];
    if (base && memcmp(&entry.key, &key, sizeof(key)) == 0) {
        *out = entry.map;
        return MTA_OK;
    }
    const bool swizzle128 = swizzle_bytes == 128;
    EncodeTiledFn fn = encode_fn();
    if (!fn) {
        set_error("cuTensorMapEncodeTiled is not available from this driver");
        return MTA_ERR_CUDA;
    }
    MTA_REQUIRE(aligned16(base) && (row_pitch_elems * 2) % 16 == 0 && (plane_pitch_elems * 2) % 16 == 0,
                "tensor map: base and pitches must be multiples of 16 bytes");
    cuuint64_t dims[3] = {cols, rows, planes};
    cuuint64_t strides[2] = {row_pitch_elems * 2, plane_pitch_elems * 2};
    MTA_REQUIRE(box_cols <= 256 && box_rows <= 256 && box_planes >= 1 && box_planes <= 256 && (box_cols * 2) % 16 == 0 && (!swizzle128 || box_cols == 64) &&
                    (swizzle_bytes != 32 || box_cols == 16) && (swizzle_bytes != 64 || box_cols == 32) &&
                    (swizzle_bytes == 0 || swizzle_bytes == 32 || swizzle_bytes == 64 || swizzle_bytes == 128),
                "tensor map: box %u x %u with a %d-byte swizzle is not supported", box_cols, box_rows, swizzle_bytes);
    cuuint32_t box[3] = {box_cols, box_rows, box_planes};
    cuuint32_t estr[3] = {1, 1, 1};
    const CUtensorMapSwizzle swizzle =
        swizzle128 ? CU_TENSOR_MAP_SWIZZLE_128B
                   : (swizzle_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : (swizzle_bytes == 32 ? CU_TENSOR_MAP_SWIZZLE_32B : CU_TENSOR_MAP_SWIZZLE_NONE));
    auto encode = [&] {
        return fn(out, CU_TENSOR_MAP_DATA_TYPE_UINT16, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    };
    CUresult r = encode();
    if (r == CUDA_ERROR_INVALID_CONTEXT) {
        // A thread whose first CUDA work is this call (autograd's, for one) has no current context yet: a driver function does
        // not set one up as the runtime's do.
        MTA_CUDA_OK(cudaFree(nullptr));
        r = encode();
    }
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
        return MTA_ERR_CUDA;
    }
    entry.key = key;
    entry.map = *out;
    return MTA_OK;
}

namespace {
using namespace tc05;

constexpr int TILE = 128;                 // rows of an operand tile / edge of a score tile
constexpr int BOX_BYTES = TILE * 128;     // one TMA box: 128 rows x 64 elements x 2 bytes = 16 KB

template <typename T> struct AbFormat;
template <> struct AbFormat<__nv_bfloat16> { static constexpr int value = 1; };
template <> struct AbFormat<__half> { static constexpr int value = 0; };

__device__ __forceinline__ uint8_t* align_1024(uint8_t* p) {
    return reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(p) + 1023) & ~uintptr_t(1023));
}

// ------------------------------------------------------------------------------------------------
// Output tile of 128 rows = sum over steps of 64 contraction indices (keys, or queries when TRANS).  Warp 0: TMA producer;
// warp 1: MMA issuer; warps 2..5: before the accumulator is complete they zero what lies above the diagonal in the few tiles
// that straddle it (128 threads; one warp doing it was a serial stretch of about a microsecond per tile) and apply the
// dropout, then they are the epilogue.
constexpr int PV_STAGES = 3;
constexpr int PV_THREADS = 192;
constexpr int PV_KEYS = 64;               // contraction indices per pipeline stage: 32 KB stages, so two CTAs fit on an SM and
                                          // one CTA's start-up and epilogue overlap the other's steady state
constexpr int PV_VBOX_BYTES = PV_KEYS * 128;   // one box of the V tile: 64 rows x 64 elements
constexpr int PV_PLANE_GROUP = 16;
constexpr int PV_DIAG = 3;                // most steps of a tile that straddle the diagonal (128 rows from any row on)

// DROP: the dropout of dropout.cuh is applied to every P tile in shared memory before its MMAs (a thread owns a row).
// TRANS: the P tile is read as its transpose: 64 query rows x 128 keys, two boxes of 64 keys.
template <typename T, int D, bool DROP, bool TRANS>
__global__ void __launch_bounds__(PV_THREADS)
pv_tc05_kernel(const __grid_constant__ CUtensorMap mp, const __grid_constant__ CUtensorMap mv, T* __restrict__ o,
               int planes, int p_row0, int S, int causal, int row_begin, int row_end, float scale, int* err_flag, DropoutSpec drop) {
    constexpr int NBOX_V = D / 64;
    constexpr int P_BYTES = BOX_BYTES;                     // 128 q x 64 k, or 64 q x 128 k
    constexpr int V_BYTES = NBOX_V * PV_VBOX_BYTES;        // 64 rows x D
    constexpr int STAGE_BYTES = P_BYTES + V_BYTES;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = align_1024(smem_raw);
    __shared__ __align__(8) uint64_t full_bar[PV_STAGES], empty_bar[PV_STAGES], drop_bar[PV_STAGES], go_bar[PV_DIAG], diag_bar[PV_DIAG],
        acc_bar;
    __shared__ uint32_t tmem_slot;

    __shared__ int abort_flag;
    if (gave_up_before(err_flag, &abort_flag)) return;
    // Heaviest tiles first (the last query tile has all keys, or the first key tile all queries), over groups of planes: plane by
    // plane, the last planes' heavy tiles start when little else is left (B1 H16 S2048: 30 us against 25); all planes at once,
    // the V tiles of 128 planes do not stay in L2 (B8 H16 S4096: 549 us against 441).
    const int n_qt = (row_end - row_begin + TILE - 1) / TILE;
    const int per_group = n_qt * PV_PLANE_GROUP, group = (int)blockIdx.x / per_group, in_group = (int)blockIdx.x % per_group;
    const int width = min(PV_PLANE_GROUP, planes - group * PV_PLANE_GROUP);
    const int bh = group * PV_PLANE_GROUP + in_group % width, t = in_group / width;
    const int tq = TRANS ? t : n_qt - 1 - t;
    const int q0 = row_begin + tq * TILE;                  // first output row (a query, or a key when TRANS)
    const int q_end = min(q0 + TILE, row_end);
    // steps [kt0, kt1) of 64 contraction indices: keys up to the tile's last query, or queries from the tile's first key on
    const int n_steps = (S + PV_KEYS - 1) / PV_KEYS;
    const int kt0 = TRANS && causal ? q0 / PV_KEYS : 0;
    const int kt1 = !TRANS && causal ? min((q_end + PV_KEYS - 1) / PV_KEYS, n_steps) : n_steps;
    // steps [d0, d1) straddle the diagonal
    const int d0 = !causal ? kt1 : (TRANS ? kt0 : min((q0 + 1) / PV_KEYS, kt1));
    const int d1 = !causal ? kt1 : (TRANS ? min((q0 + TILE - 2) / PV_KEYS + 1, kt1) : kt1);
    const int nk = kt1 - kt0;
    const int warp = warp_index(), lane = threadIdx.x & 31;

    if (warp == 0) {
        if (lane == 0) {
            for (int i = 0; i < PV_STAGES; ++i) {
                mbar_init(&full_bar[i], 1);
                mbar_init(&empty_bar[i], 1);
                mbar_init(&drop_bar[i], 4);
            }
            for (int i = 0; i < PV_DIAG; ++i) {
                mbar_init(&go_bar[i], 1);
                mbar_init(&diag_bar[i], 4);
            }
            mbar_init(&acc_bar, 1);
            fence_mbar_init();
            prefetch_tensormap(&mp);
            prefetch_tensormap(&mv);
        }
        __syncwarp();
        tmem_alloc(&tmem_slot, D < 32 ? 32 : D);
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = tmem_slot;
    pdl_wait();

    if (warp == 0) {
        if (lane == 0) {
            for (int it = 0; it < nk; ++it) {
                const int kt = kt0 + it, st = it % PV_STAGES, use = it / PV_STAGES;
                if (use > 0) mbar_wait(&empty_bar[st], (use - 1) & 1, err_flag);
                uint8_t* sp = smem + st * STAGE_BYTES;
                uint8_t* sv = sp + P_BYTES;
                mbar_expect_tx(&full_bar[st], STAGE_BYTES);
                if (TRANS) {
                    tma_load_3d(sp, &mp, &full_bar[st], q0, kt * PV_KEYS - p_row0, bh);
                    tma_load_3d(sp + P_BYTES / 2, &mp, &full_bar[st], q0 + 64, kt * PV_KEYS - p_row0, bh);
                } else {
                    tma_load_3d(sp, &mp, &full_bar[st], kt * PV_KEYS, q0 - p_row0, bh);
                }
#pragma unroll
                for (int j = 0; j < NBOX_V; ++j) tma_load_3d(sv + j * PV_VBOX_BYTES, &mv, &full_bar[st], j * 64, kt * PV_KEYS, bh);
            }
        }
    } else if (warp == 1) {
        constexpr uint32_t idesc = instr_desc_f16(AbFormat<T>::value, TRANS ? 1 : 0, 1, TILE, D);
        const uint32_t el = elect_one();
        for (int it = 0; it < nk; ++it) {
            const int kt = kt0 + it, st = it % PV_STAGES, use = it / PV_STAGES;
            uint8_t* sp = smem + st * STAGE_BYTES;
            uint8_t* sv = sp + P_BYTES;
            mbar_wait(&full_bar[st], use & 1, err_flag);
            if (DROP) mbar_wait(&drop_bar[st], use & 1, err_flag);                      // the dropout has been applied
            if (kt >= d0 && kt < d1) {                                                  // the part above the diagonal becomes zero
                // The warps that zero it visit few of the stages, so they cannot follow full_bar's phases themselves (a wait
                // tells two phases apart, no more): this warp, which sees every phase, calls them.
                if (!DROP && lane == 0) mbar_arrive(&go_bar[kt - d0]);
                mbar_wait_spin(&diag_bar[kt - d0], 0, err_flag);
            }
            __syncwarp();
            fence_after_sync();
#pragma unroll
            for (int kk = 0; kk < PV_KEYS / 16; ++kk) {
                const uint64_t da = TRANS ? smem_desc_sw128(smem_u32(sp) + kk * 16 * 128, P_BYTES / 2, 1024)
                                          : smem_desc_sw128(smem_u32(sp) + kk * 32, 16, 1024);
                const uint64_t db = smem_desc_sw128(smem_u32(sv) + kk * 16 * 128, PV_VBOX_BYTES, 1024);
                mma_f16_ss(tmem, da, db, idesc, (it > 0 || kk > 0) ? 1u : 0u, el);
            }
            mma_commit(&empty_bar[st], el);
            if (it == nk - 1) mma_commit(&acc_bar, el);
        }
    } else {
        const int et = (int)threadIdx.x - 64;                // 0..127
        const int flag = read_flag(err_flag);                // looked at after the loop: these warps clear the diagonal tiles first
        for (int it = DROP ? 0 : d0 - kt0; it < (DROP ? nk : d1 - kt0); ++it) {
            const int kt = kt0 + it, st = it % PV_STAGES, use = it / PV_STAGES;
            uint8_t* sp = smem + st * STAGE_BYTES;
            const int k0 = kt * PV_KEYS;
            if (DROP) mbar_wait(&full_bar[st], use & 1, err_flag);
            else mbar_wait(&go_bar[kt - d0], 0, err_flag);
            if (DROP) {
                const uint32_t thr = drop.keep_threshold();
                const float keep_scale = drop.scale();
#pragma unroll 2
                for (int ch = 0; ch < 8; ++ch) {
                    const uint32_t keep = dropout_keep8(drop.seed, (uint32_t)bh, (uint32_t)(q0 + et), (uint32_t)(kt * (PV_KEYS / 8) + ch), thr);
                    T* e8 = reinterpret_cast<T*>(sp + et * 128 + ((ch ^ (et & 7)) << 4));
#pragma unroll
                    for (int e = 0; e < 8; ++e) e8[e] = (keep >> e) & 1u ? from_f32<T>(to_f32<T>(e8[e]) * keep_scale) : from_f32<T>(0.0f);
                }
            }
            if (kt >= d0 && kt < d1) {
                // Keys above the diagonal must contribute nothing, whatever the buffer holds there: a thread takes one line of
                // 64 keys (a row of the tile; when TRANS one of the two halves of a row) and zeroes it from the first such key on.
                const int line = TRANS ? et & 63 : et, key_first = TRANS ? q0 + (et >> 6) * 64 : k0;
                const int qrow = TRANS ? k0 + line : q0 + line;
                uint8_t* lp = sp + (TRANS ? (et >> 6) * (P_BYTES / 2) : 0) + line * 128;
                int first = qrow + 1 - key_first;            // first key of the line to zero
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
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) {
                if (DROP) mbar_arrive(&drop_bar[st]);
                if (kt >= d0 && kt < d1) mbar_arrive(&diag_bar[kt - d0]);
            }
        }
        mbar_wait(&acc_bar, 0, err_flag);
        __syncwarp();
        fence_after_sync();
        const int quarter = warp & 3;                    // TMEM lanes this warp may read
        const int q = q0 + quarter * 32 + lane;
        T* orow = o + ((long)bh * S + (q < q_end ? q : q0)) * D;
#pragma unroll 1
        for (int c = 0; c < D / 32; ++c) {
            uint32_t r[32];
            tmem_ld_32x32(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(c * 32), r);
            tmem_ld_wait();
            if (q >= q_end || flag != 0) continue;
#pragma unroll
            for (int v8 = 0; v8 < 4; ++v8) {
                float f[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(r[v8 * 8 + e]) * scale;
                uint4 w;
                w.x = pack2<T>(f[0], f[1]);
                w.y = pack2<T>(f[2], f[3]);
                w.z = pack2<T>(f[4], f[5]);
                w.w = pack2<T>(f[6], f[7]);
                *reinterpret_cast<uint4*>(orow + c * 32 + v8 * 8) = w;
            }
        }
    }
    fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, D < 32 ? 32 : D);
}

template <typename T, int D, bool DROP, bool TRANS>
int launch_pv(const void* p, PlaneView pview, const void* v, void* o, int B, int H, int S, int causal, int row_begin,
              int row_end, long p_rows_stored, float scale, cudaStream_t st, DropoutSpec drop) {
    CUtensorMap mp, mv;
    int rc;
    if ((rc = make_tensor_map_3d(&mp, p, (uint64_t)B * H, (uint64_t)p_rows_stored, S, (uint64_t)pview.width, (uint64_t)pview.plane_stride, 64,
                                 TRANS ? PV_KEYS : TILE, true)))
        return rc;
    if ((rc = make_tensor_map_3d(&mv, v, (uint64_t)B * H, S, D, D, (uint64_t)S * D, 64, PV_KEYS, true))) return rc;
    int* flag = nullptr;
    if ((rc = wait_flag_ptr(&flag))) return rc;
    const int n_qt = (row_end - row_begin + TILE - 1) / TILE;
    const size_t smem = (size_t)PV_STAGES * (BOX_BYTES + (D / 64) * PV_VBOX_BYTES) + 1024;
    const unsigned grid = (unsigned)(B * H * n_qt);
    return launch_kernel<pv_tc05_kernel<T, D, DROP, TRANS>>("pv_tc05_kernel", grid, PV_THREADS, smem, st, mp, mv, static_cast<T*>(o), B * H,
                                                            pview.row0, S, causal, row_begin, row_end, scale, flag, drop);
}

template <typename T, int D>
int launch_pv_kind(const void* p, PlaneView pview, const void* v, void* o, int B, int H, int S, int causal, int row_begin, int row_end,
                   long p_rows_stored, bool trans, float scale, cudaStream_t st, DropoutSpec drop) {
#define MTA_PV_KIND(DROP, TRANS) \
    return launch_pv<T, D, DROP, TRANS>(p, pview, v, o, B, H, S, causal, row_begin, row_end, p_rows_stored, scale, st, drop)
    if (trans) MTA_PV_KIND(false, true);
    if (drop.on()) MTA_PV_KIND(true, false);
    MTA_PV_KIND(false, false);
#undef MTA_PV_KIND
}

}  // namespace

bool tc05_contractions_supported(int S, int D, int dtype, const void* a, const void* b, const void* c, PlaneView view) {
    return dtype != MTA_F32 && (D == 64 || D == 128) && view.width >= S && view.width % 8 == 0 && view.plane_stride % 8 == 0 &&
           aligned16(a) && aligned16(b) && aligned16(c);
}

int pv_tc05_launch(const void* p, PlaneView pview, long p_rows_stored, const void* v, void* o, int B, int H, int S, int D,
                   int causal, int row_begin, int row_end, int dtype, cudaStream_t st, DropoutSpec drop, bool trans, float scale) {
#define MTA_PV(TT, DD) return launch_pv_kind<TT, DD>(p, pview, v, o, B, H, S, causal, row_begin, row_end, p_rows_stored, trans, scale, st, drop)
    if (dtype == MTA_BF16) { if (D == 64) MTA_PV(__nv_bfloat16, 64); MTA_PV(__nv_bfloat16, 128); }
    if (D == 64) MTA_PV(__half, 64);
    MTA_PV(__half, 128);
#undef MTA_PV
}

// Reads and clears the flag that bounded device-side waits raise.  Synchronises the stream.
int device_wait_status(cudaStream_t st, int* timed_out) {
    int* flag = nullptr;
    if (int rc = wait_flag_ptr(&flag)) return rc;
    int h = 0;
    MTA_CUDA_OK(cudaMemcpyAsync(&h, flag, sizeof(int), cudaMemcpyDeviceToHost, st));
    MTA_CUDA_OK(cudaStreamSynchronize(st));
    int dev = 0;
    MTA_CUDA_OK(cudaGetDevice(&dev));
    if (h || *reinterpret_cast<volatile int*>(g_flag_host[dev])) {
        int zero = 0;
        MTA_CUDA_OK(cudaMemcpyAsync(flag, &zero, sizeof(int), cudaMemcpyHostToDevice, st));
        MTA_CUDA_OK(cudaStreamSynchronize(st));
        *reinterpret_cast<volatile int*>(g_flag_host[dev]) = 0;
        h = 1;
    }
    *timed_out = h;
    return MTA_OK;
}

}  // namespace mta
