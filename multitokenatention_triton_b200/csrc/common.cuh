// Shared host/device helpers of the mta_b200 library: status codes, error text, dtype plumbing.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <cstdarg>
#include <cstdio>

#include "../../include/mta_b200.h"

namespace mta {

// ---- host side -------------------------------------------------------------------------------
void set_error(const char* fmt, ...);          // thread-local message for mta_last_error()
void count_launch(int n = 1);                  // bumps the per-thread launch counter
int variant(const char* key);                  // value set through mta_set_variant (0 = auto)
int check_device();                            // MTA_OK when the current device is sm_100

#define MTA_REQUIRE(cond, ...)                                  \
    do {                                                        \
        if (!(cond)) {                                          \
            ::mta::set_error(__VA_ARGS__);                      \
            return MTA_ERR_INVALID;                             \
        }                                                       \
    } while (0)

#define MTA_CUDA_OK(expr)                                                                   \
    do {                                                                                    \
        cudaError_t e__ = (expr);                                                           \
        if (e__ != cudaSuccess) {                                                           \
            ::mta::set_error("%s failed: %s (%s:%d)", #expr, cudaGetErrorString(e__),       \
                             __FILE__, __LINE__);                                           \
            return MTA_ERR_CUDA;                                                            \
        }                                                                                   \
    } while (0)

// Launch status after a <<<>>> statement; counts the launch.
#define MTA_LAUNCH_OK(name)                                                                 \
    do {                                                                                    \
        cudaError_t e__ = cudaGetLastError();                                               \
        if (e__ != cudaSuccess) {                                                           \
            ::mta::set_error("launch of %s failed: %s", name, cudaGetErrorString(e__));     \
            return MTA_ERR_CUDA;                                                            \
        }                                                                                   \
        ::mta::count_launch();                                                              \
    } while (0)

int sm_count(int* out);                        // SMs of the current device (looked up once per device)

constexpr int MAX_DEVICES_KNOWN = 64;

// Makes `bytes` of dynamic shared memory available to KERNEL on the current device.  The attribute is a maximum, so it is only
// set when a launch needs more than any before it: setting it costs more than the launch's other host work.
template <auto KERNEL> int ensure_smem(size_t bytes) {
    static std::atomic<int> have[MAX_DEVICES_KNOWN];
    if (bytes <= 32 * 1024) return MTA_OK;      // leaves room for static arrays inside the default 48 KB
    int dev = 0;
    MTA_CUDA_OK(cudaGetDevice(&dev));
    if (dev < MAX_DEVICES_KNOWN && have[dev].load(std::memory_order_relaxed) >= (int)bytes) return MTA_OK;
    MTA_CUDA_OK(cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    if (dev < MAX_DEVICES_KNOWN) {
        int old = have[dev].load(std::memory_order_relaxed);
        while (old < (int)bytes && !have[dev].compare_exchange_weak(old, (int)bytes, std::memory_order_relaxed)) {}
    }
    return MTA_OK;
}

// Launches KERNEL so that it may start before its predecessor in the stream has ended (programmatic dependent launch): what
// it does before pdl_wait() - barriers, tensor memory, descriptors - then overlaps the predecessor's last blocks.  KERNEL must
// call pdl_wait() before it reads or writes anything that another kernel may touch; the one exception, the flag of a wait that gave up,
// is read again after it (flag_down() in tc05.cuh).
// Measured: B1 H16 S128 forward 51 -> 37 us, B1 H16 S2048 211 -> 188.  Only up to PDL_MAX_BLOCKS blocks: every block of such a
// launch starts later, and over the fifty waves of a long grid that cost more than the overlap gave (head mix of B8 H16 S4096,
// 65536 blocks: 0.15 ms of 0.77).
constexpr unsigned PDL_MAX_BLOCKS = 4096;
template <auto KERNEL, typename... Args>
int launch_kernel_early(bool early, const char* name, dim3 grid, unsigned block, size_t smem, cudaStream_t st, Args... args) {
    if (int rc = ensure_smem<KERNEL>(smem)) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = early ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, KERNEL, args...);
    if (e != cudaSuccess) {
        cudaGetLastError();
        set_error("launch of %s failed: %s", name, cudaGetErrorString(e));
        return MTA_ERR_CUDA;
    }
    count_launch();
    return MTA_OK;
}
template <auto KERNEL, typename... Args>
int launch_kernel(const char* name, dim3 grid, unsigned block, size_t smem, cudaStream_t st, Args... args) {
    return launch_kernel_early<KERNEL>((unsigned long long)grid.x * grid.y * grid.z <= PDL_MAX_BLOCKS, name, grid, block, smem, st, args...);
}

inline size_t dtype_size(int dt) { return dt == MTA_F32 ? 4 : 2; }
inline bool dtype_ok(int dt) { return dt == MTA_F32 || dt == MTA_BF16 || dt == MTA_F16; }
inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// ---- device side -----------------------------------------------------------------------------
// Waits until everything before this kernel in the stream is complete and visible (returns at once in an ordinary launch), then
// lets the next kernel begin its own setup.  In this order, so that a kernel that has started knows its predecessors' predecessors
// to be complete; and after this kernel's tensor memory is allocated: the next kernel's blocks could otherwise take columns that a
// block of this one still needs, and wait for it.
// A kernel launched with `early_weights` reads its weights before it calls this, while its predecessor still runs.  Only kernels
// that are not the first of a library call may: the call's first kernel waits for everything before the call, the weights'
// writers among it, and no later kernel of the call starts before that.
__device__ __forceinline__ void pdl_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <typename T> __device__ __forceinline__ float to_f32(T v);
template <> __device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <> __device__ __forceinline__ float to_f32<__half>(__half v) { return __half2float(v); }

template <typename T> __device__ __forceinline__ T from_f32(float v);
template <> __device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <> __device__ __forceinline__ __half from_f32<__half>(float v) { return __float2half_rn(v); }

// Two floats rounded to a 16-bit T, the first in the low half of the word.
template <typename T> __device__ __forceinline__ uint32_t pack2(float lo, float hi);
template <> __device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float lo, float hi) {
    const __nv_bfloat162 r = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&r);
}
template <> __device__ __forceinline__ uint32_t pack2<__half>(float lo, float hi) {
    const __half2 r = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&r);
}

// Round a float to T and back: the place where a 16-bit run of the reference rounds an intermediate.
template <typename T> __device__ __forceinline__ float round_to(float v) { return to_f32<T>(from_f32<T>(v)); }

// Weight element `i` of an array whose dtype is only known at run time (weights are tiny).
__device__ __forceinline__ float load_weight(const void* w, long i, int w_dtype) {
    if (w_dtype == MTA_F32) return reinterpret_cast<const float*>(w)[i];
    if (w_dtype == MTA_BF16) return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(w)[i]);
    return __half2float(reinterpret_cast<const __half*>(w)[i]);
}

// Stores v as element `i` of an array whose dtype is only known at run time (weight gradients are tiny).
__device__ __forceinline__ void store_weight(void* w, long i, int w_dtype, float v) {
    if (w_dtype == MTA_F32) reinterpret_cast<float*>(w)[i] = v;
    else if (w_dtype == MTA_BF16) reinterpret_cast<__nv_bfloat16*>(w)[i] = __float2bfloat16_rn(v);
    else reinterpret_cast<__half*>(w)[i] = __float2half_rn(v);
}

template <typename T> struct DTypeOf;
template <> struct DTypeOf<float> { static constexpr int value = MTA_F32; };
template <> struct DTypeOf<__nv_bfloat16> { static constexpr int value = MTA_BF16; };
template <> struct DTypeOf<__half> { static constexpr int value = MTA_F16; };

// A view of score planes stored as [plane][row - row0][col]: the same kernels serve whole (N,C,H,W)
// tensors (row0 = 0, plane_stride = H*W) and row-range scratch buffers of the fused forward.
struct PlaneView {
    long plane_stride;   // elements between consecutive planes
    int row0;            // absolute index of the first stored row
    int width;           // row pitch = number of columns
    __host__ __device__ long at(long plane, int row, int col) const {
        return plane * plane_stride + (long)(row - row0) * width + col;
    }
};

}  // namespace mta
