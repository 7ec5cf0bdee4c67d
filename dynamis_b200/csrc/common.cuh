// Shared device/host helpers for the dynb kernels (sm_100a only).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/dynb.h"

namespace dynb {

// ---- small vector type usable for float and double records -----------------------------
template <typename T> struct Vec4;
template <> struct __align__(16) Vec4<float> { float x, y, z, w; };
template <> struct __align__(32) Vec4<double> { double x, y, z, w; };

template <typename T> struct IntOf;
template <> struct IntOf<float> { using type = int32_t; };
template <> struct IntOf<double> { using type = int64_t; };

__device__ __forceinline__ float bits_to_real(int32_t v, float) { return __int_as_float(v); }
__device__ __forceinline__ double bits_to_real(int32_t v, double) { return __longlong_as_double((long long)v); }
__device__ __forceinline__ int32_t real_to_bits(float v) { return __float_as_int(v); }
__device__ __forceinline__ int32_t real_to_bits(double v) { return (int32_t)__double_as_longlong(v); }

// ---- order-preserving float <-> unsigned maps for atomicMin / atomicMax ----------------
__device__ __forceinline__ uint32_t ordered_u32(float f)
{
    uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float unordered_f32(uint32_t u)
{
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}
__device__ __forceinline__ unsigned long long ordered_u64(double f)
{
    unsigned long long u = (unsigned long long)__double_as_longlong(f);
    return (u & 0x8000000000000000ull) ? ~u : (u | 0x8000000000000000ull);
}
__device__ __forceinline__ double unordered_f64(unsigned long long u)
{
    return __longlong_as_double((long long)((u & 0x8000000000000000ull) ? (u & 0x7fffffffffffffffull) : ~u));
}

// ---- warp primitives ---------------------------------------------------------------------
__device__ __forceinline__ int warp_excl_scan(int v, int lane, int* total)
{
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    *total = __shfl_sync(0xffffffffu, x, 31);
    return x - v;
}

__device__ __forceinline__ uint32_t lanemask_lt()
{
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// ---- chained launches ----------------------------------------------------------------------
// A kernel of a chain is launched while its predecessor still runs: its blocks take the places that the predecessor's leave, and wait in
// chain_begin() until that grid has ended and what it wrote can be seen.  Every thread of such a kernel calls it first, before the
// first access to memory, so that the end of a grid implies the end of all grids before it.  Pointers to what predecessors write
// are not declared __restrict__ in these kernels: the compiler may move reads through such a pointer in front of the wait.
// 1 to 2 us of every pair of short kernels: KD-tree of 1 M atoms 274 -> 242 us, rebuild 438 -> 403, refresh 696 -> 648, graph of 32 k atoms 111 -> 96.
__device__ __forceinline__ void chain_begin()
{
    asm volatile("griddepcontrol.launch_dependents;\n\tgriddepcontrol.wait;" ::: "memory");
}
template <typename... P, typename... A>
static inline cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args)
{
    cudaLaunchAttribute overlap;
    overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    overlap.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config = {};
    config.gridDim = grid;
    config.blockDim = block;
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    config.attrs = &overlap;
    config.numAttrs = 1;
    return cudaLaunchKernelEx(&config, kernel, static_cast<P>(args)...);
}

// ---- host-side launch check --------------------------------------------------------------
#define DYNB_CUDA_OK(expr)                                \
    do {                                                  \
        cudaError_t _e = (expr);                          \
        if (_e != cudaSuccess) return dynb::fail_cuda(_e, #expr); \
    } while (0)

int fail_cuda(cudaError_t e, const char* what);
int fail_arg(const char* what);
void set_last_error(const char* msg);

// Where the device can write to `host` (16-byte aligned pinned memory), or nullptr.
static inline void* device_view_of_host(void* host)
{
    if (reinterpret_cast<uintptr_t>(host) % 16 != 0) return nullptr;
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, host) != cudaSuccess) {
        (void)cudaGetLastError();
        return nullptr;
    }
    return at.type == cudaMemoryTypeHost ? at.devicePointer : nullptr;
}

static inline int64_t align_up(int64_t v, int64_t a) { return (v + a - 1) / a * a; }
static inline int sm_count_cached()
{
    static int cached[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    if (cached[dev] == 0) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
        cached[dev] = n;
    }
    return cached[dev];
}

}  // namespace dynb
