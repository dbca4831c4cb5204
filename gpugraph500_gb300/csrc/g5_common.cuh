// g5_common.cuh -- shared definitions of the libg5bfs CUDA sources.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>
#include <cstdio>

#include "g5bfs.h"

#define G5_NUM_SMS_DEFAULT 152

namespace g5 {

// Maps a CUDA error to a status code (allocation failures are OOM).
inline g5_status cuda_status(cudaError_t e)
{
    if (e == cudaSuccess) return G5_OK;
    if (e == cudaErrorMemoryAllocation) return G5_ERR_OOM;
    if (e == cudaErrorNoDevice || e == cudaErrorInsufficientDriver) return G5_ERR_NO_DEVICE;
    return G5_ERR_CUDA;
}

// Returns from the enclosing function with a status if a CUDA call fails.
#define G5_CUDA(call)                                                            \
    do {                                                                         \
        cudaError_t g5_e_ = (call);                                              \
        if (g5_e_ != cudaSuccess) {                                              \
            if (getenv("G5_VERBOSE"))                                            \
                fprintf(stderr, "g5: %s failed at %s:%d: %s\n", #call, __FILE__, \
                        __LINE__, cudaGetErrorString(g5_e_));                    \
            return ::g5::cuda_status(g5_e_);                                     \
        }                                                                        \
    } while (0)

#define G5_TRY(call)                       \
    do {                                   \
        g5_status g5_s_ = (call);          \
        if (g5_s_ != G5_OK) return g5_s_;  \
    } while (0)

// Number of SMs of the current device (cached per process).
int num_sms();

// True if p is a device or managed pointer.
bool is_device_ptr(const void *p);

// Grid of `per_sm` blocks per SM.
inline int grid_for(int per_sm) { return num_sms() * per_sm; }

// SMs of a cooperative grid that would otherwise take them all.  Such a grid
// begins when every block of it has its place, so one block of some other
// stream's long kernel (one that polls a flag, say) would hold it up until that
// kernel ends: 49 ms for a search of 0.2 ms beside a kernel of 50.  Two SMs are
// left out; us per search with 0, 2, 4 and 8 left out: scale 16 44.1, 43.8, 43.9,
// 44.1; 20 70.2, 70.6, 70.5, 71.2; 22 148.5, 149.1, 149.0, 149.2; 24 375, 378,
// 378, 382; 26 1266, 1279, 1285, 1312; per batch of 64 roots scale 22 2074, 2088,
// 2112, 2153; 24 5710, 5740, 5799, 5892.
constexpr int kSpareSms = 2;
inline int meeting_sms() { return num_sms() > 4 * kSpareSms ? num_sms() - kSpareSms : num_sms(); }

// Owning device buffer (freed on scope exit unless released).
template <class T>
struct DevBuf {
    T *p = nullptr;
    ~DevBuf()
    {
        if (p) cudaFree(p);
    }
    g5_status alloc(size_t count)
    {
        G5_CUDA(cudaMalloc(&p, sizeof(T) * (count ? count : 1)));
        return G5_OK;
    }
    T *release()
    {
        T *r = p;
        p = nullptr;
        return r;
    }
};

// Launches kern on s; with pdl, as a programmatic dependent of the kernel
// before it on the stream (the kernel must call g5_pdl_sync first).
template <typename... KArgs, typename... Args>
cudaError_t launch(bool pdl, void (*kern)(KArgs...), dim3 grid, dim3 block, cudaStream_t s, Args... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, args...);
}

// As launch(), with smem bytes of dynamic shared memory.
template <typename... KArgs, typename... Args>
cudaError_t launch_dyn(bool pdl, void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                       Args... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, args...);
}

}  // namespace g5

// Device-side error flags (bit set in a status word).
enum : uint32_t {
    G5_DEVERR_CAPACITY = 1u,
    G5_DEVERR_CORRUPT = 2u,
    G5_DEVERR_MISMATCH = 4u,
    G5_DEVERR_LEVELS = 8u,
    G5_DEVERR_WAIT = 16u,  // a bounded device wait ran out
};

__device__ __forceinline__ int g5_lane() { return threadIdx.x & 31; }

// Programmatic dependent launch: waits until the kernel before this one on
// the stream has finished and its writes are visible, then lets the next
// launch start setting up while this one runs.  Both are no-ops for an
// ordinary launch; a kernel calls this before it reads anything.
__device__ __forceinline__ void g5_pdl_sync()
{
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
}
__device__ __forceinline__ unsigned g5_lanemask_lt()
{
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

__device__ __forceinline__ uint64_t warp_sum_u64(uint64_t v)
{
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    return v;
}

__device__ __forceinline__ uint32_t warp_excl_u32(uint32_t x, uint32_t &total)
{
    const int lane = g5_lane();
    uint32_t inc = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, inc, o);
        if (lane >= o) inc += y;
    }
    total = __shfl_sync(0xFFFFFFFFu, inc, 31);
    return inc - x;
}

// Sum over the warp of values below 2^51, in two warp reductions.
__device__ __forceinline__ uint64_t warp_add_u51(uint64_t x)
{
    const uint64_t lo = __reduce_add_sync(0xFFFFFFFFu, (uint32_t)(x & 0xFFFFFFu));
    const uint64_t hi = __reduce_add_sync(0xFFFFFFFFu, (uint32_t)(x >> 24));
    return lo + (hi << 24);
}

// Arrivals of a grid's blocks in the top 12 bits of a word that may also add up
// a value below 2^52, so that a reader knows the value by itself to be complete.
constexpr int kArrive = 52;
constexpr unsigned long long kValueMask = (1ull << kArrive) - 1;
constexpr int kMaxBlocks = 4000;  // blocks of such a grid at most
#ifndef G5_MEET_NS  // (a test sets its own)
#define G5_MEET_NS (10ull * 1000 * 1000 * 1000)
#endif
constexpr unsigned long long kMeetNs = G5_MEET_NS;

// Polls until each of the K words at p holds the arrivals of every block (grid
// form), their loads issued together; false if a block gave up.  Every wait
// ends: past kMeetNs the block gives up itself.
template <int K>
__device__ __forceinline__ bool await(const unsigned long long *p, unsigned *abort, unsigned long long *value)
{
    const unsigned long long all = gridDim.x;
    unsigned long long t0 = 0;
    uint32_t polls = 0;
    for (;;) {
        unsigned long long x[K];
#pragma unroll
        for (int k = 0; k < K; ++k) x[k] = *(const volatile unsigned long long *)(p + k);
        bool done = true;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            done = done && (x[k] >> kArrive) == all;
            value[k] = x[k] & kValueMask;
        }
        if (done) return true;
        if ((++polls & 255u) == 0) {
            unsigned long long t;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
            if (!t0) t0 = t;
            if (t - t0 > kMeetNs) *(volatile unsigned *)abort = 1;
            if (*(volatile unsigned *)abort) return false;
        }
    }
}

// a > b / c as double arithmetic gives it.  The FP64 units are few and slow
// here, so single precision decides unless the two sides are within its
// rounding (three roundings of 2^-24, far inside the margin).
__device__ __forceinline__ bool above_quotient(uint64_t x, uint64_t y, double c)
{
    const float l = (float)x * (float)c, r = (float)y;
    if (l > r * 1.00001f) return true;
    if (l < r * 0.99999f) return false;
    return (double)x > (double)y / c;
}

// a < b / c, likewise.
__device__ __forceinline__ bool below_quotient(uint64_t x, uint64_t y, double c)
{
    const float l = (float)x * (float)c, r = (float)y;
    if (l < r * 0.99999f) return true;
    if (l > r * 1.00001f) return false;
    return (double)x < (double)y / c;
}

// Work items per warp step of a list of nitems over nw warps: the fewest steps of
// at most 32 items, all warps alike.  (Lists of 2^32 items and more, which no
// graph in 280 GB has, are cut as if they were shorter; 64-bit divisions are a
// call.)
__device__ __forceinline__ uint32_t items_per_step(uint64_t nitems, uint32_t nw)
{
    if (nitems <= nw) return 1u;
    const uint32_t per = (uint32_t)min(nitems, (uint64_t)0xFFFFFFFFu) / nw + 1, steps = (per + 31) / 32;
    return (per + steps - 1) / steps;
}

// Steps of ipw items that a list of nitems makes.
__device__ __forceinline__ uint64_t item_steps(uint64_t nitems, uint32_t ipw)
{
    return nitems >> 32 ? nitems : ((uint32_t)nitems - 1) / ipw + 1;
}
