// common.cuh -- shared helpers of libpcd_gb300 (sm_103a).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <map>
#include <mutex>
#include <string>
#include <utility>

#include "../../include/pcd.h"

namespace pcd {

// Records the text of the last failure for pcd_last_error().
void set_error(const std::string &msg);
// Counts kernel launches issued by the library (direct launches + graph nodes).
void count_launches(unsigned long long n);

#define PCD_CUDA(call)                                                                     \
    do {                                                                                   \
        cudaError_t e_ = (call);                                                           \
        if (e_ != cudaSuccess) {                                                           \
            cudaGetLastError(); /* reported here, not by the next launch's check */        \
            ::pcd::set_error(std::string(#call) + ": " + cudaGetErrorString(e_) + " (" +    \
                             __FILE__ + ":" + std::to_string(__LINE__) + ")");             \
            return PCD_DEVICE_ERROR;                                                       \
        }                                                                                  \
    } while (0)

#define PCD_TRY(expr)                                                                      \
    do {                                                                                   \
        int s_ = (expr);                                                                   \
        if (s_ != PCD_OK) return s_;                                                       \
    } while (0)

// Checks the launch that just happened on the stream.
#define PCD_LAUNCHED(n)                                                                    \
    do {                                                                                   \
        PCD_CUDA(cudaGetLastError());                                                      \
        ::pcd::count_launches(n);                                                          \
    } while (0)

__device__ __forceinline__ float warp_sum_f(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Max that ignores NaN on the left operand's side the way the reference's
// `if (abs_delta > max_update)` does (solver.cpp:51-53).
__device__ __forceinline__ double nan_skip_max(double m, double v) { return v > m ? v : m; }

__device__ __forceinline__ double warp_max(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = nan_skip_max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

__device__ __forceinline__ double warp_min(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Block-wide reduction of up to 4 doubles (sum/max selectable per slot via
// OPS bits: bit k set = max for slot k).  Result valid in thread 0.
template <int N, unsigned OPS>
__device__ __forceinline__ void block_reduce(double (&v)[N])
{
    __shared__ double sm[32][N];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int nw = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int k = 0; k < N; k++) v[k] = ((OPS >> k) & 1u) ? warp_max(v[k]) : warp_sum(v[k]);
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < N; k++) sm[wid][k] = v[k];
    __syncthreads();
    if (wid == 0) {
#pragma unroll
        for (int k = 0; k < N; k++) {
            // lanes past the last warp hold each slot's identity: 0 for a sum,
            // -inf for a max (so signed maxima come out right as well)
            double x = lane < nw ? sm[lane][k] : (((OPS >> k) & 1u) ? -__longlong_as_double(0x7ff0000000000000ll) : 0.0);
            v[k] = ((OPS >> k) & 1u) ? warp_max(x) : warp_sum(x);
        }
    }
    __syncthreads();
}

// Zeroes device memory before work on any stream can use it: the contexts' streams
// do not wait for the default stream, on which cudaMemset runs, nor does the
// host wait for it.
inline cudaError_t zero_now(void *p, size_t bytes)
{
    const cudaError_t e = cudaMemset(p, 0, bytes);
    return e == cudaSuccess ? cudaStreamSynchronize(cudaStreamLegacy) : e;
}

// Lets fn be launched with all of an SM's shared memory that its static part
// leaves.  The limit belongs to the function, not to a context: set to what one
// plan needs, a smaller plan of another thread's context could lower it between the
// set and the launch, which then failed with an invalid value.
inline cudaError_t allow_shared(const void *fn)
{
    static std::mutex mu;
    static std::map<std::pair<int, const void *>, int> most;  // of the functions met so far
    int dev = 0, bytes = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    {
        std::lock_guard<std::mutex> lk(mu);
        const auto key = std::make_pair(dev, fn);
        auto it = most.find(key);
        if (it == most.end()) {
            cudaFuncAttributes at;
            if ((e = cudaFuncGetAttributes(&at, fn)) != cudaSuccess) return e;
            if ((e = cudaDeviceGetAttribute(&bytes, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) != cudaSuccess)
                return e;
            it = most.emplace(key, bytes - (int)at.sharedSizeBytes).first;
        }
        bytes = it->second;
    }
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

inline int ceil_div(long a, long b) { return (int)((a + b - 1) / b); }

}  // namespace pcd
