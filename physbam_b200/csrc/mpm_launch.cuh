// Reductions to one host value.
#pragma once
#include <cuda_runtime.h>

namespace mpm {

// Maximum over a grid of at most 1024 threads per CTA of a non-negative value per
// thread, to *host (pinned memory; the host reads it after a synchronize).
// state: two zeroed words, the maximum's bits so far and the finished CTAs; the CTA
// that finishes last hands the value over and zeroes them again.
__device__ __forceinline__ void grid_max(double v, unsigned long long* state, double* host)
{
    __shared__ double sh[32];
#pragma unroll
    for(int o = 16; o; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    if((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    if(threadIdx.x) return;
    for(unsigned w = 1; w < blockDim.x >> 5; w++) v = fmax(v, sh[w]);
    atomicMax(state, (unsigned long long)__double_as_longlong(v));
    __threadfence();
    if(atomicAdd(state + 1, 1ull) != gridDim.x - 1) return;
    __threadfence();
    *host = __longlong_as_double((long long)atomicExch(state, 0ull));
    state[1] = 0ull;
}

}  // namespace mpm
