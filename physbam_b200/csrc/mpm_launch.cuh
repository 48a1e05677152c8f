// Launches of a substep's chain of kernels, and reductions to one host value.
#pragma once
#include <cuda_runtime.h>

namespace mpm {

// Programmatic dependent launch: a kernel launched by launch_chained may be set up,
// and its CTAs take freed SM resources, while the last CTAs of the kernel before it
// in the stream still run.  Every chained kernel begins with chain_begin(), which
// returns once the kernel before it has completed and its writes are visible; it
// reads and writes no global memory before that.  Per call, captured graphs: 2D
// block 2.21 -> 2.05 ms, 32^3 box 2.32 -> 2.29, an adaptive frame 2.92 -> 2.78 (its
// substeps run eagerly), spheres 4.85 -> 4.82.  No trigger of its own lets the next
// kernel come up earlier: with one at the kernels' start the waiting CTAs cost the
// 32^3 box 8 % (2.52 ms) and gained the spheres 1 %.
__device__ __forceinline__ void chain_begin() { cudaGridDependencySynchronize(); }

template<class... P, class... A>
inline void launch_chained(void (*kernel)(P...), unsigned grid, unsigned threads, size_t smem, cudaStream_t stream, A&&... args)
{
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, P(args)...);   // errors: MPM_LAUNCHED reads them
}

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
