// coop.cuh -- cooperative launches and the bounded grid barrier of their kernels.
#pragma once
#include <algorithm>

#include "mgm_internal.cuh"

namespace mgm {

#ifndef MGM_BARRIER_POLLS
#define MGM_BARRIER_POLLS (1L << 20)
#endif

// Grid barrier of a cooperative launch (all CTAs resident): thread 0 of each
// CTA arrives on a counter; the last arrival resets it and advances the
// generation the others wait on (polled without sleeping: the wait is a few
// microseconds).  The wait is bounded (MGM_BARRIER_POLLS of L2, under a second);
// when it runs out the CTA records the error and the kernel's CTAs
// return at their next barrier.  Returns false once any CTA has given up.
__device__ __forceinline__ bool grid_barrier(unsigned *bar, int *err, unsigned &gen)
{
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        int good = 1;
        __threadfence();
        const unsigned arrived = atomicAdd(&bar[0], 1u) + 1u;
        if (arrived == gridDim.x) {
            atomicExch(&bar[0], 0u);
            __threadfence();
            atomicAdd(&bar[1], 1u);
        } else {
            long spins = 0;
            while (*(volatile unsigned *)&bar[1] == gen) {
                if (++spins > MGM_BARRIER_POLLS || ((spins & 255) == 0 && *(volatile int *)err)) {
                    atomicExch(err, 1);
                    good = 0;
                    break;
                }
            }
        }
        __threadfence();
        gen++;
        ok = good && *(volatile int *)err == 0;
    }
    __syncthreads();
    return ok != 0;
}

// CTAs of that size that the device (as much of it as the process may use)
// holds at once: the most a cooperative launch may have
template <class... P>
inline int cooperative_ctas(void (*kern)(P...), int block, size_t smem)
{
    int dev = 0, sms = 0, per_sm = 0;
    MGM_CUDA(cudaGetDevice(&dev));
    MGM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    MGM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, block, smem));
    return std::max(1, sms * per_sm);
}

template <class... P, class... A>
inline cudaError_t launch_cooperative(void (*kern)(P...), int grid, int block, size_t smem, cudaStream_t s, A... args)
{
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}

// after the launch: the error flag that its barriers set
inline void check_barrier(int err, const char *what)
{
    if (err != 0) throw Error{4 /* MGM_ERR_TIMEOUT */, std::string(what) + ": a grid barrier's wait ran out"};
}

}  // namespace mgm
