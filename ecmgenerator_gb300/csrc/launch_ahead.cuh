/*
 * launch_ahead.cuh -- kernels that follow one another on a stream without an
 * event between them are launched ahead: the next kernel's blocks come in as
 * the blocks of the one before end, and wait for its writes before they touch
 * memory (programmatic launch).  What it saves is a launch's latency between
 * short kernels: kNN of 3,000 agents 29.2 -> 26.8 us, of a million 243 -> 237,
 * the kd-tree tick of 250,000 1,124 -> 1,109.  Let in earlier, from the first
 * instruction of the kernel before, the chain of the kd-tree's 90 kernels
 * filled the SMs with waiting blocks (1,201 us of device time against 1,089);
 * the others did not care.
 *
 * Every block of such a kernel calls wait_for_previous() before its first
 * access, so that the end of a kernel implies the end of all before it; and
 * what the kernel before writes is not read through const __restrict__
 * pointers, whose loads the compiler may move above the wait.
 */
#ifndef ECMG_LAUNCH_AHEAD_CUH
#define ECMG_LAUNCH_AHEAD_CUH

#include <cuda_runtime.h>

namespace ecmg {

__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... P, class... A>
static cudaError_t launch_ahead(void (*kern)(P...), int blocks, int threads, size_t smem, cudaStream_t s, A... args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, P(args)...);
}

}  // namespace ecmg

#endif
