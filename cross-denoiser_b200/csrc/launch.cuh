// Programmatic dependent launch: a kernel that follows another of the chain
// on its stream is launched before that one has ended, so its launch and its
// prologue (barriers, shared-memory tables) run under the other's last CTAs.
//
// Rules, for every kernel launched with launch_chained():
//   * chain_wait() comes before its first access to global memory, read or
//     write: it returns once the kernel before it has completed and its
//     writes are visible (that kernel's own chain_wait orders the ones before);
//   * its inputs are read with plain loads through pointers without
//     __restrict__ (or by cp.async, bulk and TMA copies): it is resident while
//     its predecessor writes them, so they are not read-only for its lifetime,
//     as __ldg and the loads that the compiler may make of const __restrict__
//     pointers require; and such loads, which memory is held never to change
//     under, are not tied down by chain_wait()'s clobber.  __restrict__ stays
//     on pointers that a kernel only writes;
//   * chain_next() lets the next kernel's CTAs start; a kernel that allocates
//     TMEM does so after chain_wait() and calls chain_next() after the
//     allocation, so no waiting CTA ever holds TMEM that an earlier kernel's
//     CTA still has to allocate.  Where a grid is about one wave it is left
//     out: the next kernel's CTAs then start as this one's end, not in the
//     slots that the wave leaves free (temporal.cu).
// A kernel launched any other way after one of these starts when it has
// ended, as always.  On the U-Net's 14 forward and 15 chained backward
// kernels (the nine weight gradients are launched plainly): prediction at
// 1920x1080 315 -> 295 us, a training pass at 2560x1440 1498 -> 1447 us, a
// whole 256x256 training step 455 -> 427 us.
#pragma once
#include <utility>
#include <cuda_runtime.h>

namespace cd {

__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... P, typename... A>
cudaError_t launch_chained(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A &&...args)
{
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...);
    const cudaError_t last = cudaGetLastError();
    return e != cudaSuccess ? e : last;
}

}  // namespace cd
