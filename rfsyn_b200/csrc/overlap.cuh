// overlap.cuh -- kernels of a step overlap their launches.
//
// A small scene's step is a chain of short kernels, and so is the network's
// training step; each link costs the launch and the drain of the kernel before
// it (~2 us on B200).  Inside the step graphs the links are programmatic: a
// kernel's CTAs start once every CTA of the kernel before it has started
// (grid_launch_next, first thing in each kernel) and do what reads no other
// kernel's results; grid_wait then holds them until that kernel has ended and
// its writes are visible.  Every CTA of a kernel that is launched with the link
// passes grid_wait, also one without work, so the kernels' ends keep their
// order.  Kernels launched without it (the network's bias sums and weight
// gradients on streams of their own, its update) stand behind full edges.
//
// A kernel is then resident while the one before it still writes, so nothing
// that a step writes is read through the read-only path (__ldg, const
// __restrict__ loads), whose data must not change while the kernel lives and
// whose loads the compiler may move across grid_wait.
#pragma once
#include <cuda_runtime.h>

namespace rfb {

__device__ __forceinline__ void grid_launch_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Launches a step kernel, with overlap as a programmatic dependent of the
// kernel before it in the stream.
template <typename... P, typename... A>
static inline void launch_step(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, bool overlap,
                               const A &...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = overlap ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace rfb
