// Kernels that start before the one in front of them on the stream is done (programmatic dependent
// launch).  The front kernel calls let_next_kernel_start(); the one behind, launched with
// launch_early, has its CTAs on the SMs when the front one ends and waits in
// wait_for_previous_kernel() until all of its writes are visible.  A chain stays in order because
// every warp that works waits: the vector kernels first of all, the facet kernel before it touches
// y.  What the facet kernel reads before that (x, geometry) the volume kernel in front of it does
// not write, and that one is launched plainly, so whatever wrote x is done when it starts.  Both
// calls do nothing in a plain launch.
#pragma once

#include <cuda_runtime.h>

namespace tdg {

__device__ __forceinline__ void let_next_kernel_start() { asm volatile("griddepcontrol.launch_dependents;\n" ::); }
__device__ __forceinline__ void wait_for_previous_kernel() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

// early false: a plain launch.
template <class... P, class... A>
bool launch_programmatic(bool early, void (*kern)(P...), dim3 grid, int threads, size_t smem, cudaStream_t s,
                         A... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = dim3(threads);
    c.dynamicSmemBytes = smem;
    c.stream = s;
    c.attrs = &at;
    c.numAttrs = early ? 1 : 0;
    return cudaLaunchKernelEx(&c, kern, static_cast<P>(args)...) == cudaSuccess;
}

// The short solver kernels, whose launches into a stream capture are plain: with an edge at every kernel of
// a CG iteration the edges cost more than they hide (block-Jacobi CG at 2D p4 Poisson, 8,192 triangles,
// replayed in blocks of 8 iterations: 71.7 ms with them, 65.3 without).
template <class... P, class... A>
bool launch_early(bool early, void (*kern)(P...), dim3 grid, int threads, size_t smem, cudaStream_t s, A... args) {
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    early = early && cudaStreamIsCapturing(s, &capture) == cudaSuccess && capture == cudaStreamCaptureStatusNone;
    return launch_programmatic(early, kern, grid, threads, smem, s, args...);
}

}  // namespace tdg
