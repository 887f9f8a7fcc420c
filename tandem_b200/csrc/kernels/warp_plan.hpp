// Launch shapes of the warp-tile kernels (apply_warp.cuh, apply_warp32.cuh).
#pragma once

#include "apply_warp.cuh"
#include "dispatch.hpp"
#include "early.cuh"
#include "per_device.hpp"

#include "../../../include/tandem_b200.h"

#include <algorithm>
#include <cuda_runtime.h>

namespace tdg {

// Dynamic shared memory a CTA may take beside the kernels' static arrays.
inline size_t shared_limit() {
    static PerDevice limit;
    const int v = limit.get([] {
        int dev = 0, optin = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        return optin - 2048;
    });
    return v > 0 ? static_cast<size_t>(v) : size_t(0);
}

// Grid, warps per CTA (one persistent CTA per SM) and split of `nwork` items of `nblk` blocks each.
struct Plan {
    int grid, warps;
    WarpSplit split;
};
// most: warps the launch bound and shared memory allow; ctas: the caller's limit (4 warps each, 0
// none); mma: products of an item; least: the smallest item worth splitting.  A last round that fills less than 85 % of the warps is split (a
// whole-item round of 8 warps then costs about as much as its split form: 41 k clocks at 3D p4
// elasticity).  Items of fewer
// products than `least` stay whole: their time is the latency of their loads, which every part would
// pay again.  FP64: 256 (4 k clocks of its pipe; no shape between 128 and 256 gained).  FP32, with
// three products and two splits each: 128 (one tile per SM, 3D p4 Poisson, 162 tetrahedra: 25.1 us
// whole, 17.1 split; 3D p2 elasticity volume, 78 products: 5.0 whole, 6.5 split).
constexpr int kSplit64 = 256, kSplit32 = 128;
inline Plan make_plan(int most, int64_t nwork, int nblk, int mma, int least, int ctas) {
    const int sms = device_sm_count();
    Plan p;
    if (ctas > 0) most = std::min(most, 4 * ctas);
    if (mma < least) nblk = 1;
    const int64_t share = (nwork + sms - 1) / sms;  // items per SM
    p.warps = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(most, share * nblk)));
    p.grid = static_cast<int>(std::min<int64_t>(sms, nwork));
    const int64_t all = static_cast<int64_t>(p.grid) * p.warps, rest = nwork % all;
    p.split.whole = nwork - rest;
    p.split.parts = std::min(nblk, p.warps);
    if (rest * 100 >= all * 85 || p.split.parts == 1) p.split.whole = nwork + (rest ? all - rest : 0);
    return p;
}

// Launches a facet kernel behind the volume kernel of the same apply: `early` lets its CTAs start where
// that kernel leaves an SM's shared memory and registers, before its last CTA is done.  Only behind a
// kernel of which this one reads nothing before its wait.  Small meshes are a chain of latencies
// (launch, tables, coefficients, geometry, products), which the two kernels then share; large ones
// fill the tail of the volume kernel.  FP64 apply without / with it, us: 3D p4 elasticity 162 tetrahedra
// 23.1 / 14.3, 48,000 368 / 364; 3D p2 elasticity 7,986 29.7 / 26.3; 3D p3 Poisson 13,182 34.8 / 31.8;
// 2D p4 elasticity, 19,886 triangles in a batch 29.8 / 28.1.  Under capture too, per apply of a replayed
// chain: 3D p2 elasticity, 162 tetrahedra 14.1 / 9.6, p4 21.8 / 14.7; 2D p4 Poisson, 8,192 triangles 9.3 / 8.4;
// block-Jacobi CG in replayed blocks, 3D p2 elasticity, 162 tetrahedra 11.8 / 10.1 ms, p4 29.6 / 25.0.
template <class... P, class... A>
int launch_facet_kernel(bool early, void (*kern)(P...), int grid, int threads, size_t smem, cudaStream_t s, A... args) {
    return launch_programmatic(early, kern, dim3(grid), threads, smem, s, args...) ? 0 : TDG_E_CUDA;
}

template <class K>
int allow_shared(K kern, PerDevice& ready) {
    const int ok = ready.get([&] {
        return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(shared_limit())) ==
               cudaSuccess;
    });
    return ok > 0 ? 0 : TDG_E_CUDA;
}

}  // namespace tdg
