// Instances and launchers of the block-Jacobi kernels.
#include "bjacobi.cuh"
#include "dispatch.hpp"
#include "per_device.hpp"

#include "../../../include/tandem_b200.h"

#include <algorithm>
#include <type_traits>

namespace tdg {

namespace {

template <class S>
int run_assemble(DevOp<double> const& op, double* blk, cudaStream_t s) {
    const size_t smem = sizeof(double) * static_cast<size_t>(bjac_assemble_smem_doubles<S>(op.Nq, op.nq));
    auto kern = bjac_assemble_kernel<S>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) !=
        cudaSuccess)
        return TDG_E_CUDA;
    if (op.E > 0x7fffffff) return TDG_E_INVALID;
    kern<<<static_cast<unsigned>(op.E), 256, smem, s>>>(op, blk);
    return cudaGetLastError() == cudaSuccess ? 0 : TDG_E_CUDA;
}

template <int D, int N>
int assemble_kind(int kind, DevOp<double> const& op, double* blk, cudaStream_t s) {
    if (kind == kPoisson) return run_assemble<Shape<D, N, kPoisson>>(op, blk, s);
    return run_assemble<Shape<D, N, kElasticity>>(op, blk, s);
}

template <int D>
int assemble_deg(int N, int kind, DevOp<double> const& op, double* blk, cudaStream_t s) {
    switch (N) {
        case 1: return assemble_kind<D, 1>(kind, op, blk, s);
        case 2: return assemble_kind<D, 2>(kind, op, blk, s);
        case 3: return assemble_kind<D, 3>(kind, op, blk, s);
        case 4: return assemble_kind<D, 4>(kind, op, blk, s);
        default: return TDG_E_INVALID;
    }
}

template <int BS, typename T>
int run_invert(int64_t E, const double* blk, T* inv, int* status, cudaStream_t s) {
    const size_t smem = sizeof(double) * (static_cast<size_t>(BS) * BS + BS);
    auto kern = bjac_invert_kernel<BS, T>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) !=
        cudaSuccess)
        return TDG_E_CUDA;
    if (E > 0x7fffffff) return TDG_E_INVALID;
    kern<<<static_cast<unsigned>(E), 256, smem, s>>>(blk, inv, status);
    return cudaGetLastError() == cudaSuccess ? 0 : TDG_E_CUDA;
}

template <int BS, typename TM, typename TV, int RB>
int run_rows(int64_t E, const TM* inv, const TV* r, TV* z, int nrhs, int64_t ld, cudaStream_t s) {
    constexpr int TE = (256 / BS) > 0 ? (256 / BS) : 1;
    const int64_t ntiles = (E + TE - 1) / TE;
    int64_t grid = static_cast<int64_t>(device_sm_count()) * 8;
    if (grid > ntiles) grid = ntiles;
    if (grid < 1) grid = 1;
    dim3 g(static_cast<unsigned>(grid), static_cast<unsigned>((nrhs + RB - 1) / RB));
    launch_early(true, bjac_apply_kernel<BS, TM, TV, RB>, g, 256, 0, s, E, inv, r, z, nrhs, ld);
    return cudaGetLastError() == cudaSuccess ? 0 : TDG_E_CUDA;
}

template <int BS, typename TM, typename TV>
int run_stream(int64_t E, const TM* inv, const TV* r, TV* z, cudaStream_t s) {
    using L = BjacStream<BS, TM>;
    constexpr size_t smem = L::smem(sizeof(TV));
    auto kern = bjac_stream_kernel<BS, TM, TV>;
    static PerDevice resident;
    const int per_sm = resident.get([&] {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) !=
            cudaSuccess)
            return 0;
        int n = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, 256, smem) != cudaSuccess || n < 1) n = 1;
        return n;
    });
    if (per_sm < 1) return TDG_E_CUDA;
    const int64_t pairs = ((E + L::TE - 1) / L::TE + 1) / 2;  // two teams per CTA
    int64_t grid = static_cast<int64_t>(device_sm_count()) * per_sm;
    if (grid > pairs) grid = pairs;
    kern<<<static_cast<unsigned>(grid), 256, smem, s>>>(E, inv, r, z);
    return cudaGetLastError() == cudaSuccess ? 0 : TDG_E_CUDA;
}

// Inverses up to this size stay in L2 and a row's second access costs nothing: 8,192 blocks of 15
// (7.9 MB) 3.98 us by rows, 4.27 us streamed; 10,368 blocks of 105 (462 MB) 172 and 84 us.
constexpr int64_t kStreamBytes = int64_t(32) << 20;

// Rows, as few groups of up to five columns as they fill, evenly.
template <int BS, typename TM, typename TV>
int run_row_groups(int64_t E, const TM* inv, const TV* r, TV* z, int nrhs, int64_t ld, cudaStream_t s) {
    const int groups = (nrhs + 4) / 5;
    switch ((nrhs + groups - 1) / groups) {
        case 1: return run_rows<BS, TM, TV, 1>(E, inv, r, z, nrhs, ld, s);
        case 2: return run_rows<BS, TM, TV, 2>(E, inv, r, z, nrhs, ld, s);
        case 3: return run_rows<BS, TM, TV, 3>(E, inv, r, z, nrhs, ld, s);
        case 4: return run_rows<BS, TM, TV, 4>(E, inv, r, z, nrhs, ld, s);
        default: return run_rows<BS, TM, TV, 5>(E, inv, r, z, nrhs, ld, s);
    }
}

// One right-hand side: bound by the inverses, streamed.  Several: by rows, each column apart, while all of
// them fit beside each other (a CTA and column per quarter of an SM); else on the tensor pipe (FP64
// vectors, blocks from 10: below, a fragment is mostly padding), where eight columns cost what one
// does: from five columns on, or from two where four warps share an element.  The conversions of FP32
// inverses weigh on the tensor form, so above 16 they take rows up to five columns, the 105 x 105
// ones too.  us, by rows / tensor pipe: 35 x 35, 6,000 elements, 2 columns 11.6 / 23.0, 4 19.1 / 23.1, 8 31.4 /
// 24.0, FP32 inverses 5 18.9 / 25.0; 105 x 105, 6,000 elements, 2 columns 116 / 94 (FP32 inverses 89 / 152),
// 8 257 / 112; 30 x 30, 48 elements, 8 columns 4.8 / 6.5.
template <int BS, typename TM, typename TV>
int run_bapply(int64_t E, const TM* inv, const TV* r, TV* z, int nrhs, int64_t ld, cudaStream_t s) {
    if (nrhs == 1 && E * bjac_packed_size(BS) * static_cast<int64_t>(sizeof(TM)) >= kStreamBytes)
        return run_stream<BS, TM, TV>(E, inv, r, z, s);
    if constexpr (std::is_same_v<TV, double> && BS >= 10) {
        constexpr int cols = 8 * bjac_mma_tiles<BS>(), epc = 4 / bjac_mma_warps<BS>();
        constexpr bool one = bjac_mma_warps<BS>() == 1, f32 = sizeof(TM) == 4;
        constexpr int few = f32 && BS > 16 && (one || BS > 60) ? 5 : (one ? 4 : 1);  // columns taken by rows
        constexpr int te = 256 / BS;
        const bool beside = few > 1 && (E + te - 1) / te * nrhs <= 4 * static_cast<int64_t>(device_sm_count());
        if (nrhs > few && !beside) {
            const int64_t grid = std::min<int64_t>((E + epc - 1) / epc, static_cast<int64_t>(device_sm_count()) * 16);
            dim3 g(static_cast<unsigned>(grid), static_cast<unsigned>((nrhs + cols - 1) / cols));
            bjac_mma_kernel<BS, TM><<<g, 128, 0, s>>>(E, inv, r, z, nrhs, ld);
            return cudaGetLastError() == cudaSuccess ? 0 : TDG_E_CUDA;
        }
        if (beside) return run_rows<BS, TM, TV, 1>(E, inv, r, z, nrhs, ld, s);
    } else {
        constexpr int te = 256 / BS;
        if ((E + te - 1) / te * nrhs <= 4 * static_cast<int64_t>(device_sm_count()))
            return run_rows<BS, TM, TV, 1>(E, inv, r, z, nrhs, ld, s);
    }
    return run_row_groups<BS, TM, TV>(E, inv, r, z, nrhs, ld, s);
}

// Block sizes bs = binom(N + D, D) * Q for D in {2, 3}, N in [1, 4], Q in {1, D}.
#define TDG_FOR_EACH_BS(X) \
    X(1) X(2) X(3) X(4) X(6) X(10) X(12) X(15) X(20) X(30) X(35) X(60) X(105)

}  // namespace

int launch_bjac_assemble(int D, int N, int kind, DevOp<double> const& op, double* blk, cudaStream_t s) {
    if (D == 2) return assemble_deg<2>(N, kind, op, blk, s);
    if (D == 3) return assemble_deg<3>(N, kind, op, blk, s);
    return TDG_E_INVALID;
}

template <typename T>
int launch_bjac_invert(int bs, int64_t E, const double* blk, T* inv, int* status, cudaStream_t s) {
    switch (bs) {
#define TDG_CASE(B) \
    case B: return run_invert<B, T>(E, blk, inv, status, s);
        TDG_FOR_EACH_BS(TDG_CASE)
#undef TDG_CASE
        default: return TDG_E_INVALID;
    }
}

template <typename TM, typename TV>
int launch_bjac_apply(int bs, int64_t E, const TM* inv, const TV* r, TV* z, int nrhs, int64_t ld,
                      cudaStream_t s) {
    switch (bs) {
#define TDG_CASE(B) \
    case B: return run_bapply<B, TM, TV>(E, inv, r, z, nrhs, ld, s);
        TDG_FOR_EACH_BS(TDG_CASE)
#undef TDG_CASE
        default: return TDG_E_INVALID;
    }
}

template int launch_bjac_invert<double>(int, int64_t, const double*, double*, int*, cudaStream_t);
template int launch_bjac_invert<float>(int, int64_t, const double*, float*, int*, cudaStream_t);
template int launch_bjac_apply<double, double>(int, int64_t, const double*, const double*, double*, int, int64_t,
                                               cudaStream_t);
template int launch_bjac_apply<float, float>(int, int64_t, const float*, const float*, float*, int, int64_t,
                                             cudaStream_t);
template int launch_bjac_apply<float, double>(int, int64_t, const float*, const double*, double*, int, int64_t,
                                              cudaStream_t);

}  // namespace tdg
