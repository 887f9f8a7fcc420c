// Instances and launcher of the FP64 volume kernel in passes (apply_face2.cuh).
#include "apply_face2.cuh"
#include "dispatch.hpp"

#include "../../../include/tandem_b200.h"

namespace tdg {

namespace {

template <class S>
int run_vol2(int64_t E, int Nq, const double* tables, WarpGeo const& wg, const double* x, double* y, int nrhs,
             int64_t ld, cudaStream_t s, int ctas, int qc) {
    using L = MmaTile<S>;
    const Vol2Layout<S> vl = vol2_layout<S>(Nq, qc < Nq ? qc : Nq);
    const size_t smem = sizeof(double) * static_cast<size_t>(vl.total);
    auto kern = vol2_kernel<S>;
    static size_t configured = 0;  // dynamic shared memory (grows)
    static int per_sm = 1;
    if (configured < smem) {
        int dev = 0, optin = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        if (smem + 1024 > static_cast<size_t>(optin)) return TDG_E_INVALID;
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) !=
            cudaSuccess)
            return TDG_E_CUDA;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, L::NT, smem) != cudaSuccess || per_sm < 1)
            per_sm = 1;
        configured = smem;
    }
    const int64_t work = (E + L::TE - 1) / L::TE * nrhs;
    int64_t grid = static_cast<int64_t>(device_sm_count()) * ((ctas > 0 && ctas < per_sm) ? ctas : per_sm);
    if (grid > work) grid = work;
    kern<<<static_cast<unsigned>(grid), L::NT, smem, s>>>(E, Nq, wg, tables, x, y, ld, nrhs, vl.qc);
    return cudaGetLastError() == cudaSuccess ? 0 : TDG_E_CUDA;
}

template <int D, int N>
int vol2_kind(int kind, int64_t E, int Nq, const double* tables, WarpGeo const& wg, const double* x, double* y,
              int nrhs, int64_t ld, cudaStream_t s, int ctas, int qc) {
    if (kind == kPoisson) return run_vol2<Shape<D, N, kPoisson>>(E, Nq, tables, wg, x, y, nrhs, ld, s, ctas, qc);
    return run_vol2<Shape<D, N, kElasticity>>(E, Nq, tables, wg, x, y, nrhs, ld, s, ctas, qc);
}

template <int D>
int vol2_deg(int N, int kind, int64_t E, int Nq, const double* tables, WarpGeo const& wg, const double* x, double* y,
             int nrhs, int64_t ld, cudaStream_t s, int ctas, int qc) {
    switch (N) {
        case 1: return vol2_kind<D, 1>(kind, E, Nq, tables, wg, x, y, nrhs, ld, s, ctas, qc);
        case 2: return vol2_kind<D, 2>(kind, E, Nq, tables, wg, x, y, nrhs, ld, s, ctas, qc);
        case 3: return vol2_kind<D, 3>(kind, E, Nq, tables, wg, x, y, nrhs, ld, s, ctas, qc);
        case 4: return vol2_kind<D, 4>(kind, E, Nq, tables, wg, x, y, nrhs, ld, s, ctas, qc);
        default: return TDG_E_INVALID;
    }
}

}  // namespace

int launch_vol2(int D, int N, int kind, int64_t E, int Nq, const double* tables, WarpGeo const& wg, const double* x,
                double* y, int nrhs, int64_t ld, cudaStream_t s, int ctas, int qc) {
    if (nrhs < 1 || !tables || !wg.vol || qc <= 0 || qc % face2_pass_step(D) != 0) return TDG_E_INVALID;
    if (D == 2) return vol2_deg<2>(N, kind, E, Nq, tables, wg, x, y, nrhs, ld, s, ctas, qc);
    if (D == 3) return vol2_deg<3>(N, kind, E, Nq, tables, wg, x, y, nrhs, ld, s, ctas, qc);
    return TDG_E_INVALID;
}

}  // namespace tdg
