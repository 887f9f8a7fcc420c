// Instances and launchers of the warp-tile FP64 apply (apply_warp.cuh).
#include "apply_warp.cuh"
#include "warp_plan.hpp"
#include "dispatch.hpp"

#include "../../../include/tandem_b200.h"

namespace tdg {

namespace {

template <class S, bool TG>
int launch_facets(int nq, WarpGeo const& wg, const double* x, double* y, int nrhs, int64_t ld, cudaStream_t s,
                  int ctas, bool early, int most, size_t tab, size_t per_warp) {
    static PerDevice ready;
    auto kern = facew_kernel<S, TG>;
    if (int rc = allow_shared(kern, ready)) return rc;
    const int64_t nwork = static_cast<int64_t>(wg.nftiles) * nrhs;
    Plan p = make_plan(most, nwork, WarpBlocks(nq).count(), 2 * S::Q * warp_facet_frags<S>(nq), kSplit64, ctas);
    p.split.whole = std::min(p.split.whole, nwork);
    return launch_facet_kernel(early, kern, p.grid, 32 * p.warps, tab + p.warps * per_warp, s, nq, wg, p.split, x, y, ld,
                               nrhs);
}

template <class S>
int run_facets(int nq, WarpGeo const& wg, const double* x, double* y, int nrhs, int64_t ld, cudaStream_t s, int ctas,
               bool early) {
    using L = WarpTile<S>;
    if (wg.nftiles == 0) return 0;
    const size_t limit = shared_limit();
    const size_t tab = sizeof(double) * 32 * static_cast<size_t>(wg.face_tables) * warp_facet_frags<S>(nq);
    const size_t per_warp = sizeof(double) * facet_warp_doubles<S>(nq);
    if (per_warp > limit) return TDG_E_INVALID;
    const bool fits = tab + 4 * per_warp <= limit;
    const int most = static_cast<int>(std::min<size_t>(L::FWARPS, (limit - (fits ? tab : 0)) / per_warp));
    if (fits) return launch_facets<S, false>(nq, wg, x, y, nrhs, ld, s, ctas, early, most, tab, per_warp);
    return launch_facets<S, true>(nq, wg, x, y, nrhs, ld, s, ctas, early, most, 0, per_warp);
}

template <class S, bool TG>
int launch_volume(int64_t E, int Nq, WarpGeo const& wg, const double* x, double* y, int nrhs, int64_t ld,
                  cudaStream_t s, int ctas, int most, size_t tab, size_t per_warp) {
    static PerDevice ready;
    auto kern = volw_kernel<S, TG>;
    if (int rc = allow_shared(kern, ready)) return rc;
    const int64_t nwork = (E + 7) / 8 * nrhs;
    const Plan p = make_plan(most, nwork, WarpBlocks(Nq).count(), S::Q * warp_volume_frags<S>(Nq), kSplit64, ctas);
    const size_t smem = tab + (p.split.whole < nwork ? p.warps * per_warp : 0);
    kern<<<p.grid, 32 * p.warps, smem, s>>>(E, Nq, wg, p.split, x, y, ld, nrhs);
    return cudaGetLastError() == cudaSuccess ? 0 : TDG_E_CUDA;
}

template <class S>
int run_volume(int64_t E, int Nq, WarpGeo const& wg, const double* x, double* y, int nrhs, int64_t ld, cudaStream_t s,
               int ctas) {
    using L = WarpTile<S>;
    const size_t limit = shared_limit();
    const size_t tab = sizeof(double) * 32 * static_cast<size_t>(warp_volume_frags<S>(Nq));
    const size_t per_warp = sizeof(double) * volume_warp_doubles<S>();
    if (tab + 4 * per_warp <= limit) {
        const int most = static_cast<int>(std::min<size_t>(L::VWARPS, (limit - tab) / per_warp));
        return launch_volume<S, false>(E, Nq, wg, x, y, nrhs, ld, s, ctas, most, tab, per_warp);
    }
    return launch_volume<S, true>(E, Nq, wg, x, y, nrhs, ld, s, ctas, L::VWARPS, 0, per_warp);
}

template <int D, int N>
int volume_kind(int kind, int64_t E, int Nq, WarpGeo const& wg, const double* x, double* y, int nrhs, int64_t ld,
                cudaStream_t s, int ctas) {
    if (kind == kPoisson) return run_volume<Shape<D, N, kPoisson>>(E, Nq, wg, x, y, nrhs, ld, s, ctas);
    return run_volume<Shape<D, N, kElasticity>>(E, Nq, wg, x, y, nrhs, ld, s, ctas);
}

template <int D>
int volume_deg(int N, int kind, int64_t E, int Nq, WarpGeo const& wg, const double* x, double* y, int nrhs, int64_t ld,
               cudaStream_t s, int ctas) {
    switch (N) {
        case 1: return volume_kind<D, 1>(kind, E, Nq, wg, x, y, nrhs, ld, s, ctas);
        case 2: return volume_kind<D, 2>(kind, E, Nq, wg, x, y, nrhs, ld, s, ctas);
        case 3: return volume_kind<D, 3>(kind, E, Nq, wg, x, y, nrhs, ld, s, ctas);
        case 4: return volume_kind<D, 4>(kind, E, Nq, wg, x, y, nrhs, ld, s, ctas);
        default: return TDG_E_INVALID;
    }
}

template <int D, int N>
int facets_kind(int kind, int nq, WarpGeo const& wg, const double* x, double* y, int nrhs, int64_t ld, cudaStream_t s,
                int ctas, bool early) {
    if (kind == kPoisson) return run_facets<Shape<D, N, kPoisson>>(nq, wg, x, y, nrhs, ld, s, ctas, early);
    return run_facets<Shape<D, N, kElasticity>>(nq, wg, x, y, nrhs, ld, s, ctas, early);
}

template <int D>
int facets_deg(int N, int kind, int nq, WarpGeo const& wg, const double* x, double* y, int nrhs, int64_t ld,
               cudaStream_t s, int ctas, bool early) {
    switch (N) {
        case 1: return facets_kind<D, 1>(kind, nq, wg, x, y, nrhs, ld, s, ctas, early);
        case 2: return facets_kind<D, 2>(kind, nq, wg, x, y, nrhs, ld, s, ctas, early);
        case 3: return facets_kind<D, 3>(kind, nq, wg, x, y, nrhs, ld, s, ctas, early);
        case 4: return facets_kind<D, 4>(kind, nq, wg, x, y, nrhs, ld, s, ctas, early);
        default: return TDG_E_INVALID;
    }
}

}  // namespace

int launch_facets_warp(int D, int N, int kind, int nq, WarpGeo const& wg, const double* x, double* y, int nrhs,
                       int64_t ld, cudaStream_t s, int ctas, bool early) {
    if (nrhs < 1 || (wg.nftiles > 0 && (!wg.ftab || !wg.fct))) return TDG_E_INVALID;
    if (D == 2) return facets_deg<2>(N, kind, nq, wg, x, y, nrhs, ld, s, ctas, early);
    if (D == 3) return facets_deg<3>(N, kind, nq, wg, x, y, nrhs, ld, s, ctas, early);
    return TDG_E_INVALID;
}

int launch_volume_warp(int D, int N, int kind, int64_t E, int Nq, WarpGeo const& wg, const double* x, double* y,
                       int nrhs, int64_t ld, cudaStream_t s, int ctas) {
    if (nrhs < 1 || !wg.vtab || !wg.vol) return TDG_E_INVALID;
    if (D == 2) return volume_deg<2>(N, kind, E, Nq, wg, x, y, nrhs, ld, s, ctas);
    if (D == 3) return volume_deg<3>(N, kind, E, Nq, wg, x, y, nrhs, ld, s, ctas);
    return TDG_E_INVALID;
}

}  // namespace tdg
