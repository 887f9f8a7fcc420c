// Launchers of the warp-tile FP32 kernels (apply_warp32.cuh) for one vector type and pass count; a
// source file per pair instantiates them (each takes minutes to compile).
#pragma once

#include "apply_warp32.cuh"
#include "warp_plan.hpp"

namespace tdg {

namespace {

template <class S, typename TX, int NP, bool TG>
int go_facets(int nq, WarpGeo32 const& wg, const TX* x, TX* y, int nrhs, int64_t ld, cudaStream_t s, int ctas, bool early,
              int most, size_t tab, size_t per_warp) {
    static PerDevice ready;
    auto kern = facew32_kernel<S, TX, NP, TG>;
    if (int rc = allow_shared(kern, ready)) return rc;
    const int64_t nwork = static_cast<int64_t>(wg.nftiles) * nrhs;
    Plan p = make_plan(most, nwork, WarpBlocks(nq).count(), 2 * S::Q * warp32_facet_frags<S>(nq), kSplit32, ctas);
    p.split.whole = std::min(p.split.whole, nwork);
    return launch_facet_kernel(early, kern, p.grid, 32 * p.warps, tab + p.warps * per_warp, s, nq, wg, p.split, x, y, ld,
                               nrhs);
}

template <class S, typename TX, int NP>
int run_facets32(int nq, WarpGeo32 const& wg, const TX* x, TX* y, int nrhs, int64_t ld, cudaStream_t s, int ctas,
                 bool early) {
    using L = WarpTile32<S>;
    if (wg.nftiles == 0) return 0;
    const size_t limit = shared_limit();
    const size_t tab = sizeof(float) * 64 * static_cast<size_t>(wg.face_tables) * warp32_facet_frags<S>(nq);
    const size_t per_warp = sizeof(float) * facet32_warp_floats<S>(nq);
    if (per_warp > limit) return TDG_E_INVALID;
    const bool fits = tab + 4 * per_warp <= limit;
    const int most = static_cast<int>(std::min<size_t>(L::WARPS, (limit - (fits ? tab : 0)) / per_warp));
    if (fits) return go_facets<S, TX, NP, false>(nq, wg, x, y, nrhs, ld, s, ctas, early, most, tab, per_warp);
    return go_facets<S, TX, NP, true>(nq, wg, x, y, nrhs, ld, s, ctas, early, most, 0, per_warp);
}

template <class S, typename TX, int NP, bool TG>
int go_volume(int64_t E, int Nq, WarpGeo32 const& wg, const TX* x, TX* y, int nrhs, int64_t ld, cudaStream_t s,
              int ctas, int most, size_t tab, size_t per_warp) {
    static PerDevice ready;
    auto kern = volw32_kernel<S, TX, NP, TG>;
    if (int rc = allow_shared(kern, ready)) return rc;
    const int64_t nwork = (E + 15) / 16 * nrhs;
    const Plan p = make_plan(most, nwork, WarpBlocks(Nq).count(), S::Q * warp32_volume_frags<S>(Nq), kSplit32, ctas);
    const size_t smem = tab + (p.split.whole < nwork ? p.warps * per_warp : 0);
    kern<<<p.grid, 32 * p.warps, smem, s>>>(E, Nq, wg, p.split, x, y, ld, nrhs);
    return cudaGetLastError() == cudaSuccess ? 0 : TDG_E_CUDA;
}

template <class S, typename TX, int NP>
int run_volume32(int64_t E, int Nq, WarpGeo32 const& wg, const TX* x, TX* y, int nrhs, int64_t ld, cudaStream_t s,
                 int ctas) {
    using L = WarpTile32<S>;
    const size_t limit = shared_limit();
    const size_t tab = sizeof(float) * 64 * static_cast<size_t>(warp32_volume_frags<S>(Nq));
    const size_t per_warp = sizeof(float) * volume32_warp_floats<S>();
    if (tab + 4 * per_warp <= limit) {
        const int most = static_cast<int>(std::min<size_t>(L::WARPS, (limit - tab) / per_warp));
        return go_volume<S, TX, NP, false>(E, Nq, wg, x, y, nrhs, ld, s, ctas, most, tab, per_warp);
    }
    return go_volume<S, TX, NP, true>(E, Nq, wg, x, y, nrhs, ld, s, ctas, L::WARPS, 0, per_warp);
}

// which: 0 the volume term, 1 the facet terms
template <class S, typename TX, int NP>
int run32(int which, int64_t E, int Nq, int nq, WarpGeo32 const& wg, const TX* x, TX* y, int nrhs, int64_t ld,
          cudaStream_t s, int ctas, bool early) {
    return which == 0 ? run_volume32<S, TX, NP>(E, Nq, wg, x, y, nrhs, ld, s, ctas)
                      : run_facets32<S, TX, NP>(nq, wg, x, y, nrhs, ld, s, ctas, early);
}

template <int D, int N, typename TX, int NP>
int kind32(int which, int kind, int64_t E, int Nq, int nq, WarpGeo32 const& wg, const TX* x, TX* y, int nrhs,
           int64_t ld, cudaStream_t s, int ctas, bool early) {
    if (kind == kPoisson) return run32<Shape<D, N, kPoisson>, TX, NP>(which, E, Nq, nq, wg, x, y, nrhs, ld, s, ctas, early);
    return run32<Shape<D, N, kElasticity>, TX, NP>(which, E, Nq, nq, wg, x, y, nrhs, ld, s, ctas, early);
}

template <int D, typename TX, int NP>
int deg32(int which, int N, int kind, int64_t E, int Nq, int nq, WarpGeo32 const& wg, const TX* x, TX* y, int nrhs,
          int64_t ld, cudaStream_t s, int ctas, bool early) {
    switch (N) {
        case 1: return kind32<D, 1, TX, NP>(which, kind, E, Nq, nq, wg, x, y, nrhs, ld, s, ctas, early);
        case 2: return kind32<D, 2, TX, NP>(which, kind, E, Nq, nq, wg, x, y, nrhs, ld, s, ctas, early);
        case 3: return kind32<D, 3, TX, NP>(which, kind, E, Nq, nq, wg, x, y, nrhs, ld, s, ctas, early);
        case 4: return kind32<D, 4, TX, NP>(which, kind, E, Nq, nq, wg, x, y, nrhs, ld, s, ctas, early);
        default: return TDG_E_INVALID;
    }
}

template <typename TX, int NP>
int warp32_terms_impl(int which, int D, int N, int kind, int64_t E, int Nq, int nq, WarpGeo32 const& wg, const TX* x, TX* y,
          int nrhs, int64_t ld, cudaStream_t s, int ctas, bool early) {
    if (D == 2) return deg32<2, TX, NP>(which, N, kind, E, Nq, nq, wg, x, y, nrhs, ld, s, ctas, early);
    if (D == 3) return deg32<3, TX, NP>(which, N, kind, E, Nq, nq, wg, x, y, nrhs, ld, s, ctas, early);
    return TDG_E_INVALID;
}

}  // namespace

}  // namespace tdg
