// Launcher of the face-centric FP32 apply: warp-tile kernels (apply_warp32.cuh), the volume term on the
// 5th-generation tensor cores where asked for and possible (apply_tc05.cuh).
#include "apply_warp32.cuh"
#include "dispatch.hpp"

#include "../../../include/tandem_b200.h"

#include <type_traits>

namespace tdg {

// which: 0 the volume term, 1 the facet terms; one source file per vector type and pass count
int warp32_terms_f3(int which, int D, int N, int kind, int64_t E, int Nq, int nq, WarpGeo32 const& wg, const float* x,
                    float* y, int nrhs, int64_t ld, cudaStream_t s, int ctas, bool early);
int warp32_terms_d3(int which, int D, int N, int kind, int64_t E, int Nq, int nq, WarpGeo32 const& wg, const double* x,
                    double* y, int nrhs, int64_t ld, cudaStream_t s, int ctas, bool early);
int warp32_terms_d1(int which, int D, int N, int kind, int64_t E, int Nq, int nq, WarpGeo32 const& wg, const double* x,
                    double* y, int nrhs, int64_t ld, cudaStream_t s, int ctas, bool early);

template <typename TX>
int launch_apply_warp32(int D, int N, int kind, DevOp<float> const& op, Tc32Tiles const& mt, WarpGeo32 const& wg,
                        const TX* x, TX* y, int nrhs, int64_t ld, cudaStream_t s, int ctas, bool vol05, int passes) {
    if (passes != 3 && !(passes == 1 && std::is_same_v<TX, double>)) return TDG_E_INVALID;
    if (nrhs < 1 || !wg.vtab || !wg.vol || (wg.nftiles > 0 && (!wg.ftab || !wg.fct))) return TDG_E_INVALID;
    int rc = TDG_E_INVALID;
    if (vol05) {
        rc = launch_vol_tc05<TX>(D, N, kind, op, mt, x, y, nrhs, ld, s, passes);
        if (rc && rc != TDG_E_INVALID) return rc;
    }
    const bool early = rc != 0;  // behind the warp-tile volume kernel
    for (int which = early ? 0 : 1; which < 2; ++which) {
        if constexpr (std::is_same_v<TX, float>)
            rc = warp32_terms_f3(which, D, N, kind, op.E, op.Nq, op.nq, wg, x, y, nrhs, ld, s, ctas, early);
        else if (passes == 3)
            rc = warp32_terms_d3(which, D, N, kind, op.E, op.Nq, op.nq, wg, x, y, nrhs, ld, s, ctas, early);
        else
            rc = warp32_terms_d1(which, D, N, kind, op.E, op.Nq, op.nq, wg, x, y, nrhs, ld, s, ctas, early);
        if (rc) return rc;
    }
    return 0;
}

template int launch_apply_warp32<float>(int, int, int, DevOp<float> const&, Tc32Tiles const&, WarpGeo32 const&,
                                        const float*, float*, int, int64_t, cudaStream_t, int, bool, int);
template int launch_apply_warp32<double>(int, int, int, DevOp<float> const&, Tc32Tiles const&, WarpGeo32 const&,
                                         const double*, double*, int, int64_t, cudaStream_t, int, bool, int);

}  // namespace tdg
