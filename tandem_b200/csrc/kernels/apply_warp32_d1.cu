// Warp-tile FP32 kernels: double vectors, one TF32 pass.
#include "apply_warp32_impl.cuh"

namespace tdg {

int warp32_terms_d1(int which, int D, int N, int kind, int64_t E, int Nq, int nq, WarpGeo32 const& wg, const double* x,
                    double* y, int nrhs, int64_t ld, cudaStream_t s, int ctas, bool early) {
    return warp32_terms_impl<double, 1>(which, D, N, kind, E, Nq, nq, wg, x, y, nrhs, ld, s, ctas, early);
}

}  // namespace tdg
