// Volume term of the FP64 apply in passes over the quadrature points (tdg_set_apply_tile): one CTA
// per tile of 24 columns (element, component), per pass of qc points R = T_V U into shared memory on
// the FP64 tensor pipe, the pointwise stress, Y += T_V^T R.  The coefficient blocks of the next tile
// are copied in with cp.async while the current one computes -- element-major as x holds them, at a
// component stride KS and an element stride LDU chosen so that the m8n8k4 B-fragment loads of every
// half warp hit 16 distinct 8-byte banks.  The geometry is the warp-tile kernels' (apply_warp.cuh),
// whose one-warp tiles are the faster form (3D p4 elasticity, 24,576 elements: 90 us against 127 us in
// one pass); this kernel runs where a pass height is asked for.
#pragma once

#include "apply_warp.cuh"
#include "async.cuh"

namespace tdg {

// ---- staged coefficient blocks --------------------------------------------------------------------

// True when the B-fragment addresses (k = t, n = nt * 8 + g; address (n / Q) * ldu + (n % Q) * ks
// + k) of both half warps are distinct modulo 16 doubles, for every n-tile.
__host__ __device__ constexpr bool staged_conflict_free(int Q, int ks, int ldu, int ntn) {
    for (int nt = 0; nt < ntn; ++nt)
        for (int half = 0; half < 2; ++half) {
            bool used[16] = {};
            for (int g = 4 * half; g < 4 * half + 4; ++g)
                for (int t = 0; t < 4; ++t) {
                    const int n = nt * 8 + g;
                    const int a = ((n / Q) * ldu + (n % Q) * ks + t) % 16;
                    if (used[a]) return false;
                    used[a] = true;
                }
        }
    return true;
}

// Element stride of the staged blocks: the smallest >= Q * ks (at most 16 more) that is conflict
// free, else Q * ks + 4.
__host__ __device__ constexpr int staged_ldu(int Q, int ks, int ntn) {
    for (int l = Q * ks; l < Q * ks + 16; ++l)
        if (staged_conflict_free(Q, ks, l, ntn)) return l;
    return Q * ks + 4;
}

// Component stride: the padded Nbf, or 4, 8 or 12 more where no element stride is conflict free
// with it (2D p4 elasticity: a stride of 16 puts both components' k on the same banks).
__host__ __device__ constexpr int staged_ks(int Q, int kp, int ntn) {
    for (int ks = kp; ks < kp + 16; ks += 4)
        if (staged_conflict_free(Q, ks, staged_ldu(Q, ks, ntn), ntn)) return ks;
    return kp;
}

template <class S>
struct Staged {
    using L = MmaTile<S>;
    static constexpr int KS = staged_ks(S::Q, L::KP, L::NTN);       // component stride
    static constexpr int LDU = staged_ldu(S::Q, KS, L::NTN);       // element stride
    static constexpr int UE = (L::NP + S::Q - 1) / S::Q;           // elements per staged tile
    static constexpr int USZ = UE * LDU;                           // doubles per staged tile
};

// C[M x NP] = A[M x K] U for rows [0, mrows), U staged element-major (Staged<S>), register-blocked
// over whole rows of output tiles: a warp's work item is one m-tile and all NTN n-tiles of it, so
// each k step loads one A fragment and NTN B fragments for NTN mma.
template <class S>
__device__ __forceinline__ void cta_gemm_store_rows(const double* A, const double* U, double* C, int mrows,
                                                    int ksteps, int warp, int lane) {
    using L = MmaTile<S>;
    using SU = Staged<S>;
    constexpr int Q = S::Q, NTN = L::NTN;
    const int g = lane >> 2, t = lane & 3;
    for (int mt = warp; mt < mrows / 8; mt += L::GW) {
        const double* ap = A + (mt * 8 + g) * L::LDT + t;
        const double* bp[NTN];
#pragma unroll
        for (int j = 0; j < NTN; ++j) {
            const int n = j * 8 + g;
            bp[j] = U + (n / Q) * SU::LDU + (n % Q) * SU::KS + t;
        }
        double acc[NTN][2];
#pragma unroll
        for (int j = 0; j < NTN; ++j) acc[j][0] = acc[j][1] = 0.0;
        for (int ks = 0; ks < ksteps; ++ks) {
            const double a = ap[ks * 4];
#pragma unroll
            for (int j = 0; j < NTN; ++j) dmma(acc[j], a, bp[j][ks * 4]);
        }
        double* c = C + (mt * 8 + g) * L::LDN + 2 * t;  // 16-byte aligned (LDN, 2t even)
#pragma unroll
        for (int j = 0; j < NTN; ++j) *reinterpret_cast<double2*>(c + j * 8) = make_double2(acc[j][0], acc[j][1]);
    }
}

// Issues the cp.async copies of the coefficient blocks of up to UE elements (el[te] < 0: skipped)
// from xr into the staged buffer U, one element block per warp with the lanes along the block.
template <class S, int NT>
__device__ __forceinline__ void stage_blocks(const double* __restrict__ xr, const int* el, double* U, int tid) {
    using SU = Staged<S>;
    constexpr int per_el = S::Q * S::NBF;
    const int warp = tid >> 5, lane = tid & 31;
    for (int te = warp; te < SU::UE; te += NT / 32) {
        const int e = el[te];
        if (e < 0) continue;
        double* dst = U + te * SU::LDU;
        const double* src = xr + static_cast<int64_t>(e) * S::BS;
        for (int w = lane; w < per_el; w += 32) cp_async8(dst + (w / S::NBF) * SU::KS + (w % S::NBF), src + w);
    }
}

// (tile, right-hand side) of work item `work` in the per-RHS sweep order (the tile fastest): one right-hand side
// needs no division and 32-bit division serves every item count below 2^32.
__device__ __forceinline__ void sweep_tile_rhs(int64_t work, int64_t ntiles, int nrhs, int64_t& tile, int64_t& rhs) {
    if (nrhs == 1) {
        tile = work;
        rhs = 0;
    } else if (static_cast<uint64_t>(ntiles) * static_cast<uint64_t>(nrhs) <= 0xffffffffull) {
        const uint32_t w = static_cast<uint32_t>(work), n = static_cast<uint32_t>(ntiles);
        const uint32_t r = w / n;
        rhs = r;
        tile = w - r * n;
    } else {
        rhs = work / ntiles;
        tile = work - rhs * ntiles;
    }
}

// qc: volume points per pass; every pass but the last starts its table rows on an 8-row mma tile
// (qc * D rows), so qc is a multiple of face2_pass_step(D) (dispatch.hpp).
template <class S>
struct Vol2Layout {
    int MV, qc, off_U, off_R, total;
};
template <class S>
__host__ __device__ inline Vol2Layout<S> vol2_layout(int Nq, int qc) {
    using L = MmaTile<S>;
    Vol2Layout<S> l;
    l.MV = round8(S::D * Nq);
    l.qc = qc;
    l.off_U = l.MV * L::LDT;
    l.off_R = l.off_U + 2 * Staged<S>::USZ;
    l.total = l.off_R + round8(qc * S::D) * L::LDN;
    return l;
}

template <class S>
__global__ void __launch_bounds__(MmaTile<S>::NT, 2)
    vol2_kernel(int64_t E, int Nq, WarpGeo wg, const double* __restrict__ tv, const double* __restrict__ x,
                double* __restrict__ y, int64_t ld, int nrhs, int qc) {
    using L = MmaTile<S>;
    using SU = Staged<S>;
    constexpr int D = S::D, NBF = S::NBF, Q = S::Q, BS = S::BS, VF = WarpTile<S>::VF;
    constexpr int TE = L::TE, NT = L::NT, LDN = L::LDN, LDT = L::LDT;
    const WarpBlocks blk(Nq);
    const int gstride = VF * (64 * blk.full + 32 * blk.half);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const Vol2Layout<S> lay = vol2_layout<S>(Nq, qc);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* sm = reinterpret_cast<double*>(smem_raw);
    double* TV = sm;
    double* Ub = sm + lay.off_U;
    double* R0 = sm + lay.off_R;
    __shared__ int s_el[2][SU::UE];
    for (int i = tid; i < lay.MV * LDT; i += NT) sm[i] = tv[i];
    for (int i = tid; i < 2 * SU::USZ; i += NT) Ub[i] = 0.0;  // padding stays zero, stale columns finite

    const int64_t ntiles = (E + TE - 1) / TE;
    const int64_t nwork = ntiles * nrhs;
    auto stage = [&](int64_t work, int buf) {
        int64_t tile, rhs;
        sweep_tile_rhs(work, ntiles, nrhs, tile, rhs);
        const double* xr = x + rhs * ld;
        if (tid < SU::UE) {
            const int64_t e = tile * TE + tid;
            s_el[buf][tid] = (tid < TE && e < E) ? static_cast<int>(e) : -1;
        }
        __syncthreads();
        stage_blocks<S, NT>(xr, s_el[buf], Ub + buf * SU::USZ, tid);
        cp_async_commit();
    };
    __syncthreads();
    int buf = 0;
    if (static_cast<int64_t>(blockIdx.x) < nwork) stage(blockIdx.x, 0);
    for (int64_t work = blockIdx.x; work < nwork; work += gridDim.x, buf ^= 1) {
        int64_t tile, rhs;
        sweep_tile_rhs(work, ntiles, nrhs, tile, rhs);
        double* yr = y + rhs * ld;
        const int64_t next = work + gridDim.x;
        __syncthreads();  // the previous tile is done with the other buffer
        if (next < nwork) {
            stage(next, buf ^ 1);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
        const double* U = Ub + buf * SU::USZ;
        const int* el = s_el[buf];
        double yacc[L::YPW][2][2];
#pragma unroll
        for (int j = 0; j < L::YPW; ++j) yacc[j][0][0] = yacc[j][0][1] = yacc[j][1][0] = yacc[j][1][1] = 0.0;
        for (int q0 = 0; q0 < Nq; q0 += qc) {
            const int nqc = (Nq - q0 < qc) ? (Nq - q0) : qc;
            const int rows = round8(nqc * D);
            cta_gemm_store_rows<S>(TV + q0 * D * LDT, U, R0, rows, L::KP / 4, warp, lane);
            __syncthreads();
            for (int it = tid; it < TE * nqc; it += NT) {
                const int te = it % TE, qq = it / TE, q = q0 + qq;
                const int e = el[te];
                if (e < 0) continue;
                // the point's fields in the lane-ordered geometry (8 elements x 8 points per block)
                const int b = q / 8, s = q % 8, fs = b < blk.full ? 64 : 32;
                const double* gp = wg.vol + (e / 8) * static_cast<int64_t>(gstride) + b * (VF * 64) +
                                   (b < blk.full ? ((e % 8) * 4 + s / 2) * 2 + s % 2 : (e % 8) * 4 + s);
                double f[VF], g[D][Q];
#pragma unroll
                for (int c = 0; c < VF; ++c) f[c] = gp[c * fs];
                double* rr = R0 + (qq * D) * LDN + te * Q;
#pragma unroll
                for (int a = 0; a < D; ++a)
#pragma unroll
                    for (int r = 0; r < Q; ++r) g[a][r] = rr[a * LDN + r];
                volume_flux<S>(f, g);
#pragma unroll
                for (int a = 0; a < D; ++a)
#pragma unroll
                    for (int r = 0; r < Q; ++r) rr[a * LDN + r] = g[a][r];
            }
            __syncthreads();
            cta_gemm_acc_t<L>(TV + q0 * D * LDT, R0, yacc, rows, warp, lane);
            __syncthreads();
        }
        const int g = lane >> 2, t = lane & 3;
#pragma unroll
        for (int j = 0; j < L::YPW; ++j) {
            const int tl = warp + j * L::GW;
            if (tl < L::YT) {
                const int ym = tl % L::MYT, yn = tl / L::MYT;
                const int k = ym * 8 + g;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int c = yn * 8 + 2 * t + h;
                    if (k < NBF && c < L::NC) {
                        const int te = c / Q, r = c % Q;
                        const int e = el[te];
                        if (e >= 0) yr[static_cast<int64_t>(e) * BS + k + NBF * r] = yacc[j][0][h] + yacc[j][1][h];
                    }
                }
            }
        }
    }
    cp_async_wait<0>();
}

}  // namespace tdg
