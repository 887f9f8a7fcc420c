// Block-Jacobi preconditioner on the device.
//
// assemble: the element diagonal block D_e = A_vol(e) + sum over the element's faces of the
//   facet self block (tandem's DGOperator::assemble restricted to A(e, e),
//   src/form/DGOperator.h:121-187, with Poisson::assemble_volume/skeleton/boundary,
//   app/localoperator/Poisson.cpp:225-385, and Elasticity::assemble_*, Elasticity.cpp:317-519;
//   IP lift, interior constants c00 = c10 = -1/2, boundary -1, c20 = penalty).  Blocks are
//   column-major: blk[e][col * BS + row], row = k + NBF p.
// invert: Gauss-Jordan without pivoting in shared memory; a non-positive pivot marks the block
//   as not positive definite (SIPG diagonal blocks are SPD for a sufficient penalty).
// apply: z_e = D_e^-1 r_e.  The apply is bound by reading the inverses, so they are stored as the
//   half that symmetry leaves: entry (i, (i + d) mod BS) for every row i and d = 0 .. BS / 2, d-major
//   (odd sizes hold every pair once, even ones the pairs of d = BS / 2 twice).  A row then takes two
//   entries per d, both contiguous over the rows: its own and that of row i - d; the block is staged
//   in shared memory, because the second access through L1 cost what the halved bytes gave.
//   Several FP64 right-hand sides go through the FP64 tensor pipe, one warp per element, the inverse
//   read once per 8 to 32 columns.
#pragma once

#include "apply_mma.cuh"
#include "async.cuh"
#include "early.cuh"
#include "common.cuh"

namespace tdg {

// Entries of a packed symmetric BS x BS inverse, padded to whole 16 bytes in FP32 and FP64.
__host__ __device__ constexpr int bjac_packed_size(int bs) { return ((bs / 2 + 1) * bs + 3) / 4 * 4; }

template <class S>
__host__ __device__ inline int bjac_assemble_smem_doubles(int Nq, int nq) {
    int vol = S::NBF * S::D * Nq + 2 * Nq;
    int fct = S::NBF * S::D * nq + S::NBF * nq + (S::D + 2 + 2) * nq;
    return vol > fct ? vol : fct;
}

template <class S>
__global__ void __launch_bounds__(256) bjac_assemble_kernel(DevOp<double> op, double* __restrict__ blk) {
    constexpr int D = S::D, NBF = S::NBF, Q = S::Q, BS = S::BS, DD = S::DD, NF = S::NF;
    const int Nq = op.Nq, nq = op.nq;
    const int64_t e = blockIdx.x;
    const int tid = threadIdx.x;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* sm = reinterpret_cast<double*>(smem_raw);
    double* out = blk + e * BS * BS;

    // volume: physical gradients Dx[k][i][q]
    double* sDx = sm;
    double* sC = sm + NBF * D * Nq;
    for (int it = tid; it < NBF * D * Nq; it += blockDim.x) {
        const int q = it % Nq;
        const int i = (it / Nq) % D;
        const int k = it / (Nq * D);
        double s = 0.0;
        for (int a = 0; a < D; ++a)
            s += op.vG[(e * DD + a * D + i) * Nq + q] * op.Dxi_Q[(k * D + a) * Nq + q];
        sDx[it] = s;
    }
    const int ncoef = (S::KIND == kPoisson) ? 1 : 2;
    for (int it = tid; it < ncoef * Nq; it += blockDim.x) sC[it] = op.vCoef[e * ncoef * Nq + it];
    __syncthreads();
    for (int it = tid; it < BS * BS; it += blockDim.x) {
        const int row = it % BS, col = it / BS;
        const int k = row % NBF, p = row / NBF, l = col % NBF, u = col / NBF;
        double s = 0.0;
        if constexpr (S::KIND == kPoisson) {
            for (int q = 0; q < Nq; ++q) {
                double d = 0.0;
                for (int i = 0; i < D; ++i) d += sDx[(k * D + i) * Nq + q] * sDx[(l * D + i) * Nq + q];
                s += sC[q] * d;
            }
        } else {
            for (int q = 0; q < Nq; ++q) {
                const double lam = sC[q], mu = sC[Nq + q];
                double kl = 0.0;
                for (int j = 0; j < D; ++j) kl += sDx[(k * D + j) * Nq + q] * sDx[(l * D + j) * Nq + q];
                s += lam * sDx[(k * D + p) * Nq + q] * sDx[(l * D + u) * Nq + q] +
                     mu * ((p == u ? kl : 0.0) + sDx[(k * D + u) * Nq + q] * sDx[(l * D + p) * Nq + q]);
            }
        }
        out[it] = s;
    }

    // facet self blocks
    for (int f = 0; f < NF; ++f) {
        const int4 sd = op.sides[e * NF + f];
        const int bcv = sd.y >> 8;
        const bool skel = sd.z != static_cast<int>(e);
        if (!skel && !(bcv == 3 || bcv == 5)) continue;
        const int fct = sd.x;
        const int own = skel ? (sd.y & 0xff) : 0;
        const double flip = (skel && own == 1) ? -1.0 : 1.0;
        const double c = skel ? -0.5 : -1.0;
        const double pen = op.penalty[fct];
        __syncthreads();
        double* fDx = sm;                       // [NBF][D][nq]  (Poisson: K * Dx)
        double* fE = fDx + NBF * D * nq;        // [NBF][nq]
        double* fn = fE + NBF * nq;             // [D][nq] outward normal
        double* fnl = fn + D * nq;              // [nq]
        double* fc = fnl + nq;                  // [2][nq] lam, mu
        for (int it = tid; it < NBF * D * nq; it += blockDim.x) {
            const int q = it % nq;
            const int i = (it / nq) % D;
            const int k = it / (nq * D);
            double s = 0.0;
            for (int a = 0; a < D; ++a) {
                double g;
                if constexpr (S::KIND == kPoisson) {
                    g = op.fCoef[((static_cast<int64_t>(fct) * 2 + own) * DD + a * D + i) * nq + q];
                } else {
                    g = op.fG[((static_cast<int64_t>(fct) * 2 + own) * DD + a * D + i) * nq + q];
                }
                s += g * op.Dxi_q[((f * NBF + k) * D + a) * nq + q];
            }
            fDx[it] = s;
        }
        for (int it = tid; it < NBF * nq; it += blockDim.x) fE[it] = op.E_q[f * NBF * nq + it];
        for (int it = tid; it < D * nq; it += blockDim.x)
            fn[it] = flip * op.fN[static_cast<int64_t>(fct) * D * nq + it];
        for (int it = tid; it < nq; it += blockDim.x) {
            fnl[it] = op.fNl[static_cast<int64_t>(fct) * nq + it];
            if constexpr (S::KIND != kPoisson) {
                fc[it] = op.fCoef[(static_cast<int64_t>(fct) * 4 + 2 * own + 0) * nq + it];
                fc[nq + it] = op.fCoef[(static_cast<int64_t>(fct) * 4 + 2 * own + 1) * nq + it];
            }
        }
        __syncthreads();
        for (int it = tid; it < BS * BS; it += blockDim.x) {
            const int row = it % BS, col = it / BS;
            const int k = row % NBF, p = row / NBF, l = col % NBF, u = col / NBF;
            double s = 0.0;
            for (int q = 0; q < nq; ++q) {
                const double wq = op.w[q];
                const double ek = fE[k * nq + q], el = fE[l * nq + q];
                if constexpr (S::KIND == kPoisson) {
                    double dk = 0.0, dl = 0.0;
                    for (int i = 0; i < D; ++i) {
                        dk += fDx[(k * D + i) * nq + q] * fn[i * nq + q];
                        dl += fDx[(l * D + i) * nq + q] * fn[i * nq + q];
                    }
                    s += wq * (c * dk * el + c * dl * ek + pen * ek * el * fnl[q]);
                } else {
                    const double lam = fc[q], mu = fc[nq + q];
                    double dkn = 0.0, dln = 0.0;
                    for (int j = 0; j < D; ++j) {
                        dkn += fDx[(k * D + j) * nq + q] * fn[j * nq + q];
                        dln += fDx[(l * D + j) * nq + q] * fn[j * nq + q];
                    }
                    // traction operator T[m, a, b] = lam Dx[m,a] n_b + mu (dmn delta_ab + Dx[m,b] n_a)
                    const double Tl = lam * fDx[(l * D + u) * nq + q] * fn[p * nq + q] +
                                      mu * ((u == p ? dln : 0.0) + fDx[(l * D + p) * nq + q] * fn[u * nq + q]);
                    const double Tk = lam * fDx[(k * D + p) * nq + q] * fn[u * nq + q] +
                                      mu * ((p == u ? dkn : 0.0) + fDx[(k * D + u) * nq + q] * fn[p * nq + q]);
                    s += wq * (c * ek * Tl + c * el * Tk + (p == u ? pen * ek * el * fnl[q] : 0.0));
                }
            }
            out[it] += s;
        }
    }
}

// In-place Gauss-Jordan inversion of one BS x BS block per CTA; writes the packed inverse in T.
template <int BS, typename T>
__global__ void __launch_bounds__(256)
    bjac_invert_kernel(const double* __restrict__ blk, T* __restrict__ inv, int* __restrict__ status) {
    const int64_t e = blockIdx.x;
    const int tid = threadIdx.x;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* a = reinterpret_cast<double*>(smem_raw);  // column-major a[col * BS + row]
    double* colk = a + BS * BS;                       // copy of column k
    __shared__ int bad;
    if (tid == 0) bad = 0;
    for (int i = tid; i < BS * BS; i += blockDim.x) a[i] = blk[e * BS * BS + i];
    __syncthreads();
    for (int k = 0; k < BS; ++k) {
        double piv = a[k * BS + k];
        if (!(piv > 0.0)) {
            if (tid == 0) bad = 1;
            piv = 1.0;
        }
        const double ip = 1.0 / piv;
        // save column k (multipliers), then scale row k
        for (int i = tid; i < BS; i += blockDim.x) colk[i] = a[k * BS + i];
        __syncthreads();
        for (int j = tid; j < BS; j += blockDim.x) a[j * BS + k] = (j == k ? 1.0 : a[j * BS + k]) * ip;
        __syncthreads();
        for (int it = tid; it < BS * BS; it += blockDim.x) {
            const int i = it % BS, j = it / BS;
            if (i == k) continue;
            const double fi = colk[i];
            const double rk = a[j * BS + k];
            a[it] = (j == k ? 0.0 : a[it]) - fi * rk;
        }
        __syncthreads();
    }
    constexpr int PK = bjac_packed_size(BS);
    for (int i = tid; i < PK; i += blockDim.x) {
        const int d = i / BS, row = i % BS;
        inv[e * PK + i] = d <= BS / 2 ? static_cast<T>(a[(row + d) % BS * BS + row]) : T(0);
    }
    if (tid == 0 && bad) atomicOr(status, 1);
}

// Entries d0 <= d < d1 of one row of Dinv r, added to s: m the packed inverse's row d0 at this row, rv
// the vector at this row, held twice in a row (no wrap of row + d) with RB copies 2 BS apart.
template <int BS, typename TM, typename TV, int RB>
__device__ __forceinline__ void bjac_row(const TM* m, const TV* rv, int row, int d0, int d1, TV (&s)[RB]) {
    m -= d0 * BS;
    if (d0 == 0) {
#pragma unroll
        for (int j = 0; j < RB; ++j) s[j] += static_cast<TV>(m[0]) * rv[j * 2 * BS];
        d0 = 1;
    }
    const int pairs = d1 < (BS + 1) / 2 ? d1 : (BS + 1) / 2;
#pragma unroll 8
    for (int d = d0; d < pairs; ++d) {
        const TV a = static_cast<TV>(m[d * BS]);
        const TV b = static_cast<TV>(m[d * BS - d + (row < d ? BS : 0)]);
#pragma unroll
        for (int j = 0; j < RB; ++j) s[j] += a * rv[j * 2 * BS + d] + b * rv[j * 2 * BS + BS - d];
    }
    if (BS % 2 == 0 && d1 > BS / 2) {  // held for both rows of the pair
        const TV a = static_cast<TV>(m[BS / 2 * BS]);
#pragma unroll
        for (int j = 0; j < RB; ++j) s[j] += a * rv[j * 2 * BS + BS / 2];
    }
}

// z = Dinv r for one right-hand side: teams of 128 threads, per step a team takes a tile of TE
// consecutive elements, or of a large block (over 24 KB) half its entries, while the next step's are
// copied in (cp.async): small enough stages for four teams per SM, which hide each other's
// shared-memory latency.  Bound by the inverses' bytes: 105 x 105 FP64 blocks of 10,368 elements
// 161 (whole square blocks, 5.7 TB/s) -> 84 us (5.5 TB/s on half the bytes); whole blocks as stages,
// two teams per SM, 120 us; both accesses through L1 172 us.
template <int BS, typename TM>
struct BjacStream {
    static constexpr int TT = 128, TE = TT / BS > 0 ? TT / BS : 1, PK = bjac_packed_size(BS), HD = BS / 2 + 1;
    static constexpr int PARTS = (TE == 1 && PK * sizeof(TM) > 24 * 1024) ? 2 : 1;
    static constexpr int DC = PARTS == 1 ? HD : (HD / 2 + 3) / 4 * 4;  // rows d per part: whole 16 bytes
    static constexpr int STAGE = PARTS == 1 ? TE * PK : DC * BS;       // entries
    static constexpr size_t smem(size_t vec) { return 2 * 2 * (STAGE * sizeof(TM) + TE * 2 * BS * vec); }
    static_assert(PARTS == 1 || (PK - DC * BS <= STAGE && DC * BS % 4 == 0), "parts of a block");
};
template <int BS, typename TM, typename TV>
__global__ void __launch_bounds__(256)
    bjac_stream_kernel(int64_t E, const TM* __restrict__ inv, const TV* r, TV* z) {
    using L = BjacStream<BS, TM>;
    constexpr int TE = L::TE, TT = L::TT, PK = L::PK, PARTS = L::PARTS;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int team = threadIdx.x / TT, tid = threadIdx.x % TT;
    TM* stage0 = reinterpret_cast<TM*>(smem_raw) + team * 2 * L::STAGE;
    TV* vec0 = reinterpret_cast<TV*>(smem_raw + 4 * L::STAGE * sizeof(TM)) + team * 2 * (TE * 2 * BS);
    const int64_t ntiles = (E + TE - 1) / TE, step = static_cast<int64_t>(gridDim.x) * 2;
    const int te = tid / BS, row = tid % BS;
    const bool mine = te < TE;
    const auto load = [&](int64_t tile, int part, int buf) {  // these inverses on their way
        if (tile < ntiles) {
            const int64_t e0 = tile * TE;
            const int entries = PARTS == 1 ? static_cast<int>(E - e0 < TE ? E - e0 : TE) * PK
                                           : (part ? PK - L::DC * BS : L::DC * BS);
            const char* src = reinterpret_cast<const char*>(inv + e0 * PK + part * (L::DC * BS));
            char* dst = reinterpret_cast<char*>(stage0 + buf * L::STAGE);
            for (int i = tid; i < entries * static_cast<int>(sizeof(TM)) / 16; i += TT) cp_async16(dst + i * 16, src + i * 16);
        }
        cp_async_commit();
    };
    const auto vec = [&](int64_t tile) {
        const int64_t e = tile * TE + te;
        return (mine && tile < ntiles && e < E) ? r[e * BS + row] : TV(0);
    };
    int64_t tile = static_cast<int64_t>(blockIdx.x) * 2 + team;
    if (tile >= ntiles) return;  // the whole team
    load(tile, 0, 0);
    TV cur = vec(tile);
    for (int k = 0; tile < ntiles; tile += step, ++k) {
        const int64_t e = tile * TE + te;
        const TV nxt = vec(tile + step);
        TV* v = vec0 + (k & 1) * (TE * 2 * BS) + te * 2 * BS + row;
        if (mine) v[0] = v[BS] = cur;
        cur = nxt;
        TV s[1] = {TV(0)};
#pragma unroll
        for (int part = 0; part < PARTS; ++part) {
            const int buf = (k * PARTS + part) & 1;
            load(part + 1 < PARTS ? tile : tile + step, part + 1 < PARTS ? part + 1 : 0, buf ^ 1);
            cp_async_wait<1>();
            mma_group_sync<TT>(team);
            if (mine && e < E)
                bjac_row<BS, TM, TV, 1>(stage0 + buf * L::STAGE + te * PK + row, v, row, part * L::DC,
                                        part + 1 < PARTS ? L::DC : L::HD, s);
            mma_group_sync<TT>(team);  // the stage is free again
        }
        if (mine && e < E) z[e * BS + row] = s[0];
    }
    cp_async_wait<0>();
}

// z = Dinv r, one thread per (element, row), RB right-hand sides at a time (blockIdx.y: the group).
template <int BS, typename TM, typename TV, int RB>
__global__ void __launch_bounds__(256) bjac_apply_kernel(int64_t E, const TM* __restrict__ inv,
                                                         const TV* __restrict__ r, TV* __restrict__ z,
                                                         int nrhs, int64_t ld) {
    let_next_kernel_start();
    wait_for_previous_kernel();
    constexpr int TE = (256 / BS) > 0 ? (256 / BS) : 1, PK = bjac_packed_size(BS);
    __shared__ TV sr[TE * RB * 2 * BS];
    const int rhs0 = blockIdx.y * RB;
    const int64_t ntiles = (E + TE - 1) / TE;
    const int te = threadIdx.x / BS, row = threadIdx.x % BS;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int64_t e0 = tile * TE, e = e0 + te;
        __syncthreads();
        for (int i = threadIdx.x; i < TE * RB * BS; i += blockDim.x) {
            const int t = i / (RB * BS), j = i / BS % RB, k = i % BS;
            const TV v = (e0 + t < E && rhs0 + j < nrhs) ? r[(rhs0 + j) * ld + (e0 + t) * BS + k] : TV(0);
            sr[(t * RB + j) * 2 * BS + k] = v;
            sr[(t * RB + j) * 2 * BS + BS + k] = v;
        }
        __syncthreads();
        if (te < TE && e < E) {
            TV s[RB] = {};
            bjac_row<BS, TM, TV, RB>(inv + e * PK + row, sr + te * RB * 2 * BS + row, row, 0, BS / 2 + 1, s);
#pragma unroll
            for (int j = 0; j < RB; ++j)
                if (rhs0 + j < nrhs) z[(rhs0 + j) * ld + e * BS + row] = s[j];
        }
    }
}

// z = Dinv r for groups of up to 8 NR FP64 right-hand sides (blockIdx.y: the group), Z [BS x columns] =
// Dinv R on the FP64 tensor pipe (A: the inverse, B: the columns).  Bound by the vectors' bytes (r and z may be
// the same): 15 x 15 blocks of 17,712 elements, 32 columns 109 -> 38 us.  W warps share the row tiles of an
// element: one for small blocks; four from 60, where one warp's chain of (BS / 8)(BS / 4) loads and
// products is the time (105 x 105, 6,000 elements, 8 columns: 272 us with one warp, 112 with four; 48
// elements 50 and 8.6).
template <int BS>
constexpr int bjac_mma_tiles() {  // n tiles a warp holds: their B fragments stay in registers
    return BS <= 35 ? 4 : (BS <= 60 ? 2 : 1);
}
template <int BS>
constexpr int bjac_mma_warps() {
    return BS < 60 ? 1 : 4;
}
template <int BS, typename TM>
__global__ void __launch_bounds__(128) bjac_mma_kernel(int64_t E, const TM* __restrict__ inv,
                                                       const double* r, double* z, int nrhs, int64_t ld) {
    constexpr int PK = bjac_packed_size(BS), KS = (BS + 3) / 4, MT = (BS + 7) / 8, NR = bjac_mma_tiles<BS>();
    constexpr int W = bjac_mma_warps<BS>(), EPC = 4 / W;  // elements of a CTA
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int rhs0 = blockIdx.y * 8 * NR;
    for (int64_t e = static_cast<int64_t>(blockIdx.x) * EPC + warp / W; e < E; e += static_cast<int64_t>(gridDim.x) * EPC) {
        const TM* m = inv + e * PK;
        double b[NR][KS];
#pragma unroll
        for (int n = 0; n < NR; ++n) {
            const int c = rhs0 + n * 8 + g;
            const double* rc = r + c * ld + e * BS;
#pragma unroll
            for (int ks = 0; ks < KS; ++ks) b[n][ks] = (c < nrhs && 4 * ks + t < BS) ? rc[4 * ks + t] : 0.0;
        }
        if constexpr (W > 1) __syncthreads();  // in place: every warp has read the element's rows
#pragma unroll 1
        for (int mt = warp % W; mt < MT; mt += W) {
            double acc[NR][2];
#pragma unroll
            for (int n = 0; n < NR; ++n) acc[n][0] = acc[n][1] = 0.0;
            const int i = mt * 8 + g;
#pragma unroll
            for (int ks = 0; ks < KS; ++ks) {
                const int j = 4 * ks + t;
                int d = j - i;
                if (d < 0) d += BS;
                const int at = d <= BS / 2 ? d * BS + i : (BS - d) * BS + j;
                const double a = (i < BS && j < BS) ? static_cast<double>(m[at]) : 0.0;
#pragma unroll
                for (int n = 0; n < NR; ++n)
                    if (rhs0 + n * 8 < nrhs) dmma(acc[n], a, b[n][ks]);
            }
#pragma unroll
            for (int n = 0; n < NR; ++n)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int c = rhs0 + n * 8 + 2 * t + h;
                    if (c < nrhs && i < BS) z[c * ld + e * BS + i] = acc[n][h];
                }
        }
    }
}

}  // namespace tdg
