// Warp-tile FP64 apply: the face-centric operator (a volume kernel that stores y, one pass over the
// facets that evaluates every facet once for both sides and adds into y; tandem's apply_volume /
// flux / apply_facet einsums, app/kernels/elasticity.py:201-234, poisson.py:123-140, the facet loop
// of Poisson.cpp:586-631 and Elasticity.cpp:734-801) in which one warp carries a tile of 8 elements
// or 8 facets from the coefficients to the result without a barrier and without staging products
// in shared memory.
//
// The products run on the FP64 tensor pipe (mma.sync m8n8k4) in the transposed form
//
//   forward   R[te][q]  = sum_k U[te][k] D[q][k]      A = U (rows: the tile's 8 elements), B = table
//   backward  Y[te][k]  = sum_q T[te][q] D[q][k]      A = T, B = table
//
// one accumulator tile per component r (rows te) and kind of derivative.  A lane (g = lane / 4,
// t = lane % 4) of a forward accumulator holds element g at the points 2t and 2t + 1 of a block of
// 8: the reference gradients of all components at its two points, so the pointwise stress / flux is
// register arithmetic, and its result is -- element for element -- the A fragment of the backward
// product (k index t of the mma = point 2t + h).  Nothing is exchanged between lanes.
//
// Facets use face-adapted reference coordinates: tangential directions along the face and one
// transversal direction (host/warp_tables.cpp).  In the nodal basis (elasticity) the values and
// tangential derivatives on a face depend only on the basis functions whose node lies on it (15 of
// 35 at 3D p4), so only the transversal derivative needs the full basis: 330 mma per side and
// component triple of 8 facets instead of 570 with the four full tables.
//
// By the symmetry of the nodal basis under a relabelling of the vertices all faces then share one
// table and differ only in the order of the basis functions (modal bases keep one per face).
//
// Measured on a B200 (whole apply, against the CTA-wide tile GEMMs through shared memory that these
// kernels replaced): 3D p4 elasticity, 48,000 tetrahedra 665 -> 365 us (volume 144, facets 220 apart; the
// products alone take 108 and 113 us of the FP64 pipe, the flux arithmetic 11 and 27); 2D p4 Poisson,
// 17,712 triangles x 32 columns 593 -> 238 us; 8,192 triangles 18.4 -> 11.8 us.  Facet atomics are
// not on the critical path (plain stores time the same).
//
// Facet modes: 1 interior flux, both sides; 2 boundary (Dirichlet / fault) flux, side 0; 3 interior
// flux of side 0 only with the element as its own neighbour (a boundary facet whose code is None, as
// the element-centric apply treats it).  The sum over a facet's contributions is unordered
// (atomics), so results agree with the element-centric kernels to rounding, not bit for bit.
//
// Tables: B fragments in the order the mma loops read them ([fragment][lane], conflict free),
// resident in the shared memory of the persistent CTA; shapes whose tables do not fit read them
// through L1.  Per-point geometry: the fields of 8 elements x 8 points in lane order.
#pragma once

#include "apply_mma.cuh"
#include "early.cuh"
#include "async.cuh"

#include <type_traits>

namespace tdg {

template <class S>
struct WarpTile {
    static constexpr bool NODAL = S::KIND == kElasticity;
    static constexpr int KS = (S::NBF + 3) / 4;  // k steps of a full forward product
    static constexpr int NT = (S::NBF + 7) / 8;  // n tiles of a full backward product
    // basis functions with a non-zero trace on a face, and the steps / tiles of the products that
    // need only those (modal bases: all of them)
    static constexpr int FN = NODAL ? cbinom(S::N + S::D - 1, S::D - 1) : S::NBF;
    static constexpr int KSS = (FN + 3) / 4;
    static constexpr int NTS = (FN + 7) / 8;
    // fields per volume point (Poisson: the symmetric J^-1 K W|J| J^-T; elasticity: J^-1, lam W|J|,
    // mu W|J|) and per facet point (host/warp_tables.cpp)
    static constexpr int VF = NODAL ? S::DD + 2 : S::D * (S::D + 1) / 2;
    static constexpr int SF = NODAL ? S::DD + 2 : S::D;      // per side
    static constexpr int CF = NODAL ? S::D + 1 : 1;          // shared by both sides
    static constexpr int FF = CF + 2 * SF;
    static constexpr int UF = S::Q * KS;         // A fragments of a tile's coefficients
    // Facet geometry streamed into shared memory by bulk copies (one per warp and block of points)
    // instead of register loads: it leaves the registers for 12 warps per SM, which hide the fixed
    // latency of the flux arithmetic better than 8 (3D p4 elasticity, 48,000 elements: 234 -> 220 us).
    // Smaller shapes have the registers anyway and lose (2D p4 Poisson, 32 columns: 171 -> 191 us).
    static constexpr bool STREAM = S::D == 3 && S::Q == 3 && S::N >= 3;
    // Most warps per CTA: the launch bound fixes the registers per thread.
    static constexpr int FWARPS = S::Q == 3 ? 12 : 16;  // facets
    static constexpr int VWARPS = S::Q == 3 ? (S::N >= 3 ? 8 : 12) : 16;  // volume: U, Y and a block in 250 registers
    static constexpr int FWD = S::D * KSS + KS;      // forward fragments of a full block of 8 facet points
    static constexpr int FWD_HALF = KSS + KS;        // of a half block (4 points, two kinds per n tile)
    static constexpr int BWD = S::D * NTS + NT;      // backward fragments of a half step (4 points)
    static constexpr int VPAIR = (S::D + 1) / 2;     // n tiles of a half block of volume points
};

// Points in blocks of 8; a remainder of at most 4 takes a half block.
struct WarpBlocks {
    int full, half;
    __host__ __device__ explicit WarpBlocks(int n) : full(n / 8 + (n % 8 > 4 ? 1 : 0)), half(n % 8 >= 1 && n % 8 <= 4) {}
    __host__ __device__ int steps() const { return 2 * full + half; }  // backward k steps per kind
    __host__ __device__ int count() const { return full + half; }
};

// Device data of the warp-tile apply (host/warp_tables.cpp builds them).
struct WarpGeo {
    const double* ftab = nullptr;   // facet fragments per local face (one for all of them: face_tables = 1)
    int face_tables = 0;
    const int* fperm = nullptr;     // [NF][8 NT] basis function of each permuted index (-1: none), face functions first
    const double* fct = nullptr;    // facet geometry per facet tile
    const int4* ftiles = nullptr;   // {first, count, key, 0}, key = l0 | l1 << 2 | mode << 4
    const int4* tids = nullptr;     // [tile][8] {facet (-1 unused), side-0 element, side-1 element, 0}
    int nftiles = 0;
    const double* vtab = nullptr;   // volume fragments
    const double* vol = nullptr;    // volume geometry per tile of 8 consecutive elements
    int* status = nullptr;          // device word: non-zero once a bounded wait ran out
};

// How a launch cuts its work items (tile, right-hand side): the first `whole` are one warp's each;
// of the others -- the last, partial round over the grid's warps, or all of a small mesh -- every
// block of points is an item of its own, so that they still occupy every sub-partition.
struct WarpSplit {
    int64_t whole = 0;
    int parts = 1;  // volume: warps that share one of the split items
};

// The fragment tables (n doubles, even) into shared memory, ending with a barrier.  Large tables go
// through the bulk-copy engine: one thread issues, so a CTA of few warps is not bound by its own
// loads (110 KB at 3D p4 by one warp: 67 us); up to 8 16-byte loads per thread are quicker by hand.
// False when the bounded wait ran out.
__device__ __forceinline__ bool load_tables(double* dst, const double* src, int n, unsigned long long* bar,
                                            int* status) {
    if (n / 2 <= 8 * static_cast<int>(blockDim.x)) {
        const double2* s2 = reinterpret_cast<const double2*>(src);
        double2* d2 = reinterpret_cast<double2*>(dst);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int i = threadIdx.x + j * blockDim.x;
            if (i < n / 2) d2[i] = __ldg(s2 + i);
        }
        __syncthreads();
        return true;
    }
    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        bulk_load(dst, src, static_cast<unsigned>(n * sizeof(double)), bar);
    }
    __syncthreads();
    const bool ok = mbar_wait_bounded(bar, 0);
    if (!ok) {
        if (threadIdx.x == 0 && status) atomicExch(status, 1);
        mbar_wait_bounded(bar, 0);  // once more: the copy must not outlive the CTA
    }
    return __syncthreads_and(ok) != 0;
}

template <class S>
__host__ __device__ inline int warp_volume_frags(int Nq) {
    using L = WarpTile<S>;
    const WarpBlocks b(Nq);
    return b.full * S::D * L::KS + b.half * L::VPAIR * L::KS + b.steps() * S::D * L::NT;
}

template <class S>
__host__ __device__ inline int warp_facet_frags(int nq) {  // fragments of one face
    using L = WarpTile<S>;
    const WarpBlocks b(nq);
    return b.full * L::FWD + b.half * L::FWD_HALF + b.steps() * L::BWD;
}

// B fragments at `p` ([fragment][lane]): shared memory, or global memory through L1 (TG).
template <bool TG>
struct Frags {
    const double* p;
    __device__ __forceinline__ double operator()(int f) const {
        if constexpr (TG)
            return __ldg(p + f * 32);
        else
            return p[f * 32];
    }
    __device__ __forceinline__ Frags operator+(int f) const { return {p + f * 32}; }
};

// Field f of this lane's point(s) in a block's geometry `gp` ([field][lane][point]).
template <int H>
__device__ __forceinline__ void geo_field(const double* __restrict__ gp, int f, int lane, double (&v)[H]) {
    if constexpr (H == 2) {
        const double2 d = __ldg(reinterpret_cast<const double2*>(gp + f * 64) + lane);
        v[0] = d.x;
        v[1] = d.y;
    } else {
        v[0] = __ldg(gp + f * 32 + lane);
    }
}

// Traces of one side at the block's points: tr[h][0] the value, tr[h][1 + b] the derivative along
// the face-adapted direction b (the last one transversal).
template <class S, int H, bool TG>
__device__ __forceinline__ void facet_traces(Frags<TG> tab, const double (&u)[S::Q][WarpTile<S>::KS],
                                             double (&tr)[H][S::D + 1][S::Q]) {
    using L = WarpTile<S>;
    constexpr int D = S::D, Q = S::Q, NK = H == 2 ? D + 1 : 2;
    double acc[NK][Q][2];
#pragma unroll
    for (int c = 0; c < NK; ++c)
#pragma unroll
        for (int r = 0; r < Q; ++r) acc[c][r][0] = acc[c][r][1] = 0.0;
    constexpr int NS = H == 2 ? D : 1;  // n tiles over the face functions; one more over all
#pragma unroll
    for (int ks = 0; ks < L::KSS; ++ks)
#pragma unroll
        for (int c = 0; c < NS; ++c) {
            const double b = tab(c * L::KSS + ks);
#pragma unroll
            for (int r = 0; r < Q; ++r) dmma(acc[c][r], u[r][ks], b);
        }
#pragma unroll
    for (int ks = 0; ks < L::KS; ++ks) {
        const double b = tab(NS * L::KSS + ks);
#pragma unroll
        for (int r = 0; r < Q; ++r) dmma(acc[NS][r], u[r][ks], b);
    }
#pragma unroll
    for (int c = 0; c <= D; ++c)
#pragma unroll
        for (int r = 0; r < Q; ++r) {
            if constexpr (H == 2) {
                tr[0][c][r] = acc[c][r][0];
                tr[1][c][r] = acc[c][r][1];
            } else {  // kinds 2p and 2p + 1 of one point in tile p
                tr[0][c][r] = acc[c / 2][r][c % 2];
            }
        }
}

// Weighted traction w sigma n of one side from its traces (cf: the shared fields, sf: the side's).
template <class S>
__device__ __forceinline__ void facet_traction(const double* cf, const double* sf, const double (&tr)[S::D + 1][S::Q],
                                               double (&tq)[S::Q]) {
    constexpr int D = S::D;
    if constexpr (S::KIND == kPoisson) {
        double s = 0.0;
#pragma unroll
        for (int a = 0; a < D; ++a) s += sf[a] * tr[1 + a][0];
        tq[0] = s;
    } else {
        const double lam = sf[0], mu = sf[1];
        const double* G = sf + 2;
        double nb[D], hb[D], div = 0.0;
#pragma unroll
        for (int b = 0; b < D; ++b) {
            nb[b] = hb[b] = 0.0;
#pragma unroll
            for (int j = 0; j < D; ++j) {
                nb[b] += G[b * D + j] * cf[j];
                hb[b] += tr[1 + b][j] * cf[j];
                div += G[b * D + j] * tr[1 + b][j];
            }
        }
#pragma unroll
        for (int r = 0; r < D; ++r) {
            double s = 0.0;
#pragma unroll
            for (int b = 0; b < D; ++b) s += nb[b] * tr[1 + b][r] + G[b * D + r] * hb[b];
            tq[r] = lam * div * cf[r] + mu * s;
        }
    }
}

// Gradient rows of one side's lift-back for the averaged jump uh.
template <class S>
__device__ __forceinline__ void facet_lift_rows(const double* cf, const double* sf, const double (&uh)[S::Q],
                                                double (&ga)[S::D][S::Q]) {
    constexpr int D = S::D;
    if constexpr (S::KIND == kPoisson) {
#pragma unroll
        for (int a = 0; a < D; ++a) ga[a][0] = uh[0] * sf[a];
    } else {
        const double mu = sf[1];
        const double* G = sf + 2;
        double un = 0.0;
#pragma unroll
        for (int j = 0; j < D; ++j) un += uh[j] * cf[j];
        un *= sf[0];
#pragma unroll
        for (int b = 0; b < D; ++b) {
            double nb = 0.0, vb = 0.0;
#pragma unroll
            for (int j = 0; j < D; ++j) {
                nb += G[b * D + j] * cf[j];
                vb += G[b * D + j] * uh[j];
            }
            nb *= mu;
            vb *= mu;
#pragma unroll
            for (int r = 0; r < D; ++r) ga[b][r] = un * G[b * D + r] + vb * cf[r] + nb * uh[r];
        }
    }
}

// One side's geometry of a block.  The fields of a block lie as [side 0][shared][side 1], so one
// side's part and the shared one are contiguous: side 0 reads [side][shared], side 1 [shared][side].
template <class S>
__host__ __device__ constexpr int facet_side_doubles(int H) {
    return (WarpTile<S>::CF + WarpTile<S>::SF) * 32 * H;
}

// ... loaded into registers ([field][lane][point]) ahead of the products that need them.
template <class S, int H>
struct LoadedGeo {
    using L = WarpTile<S>;
    const double* gp;  // the side's part in global memory
    double cf[L::CF][H], sf[L::SF][H];
    __device__ __forceinline__ void load(int side, int lane) {
#pragma unroll
        for (int f = 0; f < L::CF; ++f) geo_field<H>(gp, (side ? 0 : L::SF) + f, lane, cf[f]);
#pragma unroll
        for (int f = 0; f < L::SF; ++f) geo_field<H>(gp, (side ? L::CF : 0) + f, lane, sf[f]);
    }
    __device__ __forceinline__ void wait() {}
    __device__ __forceinline__ void point(int, int, int h, double (&c)[L::CF], double (&s)[L::SF]) const {
#pragma unroll
        for (int f = 0; f < L::CF; ++f) c[f] = cf[f][h];
#pragma unroll
        for (int f = 0; f < L::SF; ++f) s[f] = sf[f][h];
    }
};

// ... in the warp's shared-memory buffer ([field][point][lane]); the next block's copy is issued once
// the last point has been read.
template <class S, int H, class Arrived, class Release>
struct StreamedGeo {
    using L = WarpTile<S>;
    const double* buf;
    Arrived& arrived;
    Release& release;
    __device__ __forceinline__ void load(int, int) {}
    __device__ __forceinline__ void wait() { arrived(); }
    __device__ __forceinline__ void point(int side, int lane, int h, double (&c)[L::CF], double (&s)[L::SF]) const {
        const double* cp = buf + (side ? 0 : L::SF * 32 * H) + h * 32 + lane;
        const double* sp = buf + (side ? L::CF * 32 * H : 0) + h * 32 + lane;
#pragma unroll
        for (int f = 0; f < L::CF; ++f) c[f] = cp[f * 32 * H];
#pragma unroll
        for (int f = 0; f < L::SF; ++f) s[f] = sp[f * 32 * H];
        if (h == H - 1) release();
    }
};

// Phase 1 of a facet block: the traces of one side; side 0 combines them with the other side's
// (already in the stash when the facet has two) into the value row and the averaged jump, which
// replace it.  Stash rows of a half step: [0, Q) the trace / value row, [Q, 2Q) the traction /
// averaged jump.
template <class S, int H, bool TG, class Geo>
__device__ __forceinline__ void facet_phase1(Frags<TG> tab, const double (&u)[S::Q][WarpTile<S>::KS], Geo geo,
                                             int side, int lane, int mode, double* stash) {
    using L = WarpTile<S>;
    constexpr int Q = S::Q;
    geo.load(side, lane);
    double tr[H][S::D + 1][Q];
    facet_traces<S, H, TG>(tab, u, tr);
    geo.wait();
#pragma unroll
    for (int h = 0; h < H; ++h) {
        double c[L::CF], s[L::SF], tq[Q];
        geo.point(side, lane, h, c, s);
        facet_traction<S>(c, s, tr[h], tq);
        const double pn = c[L::CF - 1];  // penalty x weight x |n|
        double* st = stash + h * 2 * Q * 32 + lane;
#pragma unroll
        for (int r = 0; r < Q; ++r) {
            const double u0 = tr[h][0][r];
            if (side) {  // side 1 of an interior facet
                st[r * 32] = u0;
                st[(Q + r) * 32] = tq[r];
            } else if (mode == 1) {
                const double u1 = st[r * 32], t1 = st[(Q + r) * 32];
                st[r * 32] = -(0.5 * (tq[r] + t1) - pn * (u0 - u1));
                st[(Q + r) * 32] = 0.5 * (u1 - u0);
            } else if (mode == 2) {  // boundary: the side's own flux, lifted by -u
                st[r * 32] = -(tq[r] - pn * u0);
                st[(Q + r) * 32] = -u0;
            } else {  // the element is its own neighbour: no jump
                st[r * 32] = -tq[r];
                st[(Q + r) * 32] = 0.0;
            }
        }
    }
}

// Phase 2 of a facet block: one side's lift-back (side 1 with the opposite value row).
template <class S, int H, bool TG, class Geo>
__device__ __forceinline__ void facet_phase2(Frags<TG> tab, Geo geo, int side, int lane, const double* stash,
                                             double (&y)[S::Q][WarpTile<S>::NT][2]) {
    using L = WarpTile<S>;
    constexpr int D = S::D, Q = S::Q;
    const double sg = side ? -1.0 : 1.0;
    geo.load(side, lane);
    geo.wait();
#pragma unroll
    for (int h = 0; h < H; ++h) {
        double c[L::CF], s[L::SF], val[Q], uh[Q], ga[D][Q];
        geo.point(side, lane, h, c, s);
        const double* st = stash + h * 2 * Q * 32 + lane;
#pragma unroll
        for (int r = 0; r < Q; ++r) {
            val[r] = sg * st[r * 32];
            uh[r] = st[(Q + r) * 32];
        }
        facet_lift_rows<S>(c, s, uh, ga);
        const Frags<TG> tb = tab + h * L::BWD;
        // value and tangential rows act on the face functions, the transversal row on all
#pragma unroll
        for (int k = 0; k < D; ++k)
#pragma unroll
            for (int nt = 0; nt < L::NTS; ++nt) {
                const double b = tb(k * L::NTS + nt);
#pragma unroll
                for (int r = 0; r < Q; ++r) dmma(y[r][nt], k == 0 ? val[r] : ga[k - 1][r], b);
            }
#pragma unroll
        for (int nt = 0; nt < L::NT; ++nt) {
            const double b = tb(D * L::NTS + nt);
#pragma unroll
            for (int r = 0; r < Q; ++r) dmma(y[r][nt], ga[D - 1][r], b);
        }
    }
}

// Doubles of shared memory per warp of the facet kernel: the streamed geometry and the stash.
template <class S>
__host__ __device__ inline int facet_warp_doubles(int nq) {
    return (WarpTile<S>::STREAM ? facet_side_doubles<S>(2) : 0) + WarpBlocks(nq).steps() * 2 * S::Q * 32;
}

// One warp per facet tile (8 facets of one (l0, l1, mode)): phase 1 forms both sides' traces and
// tractions and from them the flux at every point (kept in the warp's stash), phase 2 lifts it back
// side by side, so only one side's result (60 registers at 3D p4 elasticity) is live at a time.
template <class S, bool TG>
__global__ void __launch_bounds__(32 * WarpTile<S>::FWARPS, 1)
    facew_kernel(int nq, WarpGeo wg, WarpSplit sp, const double* __restrict__ x, double* __restrict__ y, int64_t ld,
                 int nrhs) {
    using L = WarpTile<S>;
    constexpr int NBF = S::NBF, Q = S::Q, BS = S::BS, NF = S::NF, NP = 8 * L::NT;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nwarp = blockDim.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const WarpBlocks blk(nq);
    const int frags = warp_facet_frags<S>(nq);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* sm = reinterpret_cast<double*>(smem_raw);
    __shared__ int s_perm[NF * NP];
    __shared__ __align__(8) unsigned long long s_bar, s_gbar[L::FWARPS];
    const int tabsz = TG ? 0 : wg.face_tables * frags * 32;
    const int fstride = wg.face_tables == 1 ? 0 : frags * 32;  // between the faces' tables
    let_next_kernel_start();
    double* gbuf = sm + tabsz + warp * facet_warp_doubles<S>(nq);
    double* stash = gbuf + (L::STREAM ? facet_side_doubles<S>(2) : 0);
    for (int i = tid; i < NF * NP; i += blockDim.x) s_perm[i] = wg.fperm[i];
    if (L::STREAM && lane == 0) mbar_init(&s_gbar[warp], 1);
    if constexpr (!TG) {
        if (!load_tables(sm, wg.ftab, tabsz, &s_bar, wg.status)) return;
    } else {
        __syncthreads();
    }
    const int gstride = blk.full * L::FF * 64 + blk.half * L::FF * 32;
    const int nblk = blk.count();
    const int64_t nitems = sp.whole + (static_cast<int64_t>(wg.nftiles) * nrhs - sp.whole) * nblk;
    const int64_t stride = static_cast<int64_t>(nwarp) * gridDim.x;
    struct Item {
        int64_t tile, rhs;
        int b0, b1;  // its blocks of points
        int key;
        int4 id;     // of this lane's facet
    };
    const auto fetch = [&](int64_t item, Item& it) {
        int64_t work = item;
        it.b0 = 0;
        it.b1 = nblk;
        if (item >= sp.whole) {
            const int64_t part = item - sp.whole;
            work = sp.whole + part / nblk;
            it.b0 = static_cast<int>(part % nblk);
            it.b1 = it.b0 + 1;
        }
        work_tile_rhs(work, wg.nftiles, nrhs, it.tile, it.rhs);
        it.key = __ldg(&wg.ftiles[it.tile].z);
        it.id = __ldg(&wg.tids[it.tile * 8 + g]);
    };
    // one side's fields of block b
    const auto side_geo = [&](Item const& it, int side, int b) {
        return wg.fct + it.tile * gstride + b * (L::FF * 64) + (side ? L::SF * (b < blk.full ? 64 : 32) : 0);
    };
    unsigned late = 0;  // 2 | the phase whose wait ran out: no further waits and copies
    const auto issue = [&](Item const& it, int side, int b) {  // starts their copy into the warp's buffer
        if (lane == 0 && !late)
            bulk_load(gbuf, side_geo(it, side, b),
                      static_cast<unsigned>(facet_side_doubles<S>(b < blk.full ? 2 : 1) * sizeof(double)), &s_gbar[warp]);
    };
    unsigned parity = 0;
    const auto arrived = [&] {
        if (!late && !mbar_wait_bounded(&s_gbar[warp], parity)) {
            late = 2 | parity;  // the host reads the status word
            if (wg.status) atomicExch(wg.status, 1);
        }
        parity ^= 1;
    };
    const auto two_sided = [](Item const& it) { return (it.key >> 4) == 1; };
    int64_t item = static_cast<int64_t>(warp) * gridDim.x + blockIdx.x;
    bool waited = false;
    if (item >= nitems) return;
    Item it, nx;
    fetch(item, it);
    if (L::STREAM) issue(it, two_sided(it) ? 1 : 0, it.b0);
    for (;;) {
        const bool more = item + stride < nitems;
        nx = it;
        if (L::STREAM && more) fetch(item + stride, nx);
        const int mode = it.key >> 4;
        const bool two = two_sided(it);
        const int b0 = it.b0, bf = it.b1 < blk.full ? it.b1 : blk.full;  // full blocks [b0, bf)
        const bool bh = it.b1 > blk.full;                                 // then the half block
        int phase = 1, side = 0, b = 0;
        const auto release = [&] {  // the copy that follows block b of this phase and side
            __syncwarp();
            if (b + 1 < it.b1)
                issue(it, side, b + 1);
            else if (phase == 1)  // side 0's first, then phase 2's first
                issue(it, 0, b0);
            else if (two && !side)
                issue(it, 1, b0);
            else if (more)
                issue(nx, two_sided(nx) ? 1 : 0, nx.b0);
        };
        const auto geo = [&](auto h) {
            constexpr int H = decltype(h)::value;
            if constexpr (L::STREAM)
                return StreamedGeo<S, H, decltype(arrived), decltype(release)>{gbuf, arrived, release};
            else
                return LoadedGeo<S, H>{side_geo(it, side, b)};
        };
        using Two = std::integral_constant<int, 2>;
        using One = std::integral_constant<int, 1>;
        for (side = two ? 1 : 0; side >= 0; --side) {
            const int l = side ? (it.key >> 2) & 3 : it.key & 3;
            const int64_t e = it.id.x < 0 ? 0 : (side ? it.id.z : it.id.y);
            const double* xe = x + it.rhs * ld + e * BS;
            double u[Q][L::KS];  // face functions first
#pragma unroll
            for (int ks = 0; ks < L::KS; ++ks) {
                const int k = s_perm[l * NP + 4 * ks + t];
#pragma unroll
                for (int r = 0; r < Q; ++r) u[r][ks] = k >= 0 ? __ldg(xe + r * NBF + k) : 0.0;
            }
            const Frags<TG> tab{(TG ? wg.ftab : sm) + l * fstride + lane};
            for (b = b0; b < bf; ++b)
                facet_phase1<S, 2, TG>(tab + b * L::FWD, u, geo(Two{}), side, lane, mode, stash + b * (4 * Q * 32));
            if (bh) {
                b = blk.full;
                facet_phase1<S, 1, TG>(tab + b * L::FWD, u, geo(One{}), side, lane, mode, stash + b * (4 * Q * 32));
            }
        }
        phase = 2;
        double* yr = y + it.rhs * ld;
        for (side = 0; side <= (two ? 1 : 0); ++side) {
            const int l = side ? (it.key >> 2) & 3 : it.key & 3;
            const Frags<TG> tab = Frags<TG>{(TG ? wg.ftab : sm) + l * fstride + lane} +
                                  (blk.full * L::FWD + blk.half * L::FWD_HALF);
            double yac[Q][L::NT][2];
#pragma unroll
            for (int r = 0; r < Q; ++r)
#pragma unroll
                for (int nt = 0; nt < L::NT; ++nt) yac[r][nt][0] = yac[r][nt][1] = 0.0;
            for (b = b0; b < bf; ++b)
                facet_phase2<S, 2, TG>(tab + 2 * b * L::BWD, geo(Two{}), side, lane, stash + b * (4 * Q * 32), yac);
            if (bh) {
                b = blk.full;
                facet_phase2<S, 1, TG>(tab + 2 * b * L::BWD, geo(One{}), side, lane, stash + b * (4 * Q * 32), yac);
            }
            if (!waited) wait_for_previous_kernel();
            waited = true;
            if (it.id.x >= 0) {
                double* ye = yr + static_cast<int64_t>(side ? it.id.z : it.id.y) * BS;
#pragma unroll
                for (int nt = 0; nt < L::NT; ++nt)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int k = s_perm[l * NP + nt * 8 + h * 4 + t];
                        if (k >= 0)
#pragma unroll
                            for (int r = 0; r < Q; ++r) atomicAdd(ye + r * NBF + k, yac[r][nt][h]);
                    }
            }
        }
        if (!more) break;
        item += stride;
        if (L::STREAM)
            it = nx;
        else
            fetch(item, it);
    }
    if (L::STREAM && late) mbar_wait_bounded(&s_gbar[warp], late & 1);  // its copy must not outlive the CTA
}

// ---- volume term -------------------------------------------------------------------------------------

// Weighted stress at one point, mapped back to reference directions: g[a][r] -> T[a][r] in place.
template <class S>
__device__ __forceinline__ void volume_flux(const double* f, double (&g)[S::D][S::Q]) {
    constexpr int D = S::D;
    if constexpr (S::KIND == kPoisson) {
        double T[D];
#pragma unroll
        for (int a = 0; a < D; ++a) {
            T[a] = 0.0;
#pragma unroll
            for (int b = 0; b < D; ++b) {
                const int i = a < b ? a : b, j = a < b ? b : a;  // packed upper triangle
                T[a] += f[i * D - i * (i - 1) / 2 + j - i] * g[b][0];
            }
        }
#pragma unroll
        for (int a = 0; a < D; ++a) g[a][0] = T[a];
    } else {
        const double lam = f[0], mu = f[1];
        const double* G = f + 2;
        double J[D][D];
#pragma unroll
        for (int s = 0; s < D; ++s)
#pragma unroll
            for (int r = 0; r < D; ++r) {
                J[s][r] = 0.0;
#pragma unroll
                for (int a = 0; a < D; ++a) J[s][r] += G[a * D + s] * g[a][r];
            }
        double div = 0.0;
#pragma unroll
        for (int r = 0; r < D; ++r) div += J[r][r];
        div *= lam;
#pragma unroll
        for (int r = 0; r < D; ++r) {
            double sg[D];
#pragma unroll
            for (int j = 0; j < D; ++j) sg[j] = mu * (J[r][j] + J[j][r]) + (r == j ? div : 0.0);
#pragma unroll
            for (int a = 0; a < D; ++a) {
                double s = 0.0;
#pragma unroll
                for (int j = 0; j < D; ++j) s += G[a * D + j] * sg[j];
                g[a][r] = s;
            }
        }
    }
}

// One block of volume points: gradients, stress and the back-projection into y.
template <class S, int H, bool TG>
__device__ __forceinline__ void volume_block(Frags<TG> fwd, Frags<TG> bwd, const double (&u)[S::Q][WarpTile<S>::KS],
                                             const double* __restrict__ gp, int lane,
                                             double (&y)[S::Q][WarpTile<S>::NT][2]) {
    using L = WarpTile<S>;
    constexpr int D = S::D, Q = S::Q, NK = H == 2 ? D : L::VPAIR;
    double gf[L::VF][H];
#pragma unroll
    for (int f = 0; f < L::VF; ++f) geo_field<H>(gp, f, lane, gf[f]);
    double acc[NK][Q][2];
#pragma unroll
    for (int c = 0; c < NK; ++c)
#pragma unroll
        for (int r = 0; r < Q; ++r) acc[c][r][0] = acc[c][r][1] = 0.0;
#pragma unroll
    for (int ks = 0; ks < L::KS; ++ks)
#pragma unroll
        for (int c = 0; c < NK; ++c) {
            const double b = fwd(c * L::KS + ks);
#pragma unroll
            for (int r = 0; r < Q; ++r) dmma(acc[c][r], u[r][ks], b);
        }
#pragma unroll
    for (int h = 0; h < H; ++h) {
        double g[D][Q], f[L::VF];
#pragma unroll
        for (int i = 0; i < L::VF; ++i) f[i] = gf[i][h];
#pragma unroll
        for (int a = 0; a < D; ++a)
#pragma unroll
            for (int r = 0; r < Q; ++r) g[a][r] = H == 2 ? acc[a][r][h] : acc[a / 2][r][a % 2];
        volume_flux<S>(f, g);
#pragma unroll
        for (int a = 0; a < D; ++a)
#pragma unroll
            for (int nt = 0; nt < L::NT; ++nt) {
                const double b = bwd((h * D + a) * L::NT + nt);
#pragma unroll
                for (int r = 0; r < Q; ++r) dmma(y[r][nt], g[a][r], b);
            }
    }
}

// Doubles of shared memory per warp of the volume kernel: a split item's partial result.
template <class S>
__host__ __device__ constexpr int volume_warp_doubles() {
    return S::Q * WarpTile<S>::NT * 2 * 32;
}

// y = volume term, one warp per 8 consecutive elements; the split items' blocks are shared by
// `parts` warps of one CTA, whose partial results are summed in shared memory in part order.
template <class S, bool TG>
__global__ void __launch_bounds__(32 * WarpTile<S>::VWARPS, 1)
    volw_kernel(int64_t E, int Nq, WarpGeo wg, WarpSplit sp, const double* __restrict__ x, double* __restrict__ y,
                int64_t ld, int nrhs) {
    using L = WarpTile<S>;
    constexpr int D = S::D, NBF = S::NBF, Q = S::Q, BS = S::BS, YV = Q * L::NT * 2, WD = volume_warp_doubles<S>();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nwarp = blockDim.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const WarpBlocks blk(Nq);
    const int frags = warp_volume_frags<S>(Nq), nblk = blk.count();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* sm = reinterpret_cast<double*>(smem_raw);
    double* red = sm + (TG ? 0 : frags * 32) + lane;  // partial results of the warps, at this lane
    __shared__ __align__(8) unsigned long long s_bar;
    let_next_kernel_start();
    if constexpr (!TG) {
        if (!load_tables(sm, wg.vtab, frags * 32, &s_bar, wg.status)) return;
    }
    const Frags<TG> fwd{(TG ? wg.vtab : sm) + lane};
    const Frags<TG> bwd = fwd + (blk.full * D * L::KS + blk.half * L::VPAIR * L::KS);
    const int gstride = blk.full * L::VF * 64 + blk.half * L::VF * 32;
    const int64_t ntiles = (E + 7) / 8, nwork = ntiles * nrhs;
    // whole items are a multiple of the grid's warps, so every warp of a CTA makes the same number of
    // rounds; a round of split items holds `teams` per CTA
    const int64_t rounds = sp.whole / (static_cast<int64_t>(nwarp) * gridDim.x);
    const int teams = nwarp / sp.parts, team = warp / sp.parts, part = warp - team * sp.parts;
    const int64_t per_round = static_cast<int64_t>(teams) * gridDim.x;
    const int64_t total = rounds + (nwork > sp.whole ? (nwork - sp.whole + per_round - 1) / per_round : 0);
    for (int64_t rd = 0; rd < total; ++rd) {
        const bool split = rd >= rounds;
        int64_t work;
        int b0 = 0, b1 = nblk;
        if (!split) {
            work = (rd * nwarp + warp) * gridDim.x + blockIdx.x;
        } else {
            work = team < teams ? sp.whole + ((rd - rounds) * teams + team) * gridDim.x + blockIdx.x : nwork;
            b0 = part * nblk / sp.parts;
            b1 = (part + 1) * nblk / sp.parts;
        }
        const bool mine = work < nwork;
        int64_t tile = 0, rhs = 0;
        if (mine) work_tile_rhs(work, ntiles, nrhs, tile, rhs);
        const int64_t e = tile * 8 + g;
        double yac[Q][L::NT][2];
#pragma unroll
        for (int r = 0; r < Q; ++r)
#pragma unroll
            for (int nt = 0; nt < L::NT; ++nt) yac[r][nt][0] = yac[r][nt][1] = 0.0;
        if (mine) {
            const double* xe = x + rhs * ld + (e < E ? e : E - 1) * BS;
            const double* geo = wg.vol + tile * gstride;
            double u[Q][L::KS];
#pragma unroll
            for (int ks = 0; ks < L::KS; ++ks) {
                const int k = 4 * ks + t;
#pragma unroll
                for (int r = 0; r < Q; ++r) u[r][ks] = k < NBF ? __ldg(xe + r * NBF + k) : 0.0;
            }
            for (int b = b0; b < b1 && b < blk.full; ++b)
                volume_block<S, 2, TG>(fwd + b * D * L::KS, bwd + 2 * b * D * L::NT, u, geo + b * (L::VF * 64), lane,
                                       yac);
            if (b1 > blk.full)
                volume_block<S, 1, TG>(fwd + blk.full * D * L::KS, bwd + 2 * blk.full * D * L::NT, u,
                                       geo + blk.full * (L::VF * 64), lane, yac);
        }
        double* ye = y + rhs * ld + e * BS;
        if (!split) {
            if (mine && e < E) {
#pragma unroll
                for (int nt = 0; nt < L::NT; ++nt)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int k = nt * 8 + h * 4 + t;
                        if (k < NBF)
#pragma unroll
                            for (int r = 0; r < Q; ++r) ye[r * NBF + k] = yac[r][nt][h];
                    }
            }
        } else {
#pragma unroll
            for (int r = 0; r < Q; ++r)
#pragma unroll
                for (int nt = 0; nt < L::NT; ++nt)
#pragma unroll
                    for (int h = 0; h < 2; ++h) red[warp * WD + ((r * L::NT + nt) * 2 + h) * 32] = yac[r][nt][h];
            __syncthreads();
            if (mine && e < E)
                for (int v = part; v < YV; v += sp.parts) {
                    double s = 0.0;
                    for (int p = 0; p < sp.parts; ++p) s += red[(team * sp.parts + p) * WD + v * 32];
                    const int k = (v / 2 % L::NT) * 8 + (v % 2) * 4 + t;
                    if (k < NBF) ye[v / (2 * L::NT) * NBF + k] = s;
                }
            __syncthreads();
        }
    }
}

}  // namespace tdg
