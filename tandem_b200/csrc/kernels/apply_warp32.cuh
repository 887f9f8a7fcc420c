// Warp-tile FP32 apply: the kernels of apply_warp.cuh on mma.sync m16n8k8 with TF32 operands in the
// 3xTF32 form (apply_tc32.cuh; NP = 1: one TF32 pass, for preconditioner applies).  A warp carries 16
// elements or facets: rows g and g + 8 of an accumulator are the tile's slots g and g + 8, its
// columns 2t and 2t + 1 the two points of a lane, and a forward accumulator {c0, c1, c2, c3} is the
// backward product's A fragment {a0, a2, a1, a3} (k index t = point 2t, t + 4 = point 2t + 1).
// TX is the vectors' type: float, or double (x rounded to FP32 on load, y accumulated in FP64).
//
// Bound by the latency of dependent products, splits and flux arithmetic at the 8 to 16 warps per SM that
// 255 registers leave: at 3D p4 elasticity, 24,576 tetrahedra a third of the issue slots is used, the tensor
// pipe is busy 43 % (volume) and 24 % (facets) and DRAM 14 %.  Measured on a B200, FP32 vectors, against
// the tile products of a whole CTA behind the tcgen05 volume kernel that stood here before: the same case
// 172 us (volume 64, facets 115, overlapping; before 242: 82 and 160); 3D p2 elasticity, 7,986
// tetrahedra 16.7 us (39.2); 3D p3 Poisson, 10,368 tetrahedra 18.7 us (53.0); 2D p4 Poisson, 32
// right-hand sides on 17,712 triangles 159 us (590).
#pragma once

#include "apply_tc32.cuh"
#include "apply_warp.cuh"

namespace tdg {

template <class S>
struct WarpTile32 {
    using L64 = WarpTile<S>;
    static constexpr int NT = L64::NT, NTS = L64::NTS;  // n tiles of 8, and k steps of 8: all functions / face functions
    static constexpr int VF = L64::VF, SF = L64::SF, CF = L64::CF, FF = L64::FF;
    static constexpr int FWD = S::D * NTS + NT, FWD_HALF = NTS + NT;  // fragments of a block of facet points
    static constexpr int BWD = S::D * NTS + NT;                       // of a backward step (8 points, or 4 of a half block)
    static constexpr int VPAIR = L64::VPAIR;
    static constexpr int WARPS = S::Q == 3 ? (S::N >= 3 ? 8 : 12) : (S::D == 3 && S::N >= 3 ? 12 : 16);
};

// Device data (host/warp_tables.cpp).
struct WarpGeo32 {
    const float* ftab = nullptr;  // facet fragments per table, [fragment][lane][2]
    int face_tables = 0;
    const int* fperm = nullptr;   // as WarpGeo
    const float* fct = nullptr;   // facet geometry per tile of 16, [block][field][lane][row, point]
    const double* pen = nullptr;  // [tile][16] penalties
    const int4* ftiles = nullptr;
    const int4* tids = nullptr;   // [tile][16]
    int nftiles = 0;
    const float* vtab = nullptr;
    const float* vol = nullptr;   // per tile of 16 consecutive elements
    int* status = nullptr;
};

template <class S>
__host__ __device__ inline int warp32_facet_frags(int nq) {
    using L = WarpTile32<S>;
    const WarpBlocks b(nq);
    return b.full * L::FWD + b.half * L::FWD_HALF + b.count() * L::BWD;
}
template <class S>
__host__ __device__ inline int warp32_volume_frags(int Nq) {
    using L = WarpTile32<S>;
    const WarpBlocks b(Nq);
    return b.full * S::D * L::NT + b.half * L::VPAIR * L::NT + b.count() * S::D * L::NT;
}

// c += A B with A 16 x 4, B 4 x 8 (the four points of a half block).
__device__ __forceinline__ void mma_tf32_k4(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    asm volatile(
        "mma.sync.aligned.m16n8k4.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(b0));
}

// A and B fragments split into TF32 high and low parts.
struct SplitA {
    uint32_t h[4], l[4];
    __device__ __forceinline__ void set(int i, float v) { tf32_split(v, h[i], l[i]); }
};
struct SplitB {
    uint32_t h[2], l[2];
    __device__ __forceinline__ void set(float2 v) {
        tf32_split(v.x, h[0], l[0]);
        tf32_split(v.y, h[1], l[1]);
    }
};

// acc[c][r] += a[r] b[c] over all c < NC, r < Q, the products of one accumulator apart (small terms
// first).  K4: only k = 0..3 (a[.][0], a[.][1] and b[0]).  The tensor core truncates the accumulator
// it adds to, so the large products start from zero and are added here, rounded to nearest: 2.1e-7 ->
// 1.6e-7 against the FP64 apply at 3D p4 elasticity for no time.
template <int NP, bool K4, int NC, int Q, int NA>
__device__ __forceinline__ void mma_set(float (&acc)[NA][Q][4], int c0, const SplitA (&a)[Q], const SplitB (&b)[NC]) {
    const auto one = [&](float (&d)[4], const uint32_t (&x)[4], const uint32_t (&y)[2]) {
        if constexpr (K4)
            mma_tf32_k4(d, x[0], x[1], y[0]);
        else
            mma_tf32(d, x, y[0], y[1]);
    };
    if constexpr (NP == 3) {
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
            for (int r = 0; r < Q; ++r) one(acc[c0 + c][r], a[r].l, b[c].h);
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
            for (int r = 0; r < Q; ++r) one(acc[c0 + c][r], a[r].h, b[c].l);
    }
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        float d[Q][4] = {};
#pragma unroll
        for (int r = 0; r < Q; ++r) one(d[r], a[r].h, b[c].h);
#pragma unroll
        for (int r = 0; r < Q; ++r)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[c0 + c][r][i] += d[r][i];
    }
}

// The small products of the same alone.
template <bool K4, int NC, int Q, int NA>
__device__ __forceinline__ void mma_low(float (&acc)[NA][Q][4], const SplitA (&a)[Q], const SplitB (&b)[NC]) {
    const auto one = [&](float (&d)[4], const uint32_t (&x)[4], const uint32_t (&y)[2]) {
        if constexpr (K4)
            mma_tf32_k4(d, x[0], x[1], y[0]);
        else
            mma_tf32(d, x, y[0], y[1]);
    };
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int r = 0; r < Q; ++r) one(acc[c][r], a[r].l, b[c].h);
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int r = 0; r < Q; ++r) one(acc[c][r], a[r].h, b[c].l);
}

template <bool TG>
struct Frags32 {
    const float2* p;  // at this lane
    __device__ __forceinline__ float2 operator()(int f) const {
        if constexpr (TG)
            return __ldg(p + f * 32);
        else
            return p[f * 32];
    }
    __device__ __forceinline__ Frags32 operator+(int f) const { return {p + f * 32}; }
};

// Coefficients of the tile as A fragments: u[r][ks][i], i = 0..3: (row g, k = 8 ks + t), (g + 8, t),
// (g, t + 4), (g + 8, t + 4).
template <class S>
using Coef32 = float[S::Q][WarpTile32<S>::NT][4];

// Field f of a block at this lane: rows g, g + 8 at its H points.
template <int H>
__device__ __forceinline__ void geo_field32(const float* __restrict__ gp, int f, int lane, float (&v)[2][2]) {
    if constexpr (H == 2) {
        const float4 d = __ldg(reinterpret_cast<const float4*>(gp + f * 128) + lane);
        v[0][0] = d.x;
        v[0][1] = d.y;
        v[1][0] = d.z;
        v[1][1] = d.w;
    } else {
        const float2 d = __ldg(reinterpret_cast<const float2*>(gp + f * 64) + lane);
        v[0][0] = d.x;
        v[1][0] = d.y;
    }
}

template <class S>
__device__ __forceinline__ void facet_traction32(const float* cf, const float* sf, const float (&tr)[S::D + 1][S::Q],
                                                 float (&tq)[S::Q]) {
    constexpr int D = S::D;
    if constexpr (S::KIND == kPoisson) {
        float s = 0.0f;
#pragma unroll
        for (int a = 0; a < D; ++a) s += sf[a] * tr[1 + a][0];
        tq[0] = s;
    } else {
        const float lam = sf[0], mu = sf[1];
        const float* G = sf + 2;
        float nb[D], hb[D], div = 0.0f;
#pragma unroll
        for (int b = 0; b < D; ++b) {
            nb[b] = hb[b] = 0.0f;
#pragma unroll
            for (int j = 0; j < D; ++j) {
                nb[b] += G[b * D + j] * cf[j];
                hb[b] += tr[1 + b][j] * cf[j];
                div += G[b * D + j] * tr[1 + b][j];
            }
        }
#pragma unroll
        for (int r = 0; r < D; ++r) {
            float s = 0.0f;
#pragma unroll
            for (int b = 0; b < D; ++b) s += nb[b] * tr[1 + b][r] + G[b * D + r] * hb[b];
            tq[r] = lam * div * cf[r] + mu * s;
        }
    }
}

template <class S>
__device__ __forceinline__ void facet_lift_rows32(const float* cf, const float* sf, const float (&uh)[S::Q],
                                                  float (&ga)[S::D][S::Q]) {
    constexpr int D = S::D;
    if constexpr (S::KIND == kPoisson) {
#pragma unroll
        for (int a = 0; a < D; ++a) ga[a][0] = uh[0] * sf[a];
    } else {
        const float mu = sf[1];
        const float* G = sf + 2;
        float un = 0.0f;
#pragma unroll
        for (int j = 0; j < D; ++j) un += uh[j] * cf[j];
        un *= sf[0];
#pragma unroll
        for (int b = 0; b < D; ++b) {
            float nb = 0.0f, vb = 0.0f;
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

// Phase 1 of a facet block (facet_phase1 of apply_warp.cuh): pen[row] the penalties, whose product
// with the jump is formed in FP64 and rounded once; the shared field holds weight x |n|.
template <class S, int H, int NP, bool TG>
__device__ __forceinline__ void facet32_phase1(Frags32<TG> tab, const Coef32<S>& u, const float* __restrict__ gp,
                                               int side, int lane, int mode, const double (&pen)[2], float* stash) {
    using L = WarpTile32<S>;
    constexpr int D = S::D, Q = S::Q, NK = H == 2 ? D + 1 : 2, NS = NK - 1;
    float cf[L::CF][2][2], sf[L::SF][2][2];
#pragma unroll
    for (int f = 0; f < L::CF; ++f) geo_field32<H>(gp, (side ? 0 : L::SF) + f, lane, cf[f]);
#pragma unroll
    for (int f = 0; f < L::SF; ++f) geo_field32<H>(gp, (side ? L::CF : 0) + f, lane, sf[f]);
    float acc[NK][Q][4];
#pragma unroll
    for (int c = 0; c < NK; ++c)
#pragma unroll
        for (int r = 0; r < Q; ++r) acc[c][r][0] = acc[c][r][1] = acc[c][r][2] = acc[c][r][3] = 0.0f;
#pragma unroll
    for (int ks = 0; ks < L::NT; ++ks) {
        SplitA a[Q];
#pragma unroll
        for (int r = 0; r < Q; ++r)
#pragma unroll
            for (int i = 0; i < 4; ++i) a[r].set(i, u[r][ks][i]);
        SplitB bd[1];
        bd[0].set(tab(NS * L::NTS + ks));
        if (ks < L::NTS) {  // the face functions' kinds
            SplitB bs[NS];
#pragma unroll
            for (int c = 0; c < NS; ++c) bs[c].set(tab(c * L::NTS + ks));
            mma_set<NP, false, NS, Q>(acc, 0, a, bs);
        }
        mma_set<NP, false, 1, Q>(acc, NS, a, bd);
    }
#pragma unroll
    for (int row = 0; row < 2; ++row)
#pragma unroll
        for (int h = 0; h < H; ++h) {
            float c[L::CF], s[L::SF], tr[D + 1][Q], tq[Q];
#pragma unroll
            for (int f = 0; f < L::CF; ++f) c[f] = cf[f][row][h];
#pragma unroll
            for (int f = 0; f < L::SF; ++f) s[f] = sf[f][row][h];
#pragma unroll
            for (int k = 0; k <= D; ++k)
#pragma unroll
                for (int r = 0; r < Q; ++r) tr[k][r] = H == 2 ? acc[k][r][row * 2 + h] : acc[k / 2][r][row * 2 + k % 2];
            facet_traction32<S>(c, s, tr, tq);
            const float wn = c[L::CF - 1];
            float* st = stash + (h * 2 + row) * 2 * Q * 32 + lane;
#pragma unroll
            for (int r = 0; r < Q; ++r) {
                const float u0 = tr[0][r];
                if (side) {
                    st[r * 32] = u0;
                    st[(Q + r) * 32] = tq[r];
                } else if (mode == 1) {
                    const float u1 = st[r * 32], t1 = st[(Q + r) * 32];
                    const float pj = static_cast<float>(pen[row] * (static_cast<double>(u0) - static_cast<double>(u1)));
                    st[r * 32] = -(0.5f * (tq[r] + t1) - wn * pj);
                    st[(Q + r) * 32] = 0.5f * (u1 - u0);
                } else if (mode == 2) {
                    st[r * 32] = -(tq[r] - wn * static_cast<float>(pen[row] * static_cast<double>(u0)));
                    st[(Q + r) * 32] = -u0;
                } else {
                    st[r * 32] = -tq[r];
                    st[(Q + r) * 32] = 0.0f;
                }
            }
        }
}

// Phase 2 of a facet block: the gradient rows of one side's lift-back.
template <class S, int H, int NP, bool TG>
__device__ __forceinline__ void facet32_gradients(Frags32<TG> tab, const float* __restrict__ gp, int side, int lane,
                                                  const float* stash, float (&y)[WarpTile32<S>::NT][S::Q][4]) {
    using L = WarpTile32<S>;
    constexpr int D = S::D, Q = S::Q;
    float cf[L::CF][2][2], sf[L::SF][2][2];
#pragma unroll
    for (int f = 0; f + 1 < L::CF; ++f) geo_field32<H>(gp, (side ? 0 : L::SF) + f, lane, cf[f]);
#pragma unroll
    for (int f = 0; f < L::SF; ++f) geo_field32<H>(gp, (side ? L::CF : 0) + f, lane, sf[f]);
    float ga[D][Q][4];  // A fragment entry of (row, point h): i = row + 2 h
#pragma unroll
    for (int row = 0; row < 2; ++row)
#pragma unroll
        for (int h = 0; h < H; ++h) {
            float c[L::CF], s[L::SF], uh[Q], gr[D][Q];
#pragma unroll
            for (int f = 0; f + 1 < L::CF; ++f) c[f] = cf[f][row][h];
#pragma unroll
            for (int f = 0; f < L::SF; ++f) s[f] = sf[f][row][h];
            const float* st = stash + (h * 2 + row) * 2 * Q * 32 + lane;
#pragma unroll
            for (int r = 0; r < Q; ++r) uh[r] = st[(Q + r) * 32];
            facet_lift_rows32<S>(c, s, uh, gr);
#pragma unroll
            for (int k = 0; k < D; ++k)
#pragma unroll
                for (int r = 0; r < Q; ++r) ga[k][r][row + 2 * h] = gr[k][r];
        }
#pragma unroll
    for (int k = 0; k < D; ++k) {
        SplitA a[Q];
#pragma unroll
        for (int r = 0; r < Q; ++r)
#pragma unroll
            for (int i = 0; i < 2 * H; ++i) a[r].set(i, ga[k][r][i]);
        if (k + 1 < D) {  // the tangential rows act on the face functions
            SplitB b[L::NTS];
#pragma unroll
            for (int n = 0; n < L::NTS; ++n) b[n].set(tab((k + 1) * L::NTS + n));
            mma_set<NP, H == 1, L::NTS, Q>(y, 0, a, b);
        } else {
            SplitB b[L::NT];
#pragma unroll
            for (int n = 0; n < L::NT; ++n) b[n].set(tab(D * L::NTS + n));
            mma_set<NP, H == 1, L::NT, Q>(y, 0, a, b);
        }
    }
}

// The value rows of the lift-back, after every block's gradient rows: they hold the penalty and are
// the largest, and each product truncates the accumulator it adds to, so what comes after them costs
// accuracy (values first in each block: 8.1e-7 against the FP64 apply at 3D p4 elasticity, 24,576
// tetrahedra).  low: the small products of the split, else the high ones.
template <class S, int H, int NP, bool TG>
__device__ __forceinline__ void facet32_values(Frags32<TG> tab, int side, int lane, bool low, const float* stash,
                                               float (&y)[WarpTile32<S>::NT][S::Q][4]) {
    using L = WarpTile32<S>;
    constexpr int Q = S::Q;
    SplitA a[Q];
#pragma unroll
    for (int row = 0; row < 2; ++row)
#pragma unroll
        for (int h = 0; h < H; ++h)
#pragma unroll
            for (int r = 0; r < Q; ++r) {
                const float v = stash[((h * 2 + row) * 2 * Q + r) * 32 + lane];
                a[r].set(row + 2 * h, side ? -v : v);
            }
    SplitB b[L::NTS];
#pragma unroll
    for (int n = 0; n < L::NTS; ++n) b[n].set(tab(n));
    if (low)
        mma_low<H == 1, L::NTS, Q>(y, a, b);
    else
        mma_set<1, H == 1, L::NTS, Q>(y, 0, a, b);
}

template <class S>
__host__ __device__ inline int facet32_warp_floats(int nq) {  // stash of a warp
    return WarpBlocks(nq).steps() * 2 * 2 * S::Q * 32;
}

// One warp per tile of 16 facets of one (l0, l1, mode); see facew_kernel.
template <class S, typename TX, int NP, bool TG>
__global__ void __launch_bounds__(32 * WarpTile32<S>::WARPS, 1)
    facew32_kernel(int nq, WarpGeo32 wg, WarpSplit sp, const TX* __restrict__ x, TX* __restrict__ y, int64_t ld,
                   int nrhs) {
    using L = WarpTile32<S>;
    constexpr int NBF = S::NBF, Q = S::Q, BS = S::BS, NF = S::NF, NPM = 8 * L::NT;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nwarp = blockDim.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const WarpBlocks blk(nq);
    const int frags = warp32_facet_frags<S>(nq);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float* sm = reinterpret_cast<float*>(smem_raw);
    __shared__ int s_perm[NF * NPM];
    __shared__ __align__(8) unsigned long long s_bar;
    const int tabsz = TG ? 0 : wg.face_tables * frags * 64;
    const int fstride = wg.face_tables == 1 ? 0 : frags;
    let_next_kernel_start();
    float* stash = sm + tabsz + warp * facet32_warp_floats<S>(nq);
    for (int i = tid; i < NF * NPM; i += blockDim.x) s_perm[i] = wg.fperm[i];
    if constexpr (!TG) {
        if (!load_tables(reinterpret_cast<double*>(sm), reinterpret_cast<const double*>(wg.ftab), tabsz / 2, &s_bar,
                         wg.status))
            return;
    } else {
        __syncthreads();
    }
    const Frags32<TG> tab0{reinterpret_cast<const float2*>(TG ? wg.ftab : sm) + lane};
    const int gstride = blk.full * L::FF * 128 + blk.half * L::FF * 64;
    const int nblk = blk.count();
    const int64_t nitems = sp.whole + (static_cast<int64_t>(wg.nftiles) * nrhs - sp.whole) * nblk;
    const int64_t stride = static_cast<int64_t>(nwarp) * gridDim.x;
    bool waited = false;
    for (int64_t item = static_cast<int64_t>(warp) * gridDim.x + blockIdx.x; item < nitems; item += stride) {
        int64_t work = item, tile, rhs;
        int b0 = 0, b1 = nblk;
        if (item >= sp.whole) {
            const int64_t part = item - sp.whole;
            work = sp.whole + part / nblk;
            b0 = static_cast<int>(part % nblk);
            b1 = b0 + 1;
        }
        work_tile_rhs(work, wg.nftiles, nrhs, tile, rhs);
        const int key = __ldg(&wg.ftiles[tile].z);
        const int4 id0 = __ldg(&wg.tids[tile * 16 + g]), id1 = __ldg(&wg.tids[tile * 16 + g + 8]);
        const double pen[2] = {__ldg(&wg.pen[tile * 16 + g]), __ldg(&wg.pen[tile * 16 + g + 8])};
        const int mode = key >> 4;
        const bool two = mode == 1;
        const int bf = b1 < blk.full ? b1 : blk.full;
        const bool bh = b1 > blk.full;
        const TX* xr = x + rhs * ld;
        TX* yr = y + rhs * ld;
        const float* geo = wg.fct + tile * gstride;
        const auto side_geo = [&](int side, int b) {
            return geo + b * (L::FF * 128) + (side ? L::SF * (b < blk.full ? 128 : 64) : 0);
        };
        for (int side = two ? 1 : 0; side >= 0; --side) {
            const int l = side ? (key >> 2) & 3 : key & 3;
            const TX* x0 = xr + static_cast<int64_t>(id0.x < 0 ? 0 : (side ? id0.z : id0.y)) * BS;
            const TX* x1 = xr + static_cast<int64_t>(id1.x < 0 ? 0 : (side ? id1.z : id1.y)) * BS;
            Coef32<S> u;
#pragma unroll
            for (int ks = 0; ks < L::NT; ++ks)
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const int k = s_perm[l * NPM + 8 * ks + 4 * j + t];
#pragma unroll
                    for (int r = 0; r < Q; ++r) {
                        u[r][ks][2 * j] = k >= 0 ? static_cast<float>(__ldg(x0 + r * NBF + k)) : 0.0f;
                        u[r][ks][2 * j + 1] = k >= 0 ? static_cast<float>(__ldg(x1 + r * NBF + k)) : 0.0f;
                    }
                }
            const Frags32<TG> tab = tab0 + l * fstride;
            for (int b = b0; b < bf; ++b)
                facet32_phase1<S, 2, NP, TG>(tab + b * L::FWD, u, side_geo(side, b), side, lane, mode, pen,
                                             stash + b * (8 * Q * 32));
            if (bh)
                facet32_phase1<S, 1, NP, TG>(tab + blk.full * L::FWD, u, side_geo(side, blk.full), side, lane, mode, pen,
                                             stash + blk.full * (8 * Q * 32));
        }
        for (int side = 0; side <= (two ? 1 : 0); ++side) {
            const int l = side ? (key >> 2) & 3 : key & 3;
            const Frags32<TG> tab = tab0 + (l * fstride + blk.full * L::FWD + blk.half * L::FWD_HALF);
            float yac[L::NT][Q][4];
#pragma unroll
            for (int n = 0; n < L::NT; ++n)
#pragma unroll
                for (int r = 0; r < Q; ++r) yac[n][r][0] = yac[n][r][1] = yac[n][r][2] = yac[n][r][3] = 0.0f;
            for (int b = b0; b < bf; ++b)
                facet32_gradients<S, 2, NP, TG>(tab + b * L::BWD, side_geo(side, b), side, lane,
                                                stash + b * (8 * Q * 32), yac);
            if (bh)
                facet32_gradients<S, 1, NP, TG>(tab + blk.full * L::BWD, side_geo(side, blk.full), side, lane,
                                                stash + blk.full * (8 * Q * 32), yac);
            for (int low = NP == 3 ? 1 : 0; low >= 0; --low) {
                for (int b = b0; b < bf; ++b)
                    facet32_values<S, 2, NP, TG>(tab + b * L::BWD, side, lane, low != 0, stash + b * (8 * Q * 32), yac);
                if (bh)
                    facet32_values<S, 1, NP, TG>(tab + blk.full * L::BWD, side, lane, low != 0,
                                                 stash + blk.full * (8 * Q * 32), yac);
            }
            if (!waited) wait_for_previous_kernel();
            waited = true;
            TX* y0 = yr + static_cast<int64_t>(side ? id0.z : id0.y) * BS;
            TX* y1 = yr + static_cast<int64_t>(side ? id1.z : id1.y) * BS;
#pragma unroll
            for (int n = 0; n < L::NT; ++n)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int k = s_perm[l * NPM + n * 8 + h * 4 + t];
                    if (k < 0) continue;
#pragma unroll
                    for (int r = 0; r < Q; ++r) {
                        if (id0.x >= 0) atomicAdd(y0 + r * NBF + k, static_cast<TX>(yac[n][r][h]));
                        if (id1.x >= 0) atomicAdd(y1 + r * NBF + k, static_cast<TX>(yac[n][r][2 + h]));
                    }
                }
        }
    }
}

// ---- volume term -------------------------------------------------------------------------------------

template <class S>
__device__ __forceinline__ void volume_flux32(const float* f, float (&g)[S::D][S::Q]) {
    constexpr int D = S::D;
    if constexpr (S::KIND == kPoisson) {
        float T[D];
#pragma unroll
        for (int a = 0; a < D; ++a) {
            T[a] = 0.0f;
#pragma unroll
            for (int b = 0; b < D; ++b) {
                const int i = a < b ? a : b, j = a < b ? b : a;
                T[a] += f[i * D - i * (i - 1) / 2 + j - i] * g[b][0];
            }
        }
#pragma unroll
        for (int a = 0; a < D; ++a) g[a][0] = T[a];
    } else {
        const float lam = f[0], mu = f[1];
        const float* G = f + 2;
        float J[D][D];
#pragma unroll
        for (int s = 0; s < D; ++s)
#pragma unroll
            for (int r = 0; r < D; ++r) {
                J[s][r] = 0.0f;
#pragma unroll
                for (int a = 0; a < D; ++a) J[s][r] += G[a * D + s] * g[a][r];
            }
        float div = 0.0f;
#pragma unroll
        for (int r = 0; r < D; ++r) div += J[r][r];
        div *= lam;
#pragma unroll
        for (int r = 0; r < D; ++r) {
            float sg[D];
#pragma unroll
            for (int j = 0; j < D; ++j) sg[j] = mu * (J[r][j] + J[j][r]) + (r == j ? div : 0.0f);
#pragma unroll
            for (int a = 0; a < D; ++a) {
                float s = 0.0f;
#pragma unroll
                for (int j = 0; j < D; ++j) s += G[a * D + j] * sg[j];
                g[a][r] = s;
            }
        }
    }
}

template <class S, int H, int NP, bool TG>
__device__ __forceinline__ void volume32_block(Frags32<TG> fwd, Frags32<TG> bwd, const Coef32<S>& u,
                                               const float* __restrict__ gp, int lane,
                                               float (&y)[WarpTile32<S>::NT][S::Q][4]) {
    using L = WarpTile32<S>;
    constexpr int D = S::D, Q = S::Q, NK = H == 2 ? D : L::VPAIR;
    float gf[L::VF][2][2];
#pragma unroll
    for (int f = 0; f < L::VF; ++f) geo_field32<H>(gp, f, lane, gf[f]);
    float acc[NK][Q][4];
#pragma unroll
    for (int c = 0; c < NK; ++c)
#pragma unroll
        for (int r = 0; r < Q; ++r) acc[c][r][0] = acc[c][r][1] = acc[c][r][2] = acc[c][r][3] = 0.0f;
#pragma unroll
    for (int ks = 0; ks < L::NT; ++ks) {
        SplitA a[Q];
        SplitB b[NK];
#pragma unroll
        for (int r = 0; r < Q; ++r)
#pragma unroll
            for (int i = 0; i < 4; ++i) a[r].set(i, u[r][ks][i]);
#pragma unroll
        for (int c = 0; c < NK; ++c) b[c].set(fwd(c * L::NT + ks));
        mma_set<NP, false, NK, Q>(acc, 0, a, b);
    }
    float T[D][Q][4];  // A fragment entry of (row, point h): i = row + 2 h
#pragma unroll
    for (int row = 0; row < 2; ++row)
#pragma unroll
        for (int h = 0; h < H; ++h) {
            float g[D][Q], f[L::VF];
#pragma unroll
            for (int i = 0; i < L::VF; ++i) f[i] = gf[i][row][h];
#pragma unroll
            for (int a = 0; a < D; ++a)
#pragma unroll
                for (int r = 0; r < Q; ++r) g[a][r] = H == 2 ? acc[a][r][row * 2 + h] : acc[a / 2][r][row * 2 + a % 2];
            volume_flux32<S>(f, g);
#pragma unroll
            for (int a = 0; a < D; ++a)
#pragma unroll
                for (int r = 0; r < Q; ++r) T[a][r][row + 2 * h] = g[a][r];
        }
#pragma unroll
    for (int k = 0; k < D; ++k) {
        SplitA a[Q];
        SplitB b[L::NT];
#pragma unroll
        for (int r = 0; r < Q; ++r)
#pragma unroll
            for (int i = 0; i < 2 * H; ++i) a[r].set(i, T[k][r][i]);
#pragma unroll
        for (int n = 0; n < L::NT; ++n) b[n].set(bwd(k * L::NT + n));
        mma_set<NP, H == 1, L::NT, Q>(y, 0, a, b);
    }
}

template <class S>
__host__ __device__ constexpr int volume32_warp_floats() {  // a split item's partial result
    return S::Q * WarpTile32<S>::NT * 4 * 32;
}

// y = volume term, one warp per 16 consecutive elements; see volw_kernel.
template <class S, typename TX, int NP, bool TG>
__global__ void __launch_bounds__(32 * WarpTile32<S>::WARPS, 1)
    volw32_kernel(int64_t E, int Nq, WarpGeo32 wg, WarpSplit sp, const TX* __restrict__ x, TX* __restrict__ y,
                  int64_t ld, int nrhs) {
    using L = WarpTile32<S>;
    constexpr int D = S::D, NBF = S::NBF, Q = S::Q, BS = S::BS, YV = Q * L::NT * 4, WF = volume32_warp_floats<S>();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nwarp = blockDim.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const WarpBlocks blk(Nq);
    const int frags = warp32_volume_frags<S>(Nq), nblk = blk.count();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float* sm = reinterpret_cast<float*>(smem_raw);
    float* red = sm + (TG ? 0 : frags * 64) + lane;
    __shared__ __align__(8) unsigned long long s_bar;
    let_next_kernel_start();
    if constexpr (!TG) {
        if (!load_tables(reinterpret_cast<double*>(sm), reinterpret_cast<const double*>(wg.vtab), frags * 32, &s_bar,
                         wg.status))
            return;
    }
    const Frags32<TG> fwd{reinterpret_cast<const float2*>(TG ? wg.vtab : sm) + lane};
    const Frags32<TG> bwd = fwd + (blk.full * D * L::NT + blk.half * L::VPAIR * L::NT);
    const int gstride = blk.full * L::VF * 128 + blk.half * L::VF * 64;
    const int64_t ntiles = (E + 15) / 16, nwork = ntiles * nrhs;
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
        const int64_t e = tile * 16 + g;  // and e + 8
        float yac[L::NT][Q][4];
#pragma unroll
        for (int n = 0; n < L::NT; ++n)
#pragma unroll
            for (int r = 0; r < Q; ++r) yac[n][r][0] = yac[n][r][1] = yac[n][r][2] = yac[n][r][3] = 0.0f;
        if (mine) {
            const TX* x0 = x + rhs * ld + (e < E ? e : E - 1) * BS;
            const TX* x1 = x + rhs * ld + (e + 8 < E ? e + 8 : E - 1) * BS;
            const float* geo = wg.vol + tile * gstride;
            Coef32<S> u;
#pragma unroll
            for (int ks = 0; ks < L::NT; ++ks)
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const int k = 8 * ks + 4 * j + t;
#pragma unroll
                    for (int r = 0; r < Q; ++r) {
                        u[r][ks][2 * j] = k < NBF ? static_cast<float>(__ldg(x0 + r * NBF + k)) : 0.0f;
                        u[r][ks][2 * j + 1] = k < NBF ? static_cast<float>(__ldg(x1 + r * NBF + k)) : 0.0f;
                    }
                }
            for (int b = b0; b < b1 && b < blk.full; ++b)
                volume32_block<S, 2, NP, TG>(fwd + b * D * L::NT, bwd + b * D * L::NT, u, geo + b * (L::VF * 128), lane,
                                             yac);
            if (b1 > blk.full)
                volume32_block<S, 1, NP, TG>(fwd + blk.full * D * L::NT, bwd + blk.full * D * L::NT, u,
                                             geo + blk.full * (L::VF * 128), lane, yac);
        }
        TX* ye = y + rhs * ld + e * BS;
        if (!split) {
            if (mine) {
#pragma unroll
                for (int n = 0; n < L::NT; ++n)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int k = n * 8 + h * 4 + t;
                        if (k >= NBF) continue;
#pragma unroll
                        for (int r = 0; r < Q; ++r) {
                            if (e < E) ye[r * NBF + k] = static_cast<TX>(yac[n][r][h]);
                            if (e + 8 < E) ye[8 * BS + r * NBF + k] = static_cast<TX>(yac[n][r][2 + h]);
                        }
                    }
            }
        } else {
#pragma unroll
            for (int n = 0; n < L::NT; ++n)
#pragma unroll
                for (int r = 0; r < Q; ++r)
#pragma unroll
                    for (int i = 0; i < 4; ++i) red[warp * WF + ((n * Q + r) * 4 + i) * 32] = yac[n][r][i];
            __syncthreads();
            if (mine)
                for (int v = part; v < YV; v += sp.parts) {
                    float s = 0.0f;
                    for (int p = 0; p < sp.parts; ++p) s += red[(team * sp.parts + p) * WF + v * 32];
                    const int i = v % 4, r = v / 4 % Q, k = v / (4 * Q) * 8 + (i & 1) * 4 + t, up = i >> 1;
                    if (k < NBF && e + 8 * up < E) ye[up * 8 * BS + r * NBF + k] = static_cast<TX>(s);
                }
            __syncthreads();
        }
    }
}

}  // namespace tdg
