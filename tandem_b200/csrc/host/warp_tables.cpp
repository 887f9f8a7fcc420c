// Host-side data of the warp-tile FP64 apply (see warp_tables.hpp, kernels/apply_warp.cuh).
#include "warp_tables.hpp"

#include <algorithm>
#include <array>
#include <cmath>
#include <stdexcept>

namespace tdg {

namespace {

// Blocks of 8 points; a remainder of at most 4 takes a half block (WarpBlocks of apply_warp.cuh).
struct Blocks {
    int full, half;
    explicit Blocks(int n) : full(n / 8 + (n % 8 > 4 ? 1 : 0)), half(n % 8 >= 1 && n % 8 <= 4) {}
    int steps() const { return 2 * full + half; }
};

// Where the fields of point q of slot te (0..7) of a tile sit: offset of field 0 and the stride
// between fields.  Full blocks: lane te * 4 + t holds points 2t, 2t + 1 side by side.
struct Slot {
    int64_t base;
    int64_t stride;
};
Slot point_slot(Blocks const& b, int fields, int te, int q) {
    const int blk = q / 8;
    if (blk < b.full) {
        const int s = q % 8;
        return {static_cast<int64_t>(blk) * fields * 64 + (te * 4 + s / 2) * 2 + s % 2, 64};
    }
    return {static_cast<int64_t>(b.full) * fields * 64 + te * 4 + (q - 8 * b.full), 32};
}

// Streamed facet geometry (WarpTile::STREAM: 3D elasticity from degree 3) is read point by point
// from shared memory: [field][point of the pair][lane].
bool facet_streamed(HostOperator const& h) { return h.D == 3 && h.kind != 0 && h.N >= 3; }
Slot facet_slot(HostOperator const& h, Blocks const& b, int fields, int te, int q) {
    const int blk = q / 8;
    if (blk < b.full && facet_streamed(h)) {
        const int s = q % 8;
        return {static_cast<int64_t>(blk) * fields * 64 + (s % 2) * 32 + te * 4 + s / 2, 64};
    }
    return point_slot(b, fields, te, q);
}

int volume_fields(HostOperator const& h) { return h.kind == 0 ? h.D * (h.D + 1) / 2 : h.D * h.D + 2; }
int facet_fields(HostOperator const& h) {
    return h.kind == 0 ? 1 + 2 * h.D : h.D + 1 + 2 * (h.D * h.D + 2);
}

int opposite_vertex(int D, int f) {
    auto const fv = facet_vertices(D)[f];
    for (int v = 0; v <= D; ++v) {
        bool on = false;
        for (int i = 0; i < D; ++i) on = on || fv[i] == v;
        if (!on) return v;
    }
    return 0;
}

// Face-adapted reference directions of local face f: column b of T is direction b in reference
// coordinates -- the edges from the face's first vertex to its others, then the edge to the
// opposite vertex; Tinv its inverse (entries -1, 0, 1 for both).
void face_directions(int D, int f, double* T, double* Tinv) {
    auto const fv = facet_vertices(D)[f];
    const int opp = opposite_vertex(D, f);
    auto vert = [](int v, int c) { return v == c + 1 ? 1.0 : 0.0; };
    Dense M(D, D);
    for (int b = 0; b < D; ++b) {
        const int v = b + 1 < D ? fv[b + 1] : opp;
        for (int a = 0; a < D; ++a) M(a, b) = T[a * D + b] = vert(v, a) - vert(fv[0], a);
    }
    Dense I = invert(M);
    for (int b = 0; b < D; ++b)
        for (int a = 0; a < D; ++a) Tinv[b * D + a] = I(b, a);
}

// The basis on the faces: per face the order of its functions (face functions first) and the table
// [kind][k][q] -- kind 0 the value, kind 1 + b the derivative along direction b (nodal bases: the
// face-adapted directions).
struct FaceBasis {
    int FN = 0;             // functions with a trace on a face
    int tables = 0;         // 1: the faces share one table up to the order of the functions
    std::vector<int> perm;  // [face][NP], -1 beyond Nbf
    std::vector<std::vector<double>> tabs;
};

FaceBasis face_basis(HostOperator const& h) {
    const int D = h.D, NBF = h.Nbf, nq = h.nq, NF = h.nfaces, NP = (NBF + 7) / 8 * 8;
    const bool nodal = h.kind != 0;
    FaceBasis out;
    out.FN = NBF;
    if (nodal) {
        out.FN = 1;  // binom(N + D - 1, D - 1)
        for (int i = 1; i < D; ++i) out.FN = out.FN * (h.N + i) / i;
    }
    out.perm.assign(static_cast<size_t>(NF) * NP, -1);
    // Barycentric coordinates of node k with respect to face f's vertices, then the opposite one.
    auto bary = [&](int f, int k) {
        auto const fv = facet_vertices(D)[f];
        double const* z = &h.space.nodes()[static_cast<size_t>(k) * D];
        std::array<double, 4> b{};
        for (int i = 0; i <= D; ++i) {
            const int v = i < D ? fv[i] : opposite_vertex(D, f);
            b[i] = v ? z[v - 1] : 1.0;
            if (!v)
                for (int d = 0; d < D; ++d) b[i] -= z[d];
        }
        return b;
    };
    auto face_table = [&](int f) {
        std::vector<double> tab(static_cast<size_t>(D + 1) * NBF * nq);
        double T[9], Ti[9];
        face_directions(D, f, T, Ti);
        for (int k = 0; k < NBF; ++k)
            for (int q = 0; q < nq; ++q) {
                tab[static_cast<size_t>(k) * nq + q] = h.E_qf[f](k, q);
                for (int b = 0; b < D; ++b) {
                    double s = 0.0;
                    for (int a = 0; a < D; ++a)
                        s += (nodal ? T[a * D + b] : (a == b ? 1.0 : 0.0)) *
                             h.Dxi_qf[f][(static_cast<size_t>(k) * D + a) * nq + q];
                    tab[(static_cast<size_t>(1 + b) * NBF + k) * nq + q] = s;
                }
            }
        return tab;
    };
    // Order of the basis functions: those with a trace on the face first.  Nodal bases list every
    // face's functions by the position of their node relative to the face's vertices, so that one
    // table serves all faces (the node set and the directions are symmetric under a relabelling of
    // the vertices); without that symmetry each face keeps its own order and table.
    auto own_order = [&](int f, int* perm) {
        int n = 0;
        for (int pass = 0; pass < 2; ++pass)
            for (int k = 0; k < NBF; ++k)
                if ((!nodal || std::fabs(bary(f, k)[D]) < 1e-10) == (pass == 0)) perm[n++] = k;
    };
    auto matched_order = [&](int f, int const* first, int* perm) {
        for (int j = 0; j < NBF; ++j) {
            auto const want = bary(0, first[j]);
            perm[j] = -1;
            for (int k = 0; k < NBF; ++k) {
                auto const b = bary(f, k);
                double d = 0.0;
                for (int i = 0; i <= D; ++i) d = std::max(d, std::fabs(b[i] - want[i]));
                if (d < 1e-10) perm[j] = k;
            }
            if (perm[j] < 0) return false;
        }
        return true;
    };
    for (int f = 0; f < NF; ++f) out.tabs.push_back(face_table(f));
    auto entry = [&](int f, int kind, int k, int q) {
        return out.tabs[f][(static_cast<size_t>(kind) * NBF + k) * nq + q];
    };
    bool shared = nodal;
    own_order(0, &out.perm[0]);
    for (int f = 1; f < NF && shared; ++f) {
        int* perm = &out.perm[static_cast<size_t>(f) * NP];
        shared = matched_order(f, &out.perm[0], perm);
        for (int c = 0; c <= D && shared; ++c)
            for (int j = 0; j < NBF && shared; ++j)
                for (int q = 0; q < nq && shared; ++q) {
                    const double a = entry(0, c, out.perm[j], q);
                    shared = std::fabs(a - entry(f, c, perm[j], q)) <= 1e-10 * std::max(1.0, std::fabs(a));
                }
    }
    if (!shared)
        for (int f = 1; f < NF; ++f) own_order(f, &out.perm[static_cast<size_t>(f) * NP]);
    out.tables = shared ? 1 : NF;
    return out;
}

// Face function j (in the face's order) of `kind` at facet point q: zero beyond the basis, the points
// and, for the values and tangential derivatives, beyond the face functions.
double face_value(HostOperator const& h, FaceBasis const& fb, int f, int kind, int j, int q) {
    if (kind > h.D || j >= h.Nbf || q < 0 || q >= h.nq || (kind < h.D && j >= fb.FN)) return 0.0;
    const int NP = (h.Nbf + 7) / 8 * 8;
    return fb.tabs[f][(static_cast<size_t>(kind) * h.Nbf + fb.perm[static_cast<size_t>(f) * NP + j]) * h.nq + q];
}

}  // namespace

WarpFacetTables warp_facet_tables(HostOperator const& h) {
    const int D = h.D, NBF = h.Nbf, nq = h.nq;
    const int KS = (NBF + 3) / 4, NT = (NBF + 7) / 8;
    const FaceBasis fb = face_basis(h);
    const int KSS = (fb.FN + 3) / 4, NTS = (fb.FN + 7) / 8;
    const Blocks blk(nq);
    const int fwd = D * KSS + KS, fwd_half = KSS + KS, bwd = D * NTS + NT;
    const int frags = blk.full * fwd + blk.half * fwd_half + blk.steps() * bwd;
    WarpFacetTables out;
    out.perm = fb.perm;
    out.tables = fb.tables;
    out.frags.assign(static_cast<size_t>(out.tables) * frags * 32, 0.0);
    for (int f = 0; f < out.tables; ++f) {
        auto value = [&](int kind, int j, int q) { return face_value(h, fb, f, kind, j, q); };
        double* F = &out.frags[static_cast<size_t>(f) * frags * 32];
        int fr = 0;
        auto emit = [&](auto&& fn) {  // fn(t, n): B[k = t][n]
            for (int lane = 0; lane < 32; ++lane) F[static_cast<size_t>(fr) * 32 + lane] = fn(lane & 3, lane >> 2);
            ++fr;
        };
        for (int b = 0; b < blk.full; ++b)
            for (int c = 0; c <= D; ++c)
                for (int ks = 0; ks < (c < D ? KSS : KS); ++ks)
                    emit([&](int t, int m) { return value(c, 4 * ks + t, 8 * b + m); });
        if (blk.half)  // n tile p: column m = kind 2p + m % 2 of point m / 2
            for (int p = 0; p < 2; ++p)
                for (int ks = 0; ks < (p == 0 ? KSS : KS); ++ks)
                    emit([&](int t, int m) {
                        const int c = 2 * p + m % 2;
                        return c <= D ? value(c, 4 * ks + t, 8 * blk.full + m / 2) : 0.0;
                    });
        for (int s = 0; s < blk.steps(); ++s)
            for (int c = 0; c <= D; ++c)
                for (int nt = 0; nt < (c < D ? NTS : NT); ++nt)
                    emit([&](int t, int m) {
                        const int q = s < 2 * blk.full ? 8 * (s / 2) + 2 * t + s % 2 : 8 * blk.full + t;
                        // output column m = 2t' + h' holds permuted function 8 nt + 4 h' + t'
                        return value(c, nt * 8 + (m & 1) * 4 + (m >> 1), q);
                    });
        if (fr != frags) throw std::logic_error("warp tables: fragment count");
    }
    return out;
}

std::vector<double> warp_volume_frags(HostOperator const& h) {
    const int D = h.D, NBF = h.Nbf, Nq = h.Nq;
    const int KS = (NBF + 3) / 4, NT = (NBF + 7) / 8;
    const Blocks blk(Nq);
    std::vector<double> out;
    auto value = [&](int a, int k, int q) {
        return a < D && k < NBF && q < Nq ? h.Dxi_Q[(static_cast<size_t>(k) * D + a) * Nq + q] : 0.0;
    };
    auto emit = [&](auto&& fn) {  // fn(t, m): B[k = t][n = m]
        for (int lane = 0; lane < 32; ++lane) out.push_back(fn(lane & 3, lane >> 2));
    };
    for (int b = 0; b < blk.full; ++b)
        for (int a = 0; a < D; ++a)
            for (int ks = 0; ks < KS; ++ks) emit([&](int t, int m) { return value(a, 4 * ks + t, 8 * b + m); });
    if (blk.half)  // n tile p: column m = direction 2p + m % 2 at point m / 2
        for (int p = 0; p < (D + 1) / 2; ++p)
            for (int ks = 0; ks < KS; ++ks)
                emit([&](int t, int m) { return value(2 * p + m % 2, 4 * ks + t, 8 * blk.full + m / 2); });
    for (int s = 0; s < blk.steps(); ++s)
        for (int a = 0; a < D; ++a)
            for (int nt = 0; nt < NT; ++nt)
                emit([&](int t, int m) {
                    const int q = s < 2 * blk.full ? 8 * (s / 2) + 2 * t + s % 2 : 8 * blk.full + t;
                    return value(a, nt * 8 + (m & 1) * 4 + (m >> 1), q);
                });
    return out;
}

int64_t warp_volume_stride(HostOperator const& h) {
    const Blocks blk(h.Nq);
    return static_cast<int64_t>(volume_fields(h)) * (64 * blk.full + 32 * blk.half);
}

int64_t warp_facet_stride(HostOperator const& h) {
    const Blocks blk(h.nq);
    return static_cast<int64_t>(facet_fields(h)) * (64 * blk.full + 32 * blk.half);
}

namespace {

// The fields of facet f at point q: per side, then shared, then the other side -- elasticity lam, mu and
// J^-1 in the face-adapted directions (Ti) / w n and the last shared one; Poisson w n . (K G) (the flux
// and the lift both contract with it) / the last one: `scale` x w |n|.
template <class Put>
void facet_point_fields(HostOperator const& h, int64_t f, int q, double const* const (&Ti)[2], double scale, Put&& put) {
    const int D = h.D, DD = D * D, nq = h.nq;
    const double wq = h.w[q], last = scale * (wq * h.fNl[static_cast<size_t>(f) * nq + q]);
    double n[3];
    for (int i = 0; i < D; ++i) n[i] = wq * h.fN[(static_cast<size_t>(f) * D + i) * nq + q];
    if (h.kind == 0) {
        put(D, last);
        for (int s = 0; s < 2; ++s)
            for (int a = 0; a < D; ++a) {
                double m = 0.0;
                for (int r = 0; r < D; ++r) m += n[r] * h.fCoef[((static_cast<size_t>(f) * 2 + s) * DD + a * D + r) * nq + q];
                put(s * (D + 1) + a, m);
            }
        return;
    }
    for (int i = 0; i < D; ++i) put(2 + DD + i, n[i]);
    put(2 + DD + D, last);
    for (int s = 0; s < 2; ++s) {
        const int o = s * (2 + DD + D + 1);
        for (int c = 0; c < 2; ++c) put(o + c, h.fCoef[(static_cast<size_t>(f) * 4 + 2 * s + c) * nq + q]);
        std::vector<double> const& G = s == 0 ? h.fG0 : h.fG1;
        for (int b = 0; b < D; ++b)
            for (int i = 0; i < D; ++i) {
                double v = 0.0;
                for (int a = 0; a < D; ++a)
                    v += Ti[s][b * D + a] * G[(static_cast<size_t>(f) * DD + a * D + i) * nq + q];
                put(o + 2 + b * D + i, v);
            }
    }
}

// The volume fields of element e at point q.
template <class Put>
void volume_point_fields(HostOperator const& h, size_t e, int q, Put&& put) {
    const int D = h.D, DD = D * D, Nq = h.Nq;
    auto G = [&](int c) { return h.vG[(e * DD + c) * Nq + q]; };
    if (h.kind == 0) {
        const double c = h.vCoef[e * Nq + q];
        int f = 0;
        for (int a = 0; a < D; ++a)
            for (int b = a; b < D; ++b) {
                double m = 0.0;
                for (int i = 0; i < D; ++i) m += G(a * D + i) * G(b * D + i);
                put(f++, c * m);
            }
    } else {
        put(0, h.vCoef[(e * 2 + 0) * Nq + q]);
        put(1, h.vCoef[(e * 2 + 1) * Nq + q]);
        for (int c = 0; c < DD; ++c) put(2 + c, G(c));
    }
}

// Offset of field 0 and the field stride of point q of slot te (0..15) of an FP32 tile: lane
// (te % 8) * 4 + t, rows te and te + 8 side by side.
Slot slot32(Blocks const& b, int fields, int te, int q) {
    const int blk = q / 8, row = te / 8, g = te % 8;
    if (blk < b.full) {
        const int s = q % 8;
        return {static_cast<int64_t>(blk) * fields * 128 + (g * 4 + s / 2) * 4 + row * 2 + s % 2, 128};
    }
    return {static_cast<int64_t>(b.full) * fields * 128 + (g * 4 + q - 8 * b.full) * 2 + row, 64};
}

}  // namespace

FaceFrames::FaceFrames(HostOperator const& h) {
    double T[9];
    for (int f = 0; f < h.nfaces; ++f) face_directions(h.D, f, T, inv[f]);
}

void warp_facet_tile(HostOperator const& h, FaceFrames const& frames, int const* fids, int count, double* out) {
    std::fill_n(out, warp_facet_stride(h), 0.0);
    const int nf = facet_fields(h);
    const Blocks blk(h.nq);
    int32_t const* l = &h.loc[2 * static_cast<int64_t>(fids[0])];
    double const* const Ti[2] = {frames.inv[l[0]], frames.inv[l[1]]};
    for (int te = 0; te < count; ++te)
        for (int q = 0; q < h.nq; ++q) {
            const Slot sl = facet_slot(h, blk, nf, te, q);
            facet_point_fields(h, fids[te], q, Ti, h.penalty[fids[te]],
                               [&](int field, double v) { out[sl.base + field * sl.stride] = v; });
        }
}

void warp_volume_tile(HostOperator const& h, int64_t tile, double* out) {
    std::fill_n(out, warp_volume_stride(h), 0.0);
    const int nf = volume_fields(h);
    const Blocks blk(h.Nq);
    for (int te = 0; te < 8 && tile * 8 + te < h.E; ++te)
        for (int q = 0; q < h.Nq; ++q) {
            const Slot sl = point_slot(blk, nf, te, q);
            volume_point_fields(h, static_cast<size_t>(tile * 8 + te), q,
                                [&](int field, double v) { out[sl.base + field * sl.stride] = v; });
        }
}

// ---- FP32: tiles of 16, k steps of 8 ---------------------------------------------------------------------

WarpFacetTables32 warp_facet_tables32(HostOperator const& h) {
    const int D = h.D, NT = (h.Nbf + 7) / 8;
    const FaceBasis fb = face_basis(h);
    const int NTS = (fb.FN + 7) / 8;
    const Blocks blk(h.nq);
    WarpFacetTables32 out;
    out.perm = fb.perm;
    out.tables = fb.tables;
    for (int f = 0; f < out.tables; ++f) {
        auto emit = [&](auto&& fn) {  // fn(t, m): B[k = t][n = m], then k = t + 4
            for (int lane = 0; lane < 32; ++lane)
                for (int j = 0; j < 2; ++j) out.frags.push_back(static_cast<float>(fn((lane & 3) + 4 * j, lane >> 2)));
        };
        auto value = [&](int kind, int j, int q) { return face_value(h, fb, f, kind, j, q); };
        for (int b = 0; b < blk.full; ++b)
            for (int c = 0; c <= D; ++c)
                for (int ks = 0; ks < (c < D ? NTS : NT); ++ks)
                    emit([&](int t, int m) { return value(c, 8 * ks + t, 8 * b + m); });
        if (blk.half)
            for (int p = 0; p < 2; ++p)
                for (int ks = 0; ks < (p == 0 ? NTS : NT); ++ks)
                    emit([&](int t, int m) { return value(2 * p + m % 2, 8 * ks + t, 8 * blk.full + m / 2); });
        for (int b = 0; b < blk.full + blk.half; ++b)
            for (int c = 0; c <= D; ++c)
                for (int nt = 0; nt < (c < D ? NTS : NT); ++nt)
                    emit([&](int t, int m) {
                        // k = t is point 2t, k = t + 4 point 2t + 1; a half block has four points
                        if (b >= blk.full && t >= 4) return 0.0;
                        const int q = b < blk.full ? 8 * b + 2 * (t % 4) + t / 4 : 8 * blk.full + t;
                        return value(c, nt * 8 + (m & 1) * 4 + (m >> 1), q);
                    });
    }
    return out;
}

std::vector<float> warp_volume_frags32(HostOperator const& h) {
    const int D = h.D, NBF = h.Nbf, Nq = h.Nq, NT = (NBF + 7) / 8;
    const Blocks blk(Nq);
    std::vector<float> out;
    auto value = [&](int a, int k, int q) {
        return a < D && k < NBF && q < Nq ? h.Dxi_Q[(static_cast<size_t>(k) * D + a) * Nq + q] : 0.0;
    };
    auto emit = [&](auto&& fn) {
        for (int lane = 0; lane < 32; ++lane)
            for (int j = 0; j < 2; ++j) out.push_back(static_cast<float>(fn((lane & 3) + 4 * j, lane >> 2)));
    };
    for (int b = 0; b < blk.full; ++b)
        for (int a = 0; a < D; ++a)
            for (int ks = 0; ks < NT; ++ks) emit([&](int t, int m) { return value(a, 8 * ks + t, 8 * b + m); });
    if (blk.half)
        for (int p = 0; p < (D + 1) / 2; ++p)
            for (int ks = 0; ks < NT; ++ks)
                emit([&](int t, int m) { return value(2 * p + m % 2, 8 * ks + t, 8 * blk.full + m / 2); });
    for (int b = 0; b < blk.full + blk.half; ++b)
        for (int a = 0; a < D; ++a)
            for (int nt = 0; nt < NT; ++nt)
                emit([&](int t, int m) {
                    if (b >= blk.full && t >= 4) return 0.0;
                    const int q = b < blk.full ? 8 * b + 2 * (t % 4) + t / 4 : 8 * blk.full + t;
                    return value(a, nt * 8 + (m & 1) * 4 + (m >> 1), q);
                });
    return out;
}

int64_t warp_facet_stride32(HostOperator const& h) {
    const Blocks blk(h.nq);
    return static_cast<int64_t>(facet_fields(h)) * (128 * blk.full + 64 * blk.half);
}
int64_t warp_volume_stride32(HostOperator const& h) {
    const Blocks blk(h.Nq);
    return static_cast<int64_t>(volume_fields(h)) * (128 * blk.full + 64 * blk.half);
}

void warp_facet_tile32(HostOperator const& h, FaceFrames const& frames, int const* fids, int count, float* out) {
    std::fill_n(out, warp_facet_stride32(h), 0.0f);
    const int nf = facet_fields(h);
    const Blocks blk(h.nq);
    int32_t const* l = &h.loc[2 * static_cast<int64_t>(fids[0])];
    double const* const Ti[2] = {frames.inv[l[0]], frames.inv[l[1]]};
    for (int te = 0; te < count; ++te)
        for (int q = 0; q < h.nq; ++q) {
            const Slot sl = slot32(blk, nf, te, q);
            facet_point_fields(h, fids[te], q, Ti, 1.0,
                               [&](int field, double v) { out[sl.base + field * sl.stride] = static_cast<float>(v); });
        }
}

void warp_volume_tile32(HostOperator const& h, int64_t tile, float* out) {
    std::fill_n(out, warp_volume_stride32(h), 0.0f);
    const int nf = volume_fields(h);
    const Blocks blk(h.Nq);
    for (int te = 0; te < 16 && tile * 16 + te < h.E; ++te)
        for (int q = 0; q < h.Nq; ++q) {
            const Slot sl = slot32(blk, nf, te, q);
            volume_point_fields(h, static_cast<size_t>(tile * 16 + te), q,
                                [&](int field, double v) { out[sl.base + field * sl.stride] = static_cast<float>(v); });
        }
}

}  // namespace tdg
