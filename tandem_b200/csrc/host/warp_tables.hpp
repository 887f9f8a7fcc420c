// Host-side data of the warp-tile FP64 apply (kernels/apply_warp.cuh): B fragments of the basis
// tables in mma order and per-point geometry in lane order.
#pragma once

#include "setup.hpp"

#include <cstdint>
#include <vector>

namespace tdg {

struct WarpFacetTables {
    std::vector<double> frags;  // [table][fragment][lane]
    int tables = 0;             // 1: all faces share one table (nodal bases); else one per face
    std::vector<int> perm;      // [face][8 NT]
};
// Facet fragments per local face and the order of the basis functions on it (face functions first).
WarpFacetTables warp_facet_tables(HostOperator const& h);

// Volume fragments.
std::vector<double> warp_volume_frags(HostOperator const& h);
// Volume geometry of the tile of elements [8 tile, 8 tile + 8): warp_volume_stride(h) doubles (zero
// where there is no element or point).
int64_t warp_volume_stride(HostOperator const& h);
void warp_volume_tile(HostOperator const& h, int64_t tile, double* out);

// Inverses of the faces' adapted reference directions, formed once: the tiles are filled in parallel and
// allocate nothing there (an exception cannot leave a parallel region).
struct FaceFrames {
    double inv[4][9];
    explicit FaceFrames(HostOperator const& h);
};
// Facet geometry of one tile of up to 8 facets of one (l0, l1): `count` facet ids at `fids`; out
// holds warp_facet_stride(h) doubles.
int64_t warp_facet_stride(HostOperator const& h);
void warp_facet_tile(HostOperator const& h, FaceFrames const& frames, int const* fids, int count, double* out);

// The same for the FP32 kernels (kernels/apply_warp32.cuh): tiles of 16, fragments [table][fragment]
// [lane][2]; the facet geometry's last shared field lacks the penalty.
struct WarpFacetTables32 {
    std::vector<float> frags;
    int tables = 0;
    std::vector<int> perm;
};
WarpFacetTables32 warp_facet_tables32(HostOperator const& h);
std::vector<float> warp_volume_frags32(HostOperator const& h);
int64_t warp_facet_stride32(HostOperator const& h);
int64_t warp_volume_stride32(HostOperator const& h);
void warp_facet_tile32(HostOperator const& h, FaceFrames const& frames, int const* fids, int count, float* out);
void warp_volume_tile32(HostOperator const& h, int64_t tile, float* out);

}  // namespace tdg
