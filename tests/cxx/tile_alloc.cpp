// Counts heap allocations while the apply's geometry tiles are filled: that happens in an OpenMP parallel
// region, where a failing allocation would end the process instead of returning TDG_E_NOMEM.
#include "host/setup.hpp"
#include "host/warp_tables.hpp"

#include <cstdio>
#include <cstdlib>
#include <new>

static long g_allocations = 0;

void* operator new(std::size_t n) {
    ++g_allocations;
    if (void* p = std::malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }

int main() {
    using namespace tdg;
    long total = 0;
    for (int D = 2; D <= 3; ++D)
        for (int N = 1; N <= 4; N += 3)
            for (int kind = 0; kind < 2; ++kind) {
                // the unit simplex alone, its faces on the boundary
                auto const nodes = warp_blend_nodes(D, 1);
                const SimplexRule vol = conical_product_rule(D, 2 * N + 1), fct = conical_product_rule(D - 1, 2 * N + 1);
                std::vector<int64_t> up(2 * (D + 1), 0);
                std::vector<int32_t> loc, bc(D + 1, 3);
                for (int f = 0; f <= D; ++f) loc.insert(loc.end(), {f, f});
                HostOperator h;
                h.build(D, N, 1, kind, 1, D + 1, nodes.data(), up.data(), loc.data(), bc.data(), vol.size(), vol.x.data(),
                        vol.w.data(), fct.size(), fct.x.data(), fct.w.data());
                std::vector<double> c(static_cast<size_t>(h.Nq), 1.0);
                h.set_material(c.data(), kind ? c.data() : nullptr);
                const FaceFrames frames(h);
                std::vector<double> f64(static_cast<size_t>(warp_facet_stride(h))), v64(static_cast<size_t>(warp_volume_stride(h)));
                std::vector<float> f32(static_cast<size_t>(warp_facet_stride32(h))), v32(static_cast<size_t>(warp_volume_stride32(h)));
                const long before = g_allocations;
                for (int f = 0; f <= D; ++f) {
                    warp_facet_tile(h, frames, &f, 1, f64.data());
                    warp_facet_tile32(h, frames, &f, 1, f32.data());
                }
                warp_volume_tile(h, 0, v64.data());
                warp_volume_tile32(h, 0, v32.data());
                total += g_allocations - before;
            }
    std::printf("%ld\n", total);
    return 0;
}
