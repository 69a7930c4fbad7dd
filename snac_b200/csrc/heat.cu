// The heat-flux kernels (snac_launch.cuh).
#include "snac_launch.cuh"

namespace snac {

void run_heat_flux(ElemGrid g, bool one_phase, const Mesh& m, const Fields& F, const Config& c, int opens_step) {
    if (one_phase)
        k_heat_flux<true><<<g.blocks, ELEM_WARPS * 32, 0, g.stream>>>(m, F, c, opens_step);
    else
        k_heat_flux<false><<<g.blocks, ELEM_WARPS * 32, 0, g.stream>>>(m, F, c, opens_step);
}
void run_heat_flux_slab(ElemGrid g, bool one_phase, const Mesh& m, const Fields& F, const Config& c, int b0) {
    if (one_phase)
        k_heat_flux_slab<true><<<g.blocks, ELEM_WARPS * 32, 0, g.stream>>>(m, F, c, b0);
    else
        k_heat_flux_slab<false><<<g.blocks, ELEM_WARPS * 32, 0, g.stream>>>(m, F, c, b0);
}
void run_heat_flux_min_length_scale(ElemGrid g, bool one_phase, const Mesh& m, const Fields& F, const Config& c) {
    if (one_phase)
        k_heat_flux_min_length_scale<true><<<g.blocks, ELEM_WARPS * 32, 0, g.stream>>>(m, F, c);
    else
        k_heat_flux_min_length_scale<false><<<g.blocks, ELEM_WARPS * 32, 0, g.stream>>>(m, F, c);
}

}  // namespace snac
