// snac_launch_elements.cuh — the launches of the stress kernels and of the
// element update (snac_launch.cuh), for the files that instantiate them.
#pragma once

#include "snac_launch.cuh"

namespace snac {

template <int P>
void run_calc_stresses(ElemGrid g, bool one_phase, const Mesh& m, const Fields& F, const Config& c) {
    if (one_phase)
        k_calc_stresses<P, true><<<g.blocks, ELEM_WARPS * 32, 0, g.stream>>>(m, F, c);
    else
        k_calc_stresses<P, false><<<g.blocks, ELEM_WARPS * 32, 0, g.stream>>>(m, F, c);
}
template <int P>
void run_calc_stresses_slab(ElemGrid g, bool one_phase, const Mesh& m, const Fields& F, const Config& c, int b0) {
    if (one_phase)
        k_calc_stresses_slab<P, true><<<g.blocks, ELEM_WARPS * 32, 0, g.stream>>>(m, F, c, b0);
    else
        k_calc_stresses_slab<P, false><<<g.blocks, ELEM_WARPS * 32, 0, g.stream>>>(m, F, c, b0);
}
template <int P>
void run_fused_step(ElemGrid g, bool one_phase, const Mesh& m, const Fields& F, const Config& c) {
    if (one_phase)
        k_fused_step<P, true><<<g.blocks, ELEM_WARPS * 32, 0, g.stream>>>(m, F, c);
    else
        k_fused_step<P, false><<<g.blocks, ELEM_WARPS * 32, 0, g.stream>>>(m, F, c);
}
template <int P>
void run_fused_stress(ElemGrid g, bool one_phase, const Mesh& m, const Fields& F, const Config& c) {
    if (one_phase)
        k_fused_stress<P, true><<<g.blocks, ELEM_WARPS * 32, 0, g.stream>>>(m, F, c);
    else
        k_fused_stress<P, false><<<g.blocks, ELEM_WARPS * 32, 0, g.stream>>>(m, F, c);
}
template <int P>
void run_update_elements(ElemGrid g, const Mesh& m, const Fields& F, const Config& c, int pending) {
    k_update_elements<P><<<g.blocks, ELEM_WARPS * 32, 0, g.stream>>>(m, F, c, pending);
}
template <int P>
void run_update_elements_slab(ElemGrid g, const Mesh& m, const Fields& F, const Config& c, int b0) {
    k_update_elements_slab<P><<<g.blocks, ELEM_WARPS * 32, 0, g.stream>>>(m, F, c, b0);
}

#define SNAC_STRESS_LAUNCHES(P)                                                                              \
    template void run_calc_stresses<P>(ElemGrid, bool, const Mesh&, const Fields&, const Config&);           \
    template void run_calc_stresses_slab<P>(ElemGrid, bool, const Mesh&, const Fields&, const Config&, int); \
    template void run_fused_step<P>(ElemGrid, bool, const Mesh&, const Fields&, const Config&);              \
    template void run_fused_stress<P>(ElemGrid, bool, const Mesh&, const Fields&, const Config&)

}  // namespace snac
