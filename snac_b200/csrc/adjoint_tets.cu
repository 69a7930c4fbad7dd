// The reverse of a tet's step (snac_launch.cuh).
#include "snac_launch.cuh"

namespace snac {

template <int P>
cudaError_t run_adj_tet(int device, ElemGrid g, const Mesh& m, const Fields& F, const Config& c, const AdjState& S,
                        const AdjBufs& B, int rotate, int first_rev, double dt) {
    const cudaError_t e = allow_smem<k_adj_tet<P>>(device, sizeof(AdjSmem));
    if (e != cudaSuccess) return e;
    k_adj_tet<P><<<g.blocks, ELEM_WARPS * 32, sizeof(AdjSmem), g.stream>>>(m, F, c, S, B, rotate, first_rev, dt);
    return cudaSuccess;
}
#define SNAC_ADJ_TET(P)                                                                                          \
    template cudaError_t run_adj_tet<P>(int, ElemGrid, const Mesh&, const Fields&, const Config&, const AdjState&, \
                                        const AdjBufs&, int, int, double)
SNAC_ADJ_TET(SNAC_RHEOLOGY_ELASTIC);
SNAC_ADJ_TET(SNAC_RHEOLOGY_PLASTIC);
SNAC_ADJ_TET(SNAC_RHEOLOGY_VISCOPLASTIC);
SNAC_ADJ_TET(SNAC_RHEOLOGY_MAXWELL);

}  // namespace snac
