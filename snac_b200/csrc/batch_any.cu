// Element tiles with the run-time switch over the hooks (snac_launch.cuh).
#include "snac_launch.cuh"

namespace snac {

template <int OP>
void run_tiles(ElemGrid g, const ModelDesc* D, const int2* tiles, int n) {
    kb_elements<OP><<<g.blocks, ELEM_WARPS * 32, 0, g.stream>>>(D, tiles, n);
}
template void run_tiles<BOP_FUSED>(ElemGrid, const ModelDesc*, const int2*, int);
template void run_tiles<BOP_HEAT_FLUX>(ElemGrid, const ModelDesc*, const int2*, int);
template void run_tiles<BOP_STRESS>(ElemGrid, const ModelDesc*, const int2*, int);
template void run_tiles<BOP_FUSED_STRESS>(ElemGrid, const ModelDesc*, const int2*, int);

}  // namespace snac
