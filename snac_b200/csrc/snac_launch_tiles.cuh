// snac_launch_tiles.cuh — the launches of the batch's class tiles
// (snac_launch.cuh), for the files that instantiate them.
#pragma once

#include "snac_launch.cuh"

namespace snac {

template <int OP, int P, int TEMP>
void run_class_tiles(ElemGrid g, const ModelDesc* D, const int2* tiles, int n) {
    kb_elements_c<OP, P, TEMP><<<g.blocks, ELEM_WARPS * 32, 0, g.stream>>>(D, tiles, n);
}

#define SNAC_CLASS_TILES(OP, P, TEMP) \
    template void run_class_tiles<OP, P, TEMP>(ElemGrid, const ModelDesc*, const int2*, int)

}  // namespace snac
