// The stress kernels of the hooks without a return map, and the element update (snac_launch.cuh).
#include "snac_launch_elements.cuh"

namespace snac {
SNAC_STRESS_LAUNCHES(SNAC_RHEOLOGY_ELASTIC);
SNAC_STRESS_LAUNCHES(SNAC_RHEOLOGY_MAXWELL);
template void run_update_elements<SNAC_RHEOLOGY_ELASTIC>(ElemGrid, const Mesh&, const Fields&, const Config&, int);
template void run_update_elements<SNAC_RHEOLOGY_MAXWELL>(ElemGrid, const Mesh&, const Fields&, const Config&, int);
template void run_update_elements_slab<SNAC_RHEOLOGY_ELASTIC>(ElemGrid, const Mesh&, const Fields&, const Config&, int);
template void run_update_elements_slab<SNAC_RHEOLOGY_MAXWELL>(ElemGrid, const Mesh&, const Fields&, const Config&, int);
}  // namespace snac
