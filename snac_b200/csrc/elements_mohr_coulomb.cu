// The stress kernels of the hooks with a Mohr-Coulomb return map (snac_launch.cuh).
#include "snac_launch_elements.cuh"

namespace snac {
SNAC_STRESS_LAUNCHES(SNAC_RHEOLOGY_PLASTIC);
SNAC_STRESS_LAUNCHES(SNAC_RHEOLOGY_VISCOPLASTIC);
}  // namespace snac
