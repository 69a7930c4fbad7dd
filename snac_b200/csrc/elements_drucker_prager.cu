// The stress kernels of visco-plastic models with a Drucker-Prager phase (snac_launch.cuh).
#include "snac_launch_elements.cuh"

namespace snac {
SNAC_STRESS_LAUNCHES(SNAC_VP_DP);
}  // namespace snac
