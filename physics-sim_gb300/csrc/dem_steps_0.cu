// dem_steps_0.cu -- the step kernels of dem_steps.cuh for worlds whose scenes need bond model 0.
#include "dem_steps.cuh"

namespace demgb {
template StepsKernel steps_kernel<0>(int, bool, int);
}  // namespace demgb
