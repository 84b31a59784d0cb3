// dem_steps_3.cu -- the step kernels of dem_steps.cuh for worlds whose scenes need bond model 3.
#include "dem_steps.cuh"

namespace demgb {
template StepsKernel steps_kernel<3>(int, bool, int);
}  // namespace demgb
