// dem_steps_any.cu -- the step kernels of dem_steps.cuh for worlds of any scenes.
#include "dem_steps.cuh"

namespace demgb {
template StepsKernel steps_kernel<-1>(int, bool, int);
}  // namespace demgb
