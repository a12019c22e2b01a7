#include "gridkernels.cuh"

namespace pgmb200 {

template GridKernel gridKernel<float>(int, bool);

}  // namespace pgmb200
