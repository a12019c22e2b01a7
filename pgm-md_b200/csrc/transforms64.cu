#include "gridkernels.cuh"

namespace pgmb200 {

template GridKernel gridKernel<double>(int, bool);

}  // namespace pgmb200
