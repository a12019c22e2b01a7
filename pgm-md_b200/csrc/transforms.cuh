// The cooperative kernels compiled in a translation unit of their own (transforms.cu).
#pragma once

#include "common.cuh"

namespace pgmb200 {

// The grid-transform kernel: compiled for one cubic grid size (32, 40, 48, 64), or for any grid (kc = 0); energy: the
// final pass's variant that also sums the reciprocal energy and strain.
typedef void (*GridKernel)(Dev, int);
template <typename R> GridKernel gridKernel(int kc, bool energy);

// The persistent CG kernel, compiled for the cubic grids of pcgSizes; any other grid (kc = 0) takes the general one.
typedef void (*PcgKernel)(Dev, int);
PcgKernel pcgKernel(int kc);

}  // namespace pgmb200
