// The cooperative kernels compiled in a translation unit of their own (transforms.cu).
#pragma once

#include "common.cuh"

namespace pgmb200 {

// The grid-transform kernel: compiled for one cubic grid size (32, 40, 48, 64), or for any grid (kc = 0); energy: the
// final pass's variant that also sums the reciprocal energy and strain.
typedef void (*GridKernel)(Dev, int);
template <typename R> GridKernel gridKernel(int kc, bool energy);

// The persistent CG kernel for the pair lanes (8, 16 or 32; 4 runs as 8) and the grid's compile-time size (48, or 0:
// any).  pass 0: the CG loop; 1 / 2: one field pass of dipoles (and charges).
typedef void (*PcgKernel)(Dev, int, const double*);
PcgKernel pcgKernel(int lanes, int kc, int pass);

}  // namespace pgmb200
