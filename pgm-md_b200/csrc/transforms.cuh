// The cooperative kernels compiled in translation units of their own.
#pragma once

#include "common.cuh"

namespace pgmb200 {

// The grid-transform kernel, compiled for every cubic 2-3-5 grid of 8 to 64 points (the general kernel's run-time radices and
// index divisions cost it 6 us at 30^3), any other grid by the general one (kc = 0); energy: the final pass's variant that
// also sums the reciprocal energy and strain.
constexpr int FFTG_MIN_K = 8;
typedef void (*GridKernel)(Dev, int);
template <typename R> GridKernel gridKernel(int kc, bool energy);

// The persistent CG kernel, compiled for the same cubic grids; any other grid (kc = 0) takes the general one, and so does an
// engine of more atoms than the blocks' shared memory holds the state of (shared false: the state in global memory).
typedef void (*PcgKernel)(Dev, int, int);
PcgKernel pcgKernel(int kc, bool shared);

}  // namespace pgmb200
