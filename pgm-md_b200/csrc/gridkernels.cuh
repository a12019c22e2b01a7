// The grid-transform kernel's instances in precision R (compiled in a translation unit for each).
#pragma once

#include "transforms.cuh"

#include "gridfft.cuh"

namespace pgmb200 {

template <typename R, int K> GridKernel gridInstance(bool energy) {
    return energy ? k_fft_grid<R, K, true> : k_fft_grid<R, K, false>;
}

template <typename R> GridKernel gridKernel(int kc, bool energy) {
    switch (kc) {
    case 8: return gridInstance<R, 8>(energy);
    case 9: return gridInstance<R, 9>(energy);
    case 10: return gridInstance<R, 10>(energy);
    case 12: return gridInstance<R, 12>(energy);
    case 15: return gridInstance<R, 15>(energy);
    case 16: return gridInstance<R, 16>(energy);
    case 18: return gridInstance<R, 18>(energy);
    case 20: return gridInstance<R, 20>(energy);
    case 24: return gridInstance<R, 24>(energy);
    case 25: return gridInstance<R, 25>(energy);
    case 27: return gridInstance<R, 27>(energy);
    case 30: return gridInstance<R, 30>(energy);
    case 32: return gridInstance<R, 32>(energy);
    case 36: return gridInstance<R, 36>(energy);
    case 40: return gridInstance<R, 40>(energy);
    case 45: return gridInstance<R, 45>(energy);
    case 48: return gridInstance<R, 48>(energy);
    case 50: return gridInstance<R, 50>(energy);
    case 54: return gridInstance<R, 54>(energy);
    case 60: return gridInstance<R, 60>(energy);
    case 64: return gridInstance<R, 64>(energy);
    default: return gridInstance<R, 0>(energy);
    }
}

}  // namespace pgmb200
