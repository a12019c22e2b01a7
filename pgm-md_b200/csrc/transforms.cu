#include "transforms.cuh"

#include "gridfft.cuh"

namespace pgmb200 {

template <typename R> GridKernel gridKernel(int kc, bool energy) {
    switch (kc) {
    case 32: return energy ? k_fft_grid<R, 32, true> : k_fft_grid<R, 32, false>;
    case 40: return energy ? k_fft_grid<R, 40, true> : k_fft_grid<R, 40, false>;
    case 48: return energy ? k_fft_grid<R, 48, true> : k_fft_grid<R, 48, false>;
    case 64: return energy ? k_fft_grid<R, 64, true> : k_fft_grid<R, 64, false>;
    default: return energy ? k_fft_grid<R, 0, true> : k_fft_grid<R, 0, false>;
    }
}
template GridKernel gridKernel<float>(int, bool);
template GridKernel gridKernel<double>(int, bool);

}  // namespace pgmb200
