#include "transforms.cuh"

#include "persistent.cuh"

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

template <int GS, int KC> static PcgKernel pcgPass(int pass) {
    return pass == 0 ? k_cg_persistent<6, GS, KC, 0> : pass == 1 ? k_cg_persistent<6, GS, KC, 1> : k_cg_persistent<6, GS, KC, 2>;
}

PcgKernel pcgKernel(int lanes, int kc, int pass) {
    if (lanes >= 32)
        return kc == 48 ? pcgPass<32, 48>(pass) : pcgPass<32, 0>(pass);
    if (lanes >= 16)
        return kc == 48 ? pcgPass<16, 48>(pass) : pcgPass<16, 0>(pass);
    return kc == 48 ? pcgPass<8, 48>(pass) : pcgPass<8, 0>(pass);
}

}  // namespace pgmb200
