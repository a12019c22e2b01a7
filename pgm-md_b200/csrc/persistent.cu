// The persistent CG kernel's instances: every cubic 2-3-5 grid from 8 to 64 points, whose line transforms and index maps
// are then compile-time (at 40^3 the general kernel's run-time radices cost 180 us of an 800 us evaluation).
#include "transforms.cuh"

#include "persistent.cuh"

namespace pgmb200 {

PcgKernel pcgKernel(int kc, bool shared) {
    if (!shared)
        return k_cg_persistent<6, 0, false>;
    switch (kc) {
    case 8: return k_cg_persistent<6, 8>;
    case 9: return k_cg_persistent<6, 9>;
    case 10: return k_cg_persistent<6, 10>;
    case 12: return k_cg_persistent<6, 12>;
    case 15: return k_cg_persistent<6, 15>;
    case 16: return k_cg_persistent<6, 16>;
    case 18: return k_cg_persistent<6, 18>;
    case 20: return k_cg_persistent<6, 20>;
    case 24: return k_cg_persistent<6, 24>;
    case 25: return k_cg_persistent<6, 25>;
    case 27: return k_cg_persistent<6, 27>;
    case 30: return k_cg_persistent<6, 30>;
    case 32: return k_cg_persistent<6, 32>;
    case 36: return k_cg_persistent<6, 36>;
    case 40: return k_cg_persistent<6, 40>;
    case 45: return k_cg_persistent<6, 45>;
    case 48: return k_cg_persistent<6, 48>;
    case 50: return k_cg_persistent<6, 50>;
    case 54: return k_cg_persistent<6, 54>;
    case 60: return k_cg_persistent<6, 60>;
    case 64: return k_cg_persistent<6, 64>;
    default: return k_cg_persistent<6, 0>;
    }
}

}  // namespace pgmb200
