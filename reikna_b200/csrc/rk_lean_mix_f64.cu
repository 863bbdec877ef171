// complex128 mixed-radix passes
#include "rk_lean_mix.cuh"

namespace rk {

void lean_mix_info_f64(int mode, LeanInfo* out) {
    *out = LeanInfo{};
    out->launch = mode == MODE_POS ? &LeanMixLauncher<double, MODE_POS>::launch : &LeanMixLauncher<double, MODE_LANE>::launch;
    out->prepare = mode == MODE_POS ? &LeanMixLauncher<double, MODE_POS>::prepare : &LeanMixLauncher<double, MODE_LANE>::prepare;
}

}  // namespace rk
