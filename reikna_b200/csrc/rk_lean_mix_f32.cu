// complex64 mixed-radix passes
#include "rk_lean_mix.cuh"

namespace rk {

void lean_mix_info_f32(int mode, LeanInfo* out) {
    *out = LeanInfo{};
    out->launch = mode == MODE_POS ? &LeanMixLauncher<float, MODE_POS>::launch : &LeanMixLauncher<float, MODE_LANE>::launch;
    out->prepare = mode == MODE_POS ? &LeanMixLauncher<float, MODE_POS>::prepare : &LeanMixLauncher<float, MODE_LANE>::prepare;
}

}  // namespace rk
