// complex64 mixed-radix passes
#include "rk_lean_mix.cuh"

namespace rk {

void lean_mix_info_f32(int mode, int real, LeanInfo* out) {
    *out = LeanInfo{};
#define RK_LM(MODE, REAL) \
    if (mode == MODE && real == REAL) { \
        out->launch = &LeanMixLauncher<float, MODE, REAL>::launch; \
        out->prepare = &LeanMixLauncher<float, MODE, REAL>::prepare; \
    }
    RK_LM(MODE_POS, 0) RK_LM(MODE_LANE, 0) RK_LM(MODE_POS, 1) RK_LM(MODE_POS, 2)
#undef RK_LM
}

}  // namespace rk
