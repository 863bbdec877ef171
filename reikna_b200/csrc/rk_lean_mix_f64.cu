// complex128 mixed-radix passes
#include "rk_lean_mix.cuh"

namespace rk {

void lean_mix_info_f64(int mode, int real, LeanInfo* out) {
    *out = LeanInfo{};
#define RK_LM(MODE, REAL) \
    if (mode == MODE && real == REAL) { \
        out->launch = &LeanMixLauncher<double, MODE, REAL>::launch; \
        out->prepare = &LeanMixLauncher<double, MODE, REAL>::prepare; \
    }
    RK_LM(MODE_POS, 0) RK_LM(MODE_LANE, 0) RK_LM(MODE_POS, 1) RK_LM(MODE_POS, 2)
#undef RK_LM
}

}  // namespace rk
