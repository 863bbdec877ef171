// complex64 lean Bluestein passes with the real-spectrum step in them
#include "rk_lean_blue.cuh"

namespace rk {

#define RK_LB(LL, MODE, VAR) \
    if (L == LL && mode == MODE && var == VAR) { *out = LeanBlueLauncher<float, LL, MODE, VAR>::info(); return true; }

bool lean_blue_real_info_f32(int L, int mode, int var, LeanInfo* out) {
    RK_LB(16, MODE_POS, 6) RK_LB(32, MODE_POS, 6) RK_LB(64, MODE_POS, 6) RK_LB(128, MODE_POS, 6)
    RK_LB(256, MODE_POS, 6) RK_LB(512, MODE_POS, 6) RK_LB(1024, MODE_POS, 6) RK_LB(2048, MODE_POS, 6)
    RK_LB(4096, MODE_POS, 6) RK_LB(8192, MODE_POS, 6) RK_LB(16384, MODE_POS, 6)
    RK_LB(16, MODE_POS, 7) RK_LB(32, MODE_POS, 7) RK_LB(64, MODE_POS, 7) RK_LB(128, MODE_POS, 7)
    RK_LB(256, MODE_POS, 7) RK_LB(512, MODE_POS, 7) RK_LB(1024, MODE_POS, 7) RK_LB(2048, MODE_POS, 7)
    RK_LB(4096, MODE_POS, 7) RK_LB(8192, MODE_POS, 7) RK_LB(16384, MODE_POS, 7)
    return false;
}

}  // namespace rk
