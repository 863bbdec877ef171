// complex128 lean Bluestein passes
#include "rk_lean_blue.cuh"

namespace rk {

#define RK_LB(LL, MODE, VAR) \
    if (L == LL && mode == MODE && var == VAR) { *out = LeanBlueLauncher<double, LL, MODE, VAR>::info(); return true; }

bool lean_blue_real_info_f64(int L, int mode, int var, LeanInfo* out);

bool lean_blue_info_f64(int L, int mode, int var, LeanInfo* out) {
    RK_LB(16, MODE_POS, 1) RK_LB(32, MODE_POS, 1) RK_LB(64, MODE_POS, 1) RK_LB(128, MODE_POS, 1)
    RK_LB(256, MODE_POS, 1) RK_LB(512, MODE_POS, 1) RK_LB(1024, MODE_POS, 1) RK_LB(2048, MODE_POS, 1)
    RK_LB(4096, MODE_POS, 1) RK_LB(8192, MODE_POS, 1)
    RK_LB(16, MODE_LANE, 1) RK_LB(32, MODE_LANE, 1) RK_LB(64, MODE_LANE, 1) RK_LB(128, MODE_LANE, 1)
    RK_LB(256, MODE_LANE, 1) RK_LB(512, MODE_LANE, 1) RK_LB(1024, MODE_LANE, 1)
    RK_LB(64, MODE_POS, 3) RK_LB(128, MODE_POS, 3) RK_LB(256, MODE_POS, 3) RK_LB(512, MODE_POS, 3)
    RK_LB(1024, MODE_POS, 3)
    RK_LB(32, MODE_LANE, 3) RK_LB(64, MODE_LANE, 3) RK_LB(128, MODE_LANE, 3) RK_LB(256, MODE_LANE, 3)
    RK_LB(512, MODE_LANE, 3)
    RK_LB(32, MODE_LANE, 4) RK_LB(64, MODE_LANE, 4) RK_LB(128, MODE_LANE, 4) RK_LB(256, MODE_LANE, 4)
    RK_LB(512, MODE_LANE, 4)
    RK_LB(32, MODE_LANE, 5) RK_LB(64, MODE_LANE, 5) RK_LB(128, MODE_LANE, 5) RK_LB(256, MODE_LANE, 5)
    RK_LB(512, MODE_LANE, 5)
    return var >= 6 && lean_blue_real_info_f64(L, mode, var, out);
}

}  // namespace rk
