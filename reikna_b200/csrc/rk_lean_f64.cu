// complex128 lean line passes
#include "rk_lean.cuh"

namespace rk {

#define RK_LN(LL, MODE, VAR, TW4) \
    if (L == LL && mode == MODE && var == VAR && tw4 == TW4) { *out = LeanLauncher<double, LL, MODE, VAR, TW4>::info(); return true; }
#define RK_LN_LANE(LL) RK_LN(LL, MODE_LANE, 0, false) RK_LN(LL, MODE_LANE, 0, true)
#define RK_LN_POS(LL) RK_LN(LL, MODE_POS, 0, false)
#define RK_LN_POST(LL) RK_LN(LL, MODE_POS, 2, false)

bool lean_info_f64(int L, int mode, int var, bool tw4, LeanInfo* out) {
    RK_LN_POS(16) RK_LN_POS(32) RK_LN_POS(64) RK_LN_POS(128) RK_LN_POS(256) RK_LN_POS(512)
    RK_LN_POS(1024) RK_LN_POS(2048) RK_LN_POS(4096) RK_LN_POS(8192)
    RK_LN_POST(16) RK_LN_POST(32) RK_LN_POST(64) RK_LN_POST(128) RK_LN_POST(256) RK_LN_POST(512)
    RK_LN(2, MODE_LANE, 0, false) RK_LN(4, MODE_LANE, 0, false) RK_LN(8, MODE_LANE, 0, false)
    RK_LN(16, MODE_LANE, 0, false)
    RK_LN_LANE(32) RK_LN_LANE(64) RK_LN_LANE(128) RK_LN_LANE(256) RK_LN_LANE(512)
    RK_LN(512, MODE_LANE, 8, true)
    return false;
}

}  // namespace rk
