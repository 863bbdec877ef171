// lean passes of the real transforms, complex64 lines
#include "rk_lean_real.cuh"

namespace rk {

#define RK_LR(LL, VAR) \
    if (L == LL && var == VAR) { *out = LeanRealLauncher<float, LL, VAR>::info(); return true; }

bool lean_real_info_f32(int L, int var, LeanInfo* out) {
    RK_LR(16, 6) RK_LR(32, 6) RK_LR(64, 6) RK_LR(128, 6) RK_LR(256, 6) RK_LR(512, 6)
    RK_LR(1024, 6) RK_LR(2048, 6) RK_LR(4096, 6) RK_LR(8192, 6)
    RK_LR(16, 5) RK_LR(32, 5) RK_LR(64, 5) RK_LR(128, 5) RK_LR(256, 5) RK_LR(512, 5)
    RK_LR(1024, 5)
    RK_LR(16, 4) RK_LR(32, 4) RK_LR(64, 4) RK_LR(128, 4) RK_LR(256, 4) RK_LR(512, 4)
    RK_LR(1024, 4) RK_LR(2048, 4) RK_LR(4096, 4) RK_LR(8192, 4)
    return false;
}

}  // namespace rk
