// Programmatic dependent launch of the persistent plane and line passes.
#pragma once
#include <cuda_runtime.h>

namespace rk {

// Dependent launch of the persistent kernels: their CTAs may be placed as the CTAs of the
// kernel before them leave (which triggers nothing itself), set up, and wait here for its
// completion before they touch an array (256^3 with shift and scale 145.8 -> 141.1 us a call).
__device__ __forceinline__ void dependent_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
inline cudaLaunchAttribute dependent_launch() {
    cudaLaunchAttribute a;
    a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a.val.programmaticStreamSerializationAllowed = 1;
    return a;
}

}  // namespace rk
