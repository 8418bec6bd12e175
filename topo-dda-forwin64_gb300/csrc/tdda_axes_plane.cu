// tdda_axes_plane.cu -- the fused (y, z) plane kernels of the FP32 A-product for
// one y length, TDDA_PLANE_MY; build.py compiles this file once per length of
// TDDA_PLANE_Y (tdda_internal.cuh).
#include "tdda_axes.cuh"

namespace tdda {

#define TDDA_CAT2(a, b) a##b
#define TDDA_CAT(a, b) TDDA_CAT2(a, b)

// a == nullptr: raise the shared-memory limit of every kernel of this y length;
// Mz = 0 with a == nullptr likewise
cudaError_t TDDA_CAT(plane_, TDDA_PLANE_MY)(int Mz, const PassArgs<float>* a) {
    cudaError_t e = cudaErrorInvalidValue;
    if (!a) e = cudaSuccess;
#define TDDA_Z(MZ)                                                                             \
    if constexpr (dev::plane_fits<TDDA_PLANE_MY, MZ>()) {                                      \
        if (a && Mz == MZ) return dev::PlaneLaunch<TDDA_PLANE_MY, MZ>::run(*a);                \
        if (!a && e == cudaSuccess) e = dev::PlaneLaunch<TDDA_PLANE_MY, MZ>::configure();      \
    }
    TDDA_PLANE_Z(TDDA_Z)
#undef TDDA_Z
    return e;
}
bool TDDA_CAT(plane_has_, TDDA_PLANE_MY)(int Mz) {
#define TDDA_Z(MZ) \
    if (Mz == MZ) return dev::plane_fits<TDDA_PLANE_MY, MZ>();
    TDDA_PLANE_Z(TDDA_Z)
#undef TDDA_Z
    return false;
}

}  // namespace tdda
