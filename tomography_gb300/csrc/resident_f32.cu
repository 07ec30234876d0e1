// FP32 resident kernels: 1 to 4 inner passes of 128 columns (grids up to 543
// columns), imaging and reference modes.
#include "fdtd_resident.cuh"

namespace tomo {
template <>
ResidentFn<float> resident_kernel_for<float>(int passes, int mode) {
    if (mode == kModeBreast) {
        if (passes == 1) return &fdtd_resident_kernel<float, 1, kModeBreast>;
        if (passes == 2) return &fdtd_resident_kernel<float, 2, kModeBreast>;
        if (passes == 3) return &fdtd_resident_kernel<float, 3, kModeBreast>;
        if (passes == 4) return &fdtd_resident_kernel<float, 4, kModeBreast>;
    } else if (passes == 3) {
        return &fdtd_resident_kernel<float, 3, kModeRef>;
    }
    return nullptr;
}
}  // namespace tomo
