// FP64 resident kernels: 1 to 3 inner passes of 64 columns (grids up to 223
// columns), imaging mode.
#include "fdtd_resident.cuh"

namespace tomo {
template <>
ResidentFn<double> resident_kernel_for<double>(int passes, int mode, ResidentShape shape) {
    if (mode != kModeBreast || shape.share != 2 || shape.warps != 12) return nullptr;
    if (passes == 1) return &fdtd_resident_kernel<double, 1, kModeBreast, 2, 12>;
    if (passes == 2) return &fdtd_resident_kernel<double, 2, kModeBreast, 2, 12>;
    if (passes == 3) return &fdtd_resident_kernel<double, 3, kModeBreast, 2, 12>;
    return nullptr;
}
}  // namespace tomo
