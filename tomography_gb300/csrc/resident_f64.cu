// FP64 resident kernels: 1 to 3 inner passes of 64 columns (grids up to 223
// columns) in the imaging mode.
#include "fdtd_resident.cuh"

namespace tomo {
template <>
ResidentFn<double> resident_kernel_for<double>(int passes, int mode) {
    if (mode != kModeBreast) return nullptr;
    if (passes == 1) return &fdtd_resident_kernel<double, 1, kModeBreast>;
    if (passes == 2) return &fdtd_resident_kernel<double, 2, kModeBreast>;
    if (passes == 3) return &fdtd_resident_kernel<double, 3, kModeBreast>;
    return nullptr;
}
}  // namespace tomo
