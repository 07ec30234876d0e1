// FP32 resident kernels: 1 to 4 inner passes of 128 columns (grids up to 543
// columns), imaging and reference modes.
#include "fdtd_resident.cuh"

namespace tomo {
template <>
ResidentFn<float> resident_kernel_for<float>(int passes, int mode, ResidentShape shape) {
    const int key = mode * 10000 + passes * 1000 + shape.share * 100 + shape.warps;
    switch (key) {
#define TOMO_KERNEL(PASSES, MODE, R, W) \
    case MODE * 10000 + PASSES * 1000 + R * 100 + W: return &fdtd_resident_kernel<float, PASSES, MODE, R, W>;
        TOMO_KERNEL(1, kModeBreast, 2, 16)
        TOMO_KERNEL(1, kModeBreast, 4, 12)
        TOMO_KERNEL(2, kModeBreast, 2, 16)
        TOMO_KERNEL(3, kModeBreast, 2, 12)
        TOMO_KERNEL(3, kModeBreast, 2, 16)
        TOMO_KERNEL(4, kModeBreast, 4, 8)
        TOMO_KERNEL(3, kModeRef, 2, 12)
        TOMO_KERNEL(3, kModeRef, 2, 16)
#undef TOMO_KERNEL
    }
    return nullptr;
}
}  // namespace tomo
