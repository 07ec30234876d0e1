// Host stand-in for packed.cuh: pairs of values, each half rounded by itself.
#pragma once
#include <cuda_runtime.h>

namespace tomo {

template <typename Real>
struct alignas(2 * sizeof(Real)) Two {
    Real x, y;
};
template <typename Real>
Two<Real> add2(Two<Real> a, Two<Real> b) {
    return {a.x + b.x, a.y + b.y};
}
template <typename Real>
Two<Real> sub2(Two<Real> a, Two<Real> b) {
    return {a.x - b.x, a.y - b.y};
}
template <typename Real>
Two<Real> mul2(Two<Real> a, Two<Real> b) {
    return {a.x * b.x, a.y * b.y};
}
template <typename Real>
Two<Real> times2(Two<Real> a, Two<Real> b) {
    return {a.x * b.x, a.y * b.y};
}
template <typename Real>
Two<Real> fma2(Two<Real> a, Two<Real> b, Two<Real> c) {
    return {std::fma(a.x, b.x, c.x), std::fma(a.y, b.y, c.y)};
}
template <typename Real>
Two<Real> dup2(Real v) {
    return {v, v};
}

}  // namespace tomo
