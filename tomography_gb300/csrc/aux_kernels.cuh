// Set-up and post-process kernels of the forward path: material rasterisation,
// FP64 coefficient precompute, descriptor progress, far-field transform and
// misfit reductions.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "packed.cuh"
#include "solve_desc.h"

namespace tomo {

constexpr double kPiD = 3.141592653589793238;
constexpr double kMu0D = kPiD * 4e-7;
constexpr double kEps0D = 8.85418e-12;

// ---------------------------------------------------------------------------
// Ellipse phantom raster (breast mode).  Per candidate: ell[k] = (cx, cy, a, b,
// cos, sin) in metres; material 0 background, 1 disc, 2+k ellipse k, later
// ellipses over earlier ones.  Explicit round-to-nearest intrinsics keep the
// arithmetic free of contraction so the map is bit-identical to a host
// evaluation of the same expression order.
static __global__ void raster_ellipse_kernel(uint8_t* __restrict__ mats, int mpitch, int nx, int ny, double dx,
                                      double disc_r, const double* __restrict__ ell, int nell, size_t mat_stride) {
    const int cand = blockIdx.z;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i > nx || j > ny) return;
    const double X = __dmul_rn(__dsub_rn((double)i, __dmul_rn(0.5, (double)nx)), dx);
    const double Y = __dmul_rn(__dsub_rn((double)j, __dmul_rn(0.5, (double)ny)), dx);
    uint8_t m = 0;
    if (disc_r > 0 && __dadd_rn(__dmul_rn(X, X), __dmul_rn(Y, Y)) <= __dmul_rn(disc_r, disc_r)) m = 1;
    const double* e = ell + (size_t)cand * nell * 6;
    for (int k = 0; k < nell; ++k, e += 6) {
        const double ex = __dsub_rn(X, e[0]), ey = __dsub_rn(Y, e[1]);
        const double u = __dadd_rn(__dmul_rn(ex, e[4]), __dmul_rn(ey, e[5]));
        const double v = __dsub_rn(__dmul_rn(ey, e[4]), __dmul_rn(ex, e[5]));
        const double q = __dadd_rn(__ddiv_rn(__dmul_rn(u, u), __dmul_rn(e[2], e[2])),
                                   __ddiv_rn(__dmul_rn(v, v), __dmul_rn(e[3], e[3])));
        if (q <= 1.0) m = (uint8_t)(2 + k);
    }
    mats[(size_t)cand * mat_stride + (size_t)j * mpitch + kMatPadLeft + i] = m;
}

// Receiver flags on the antenna cells of every candidate map.
static __global__ void mark_rx_kernel(uint8_t* mats, int mpitch, size_t mat_stride, const int* rx, int nrx, int ncand) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nrx * ncand) return;
    const int cand = t / nrx, r = t % nrx;
    mats[(size_t)cand * mat_stride + (size_t)rx[2 * r + 1] * mpitch + kMatPadLeft + rx[2 * r]] |= kMatRx;
}

// Per-material update coefficients in FP64 (FDTD_GPU.cu:739-741, 1118-1120;
// FDTD_CPU.cxx:979), rounded once to the field precision.  mp = [cand][32][3]
// (eps_inf, del_eps, sigma); tabs = [cand][32][kMatCoef].
template <typename Real>
__global__ void material_table_kernel(const double* __restrict__ mp, Real* __restrict__ tabs, int ncand, int nmat,
                                      double tau, double dt, double dx) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ncand * kMaxMat) return;
    const int m = t % kMaxMat;
    Real* out = tabs + (size_t)t * kMatCoef;
    for (int c = 0; c < kMatCoef; ++c) out[c] = Real(0);
    if (m >= nmat) return;
    const double einf = mp[3 * t], deps = mp[3 * t + 1], sig = mp[3 * t + 2];
    const double kp = (1 - dt / (2 * tau)) / (1 + dt / (2 * tau));
    const double beta = kEps0D * deps * dt / (tau * (1 + dt / (2 * tau)));
    const double den = 2 * einf * kEps0D + sig * dt + beta;
    out[kCa] = (Real)((2 * einf * kEps0D - sig * dt + beta) / den);
    out[kCb] = (Real)((2 * dt / dx) / den);
    out[kCj] = (Real)(((1 + kp) * dt) / den);
    out[kBp] = (Real)(beta / dt);
    out[kCi] = (Real)((-2 * kEps0D * einf + 2 * kEps0D - sig * dt - beta) / den);
    out[kCp] = (Real)((2 * kEps0D * einf - 2 * kEps0D - sig * dt + beta) / den);
    out[kCs] = (Real)((-2 * dt) / den);
}

// Progress the active solves of one kind (wavefront or resident) by T steps after an
// advance launch: `count` of them from `first` on, around the end.  counter may be null.
template <typename Real>
__global__ void bump_kernel(SolveDesc<Real>* descs, int nsolves, int T, int* counter, int resident, int first,
                            int count) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s == 0 && counter) *counter = 0;   // work counter of the next advance launch
    if (s >= nsolves || (s - first + nsolves) % nsolves >= count) return;
    SolveDesc<Real>& D = descs[s];
    if (D.active && D.resident == resident && D.step < D.steps_total) {
        D.step += T;
        if (!D.resident) D.parity ^= 1;   // the resident kernel keeps its state in one copy
    }
}

// ---------------------------------------------------------------------------
// Far field (N2FPostProcess, FDTD_GPU.cu:553-634).  Blocks per (solve, frequency)
// share the observation angles; a warp takes an angle, lanes loop over contour points.
// The positions come in FP64, whose conversions run at the FP64 rate (two lanes a
// clock and SM): a block converts a tile of them once for its warps' angles, and one
// thread does the frequency's FP64 set-up.  One solve of 200^2, 32 frequencies: 137 ->
// 25 us, 401^2 with four incident waves 200 -> 59 us; what is left is the FP32 sine and
// cosine of every angle and point.
// geom[c] = (X, Y, face) with X, Y the contour point relative to the
// transform origin [m]; ang[a] = (cos phi, sin phi).
template <typename Real>
__device__ __forceinline__ void dev_sincos(Real a, Real* s, Real* c);
template <>
__device__ __forceinline__ void dev_sincos<float>(float a, float* s, float* c) { sincosf(a, s, c); }
template <>
__device__ __forceinline__ void dev_sincos<double>(double a, double* s, double* c) { sincos(a, s, c); }

constexpr int kFarTile = 1024;   // contour points per tile
template <typename Real>
__global__ void __launch_bounds__(256) farfield_kernel(const Real* __restrict__ acc, size_t acc_stride, const Real* __restrict__ inc, int C,
                                int nfreq,
                                const double* __restrict__ freqs, const double* __restrict__ geom,
                                const double* __restrict__ ang, int nang, double dl, int norm, double tau,
                                double nbg, float* __restrict__ D, float* __restrict__ P) {
    // geom[c] = (X, Y, face) [m]; ang[a] = (cos phi, sin phi); sums in Real.
    // nbg: refractive index of the lossless background the contour lies in
    // (k = nbg k0, eta = eta0 / nbg); 1 for the reference's vacuum transform.
    // inc (total field, may be null): the incident grid's accumulators, added to
    // every solve's own (the legacy's single sum of both, by linearity).
    const int s = blockIdx.y, f = blockIdx.x;
    const Real* a = acc + (size_t)s * acc_stride + (size_t)f * C * 8;
    const Real* ia = inc ? inc + (size_t)f * C * 8 : nullptr;
    __shared__ double setup[3];   // eta, k, prad
    __shared__ Real xs[kFarTile], ys[kFarTile];
    __shared__ uint8_t faces[kFarTile];
    if (threadIdx.x == 0) {
        const double c0 = 1.0 / sqrt(kMu0D * kEps0D), eta0 = sqrt(kMu0D / kEps0D);
        const double fr = freqs[f];
        double prad = 1.0;
        if (norm == 1) {
            double g = tau * sqrt(kPiD) * exp(-tau * tau * 2 * kPiD * fr * 2 * kPiD * fr / 4);
            prad = (0.5 / eta0) * g * g * 33.329;
        }
        setup[0] = eta0 / nbg;
        setup[1] = 2 * kPiD * fr * nbg / c0;
        setup[2] = prad;
    }
    __syncthreads();
    const Real kr = (Real)setup[1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int a0 = nw * blockIdx.z; a0 < nang; a0 += nw * gridDim.z) {
        const int ai = a0 + warp;
        const bool mine = ai < nang;
        const Real cphi = mine ? (Real)ang[2 * ai] : Real(0), sphi = mine ? (Real)ang[2 * ai + 1] : Real(0);
        Real Nr = 0, Ni = 0, Lr = 0, Li = 0;
        for (int c = lane; c < (C + 31) / 32 * 32; c += 32) {
            const int at = c % kFarTile;
            if (at < 32) {   // the next tile, at the same point of every warp
                __syncthreads();
                for (int i = threadIdx.x; i < min(kFarTile, C - (c - lane)); i += blockDim.x) {
                    const double* g = geom + 3 * (size_t)(c - lane + i);
                    xs[i] = (Real)g[0];
                    ys[i] = (Real)g[1];
                    faces[i] = (uint8_t)g[2];
                }
                __syncthreads();
            }
            if (!mine || c >= C) continue;
            Real sp, cp;
            dev_sincos<Real>(kr * (xs[at] * cphi + ys[at] * sphi), &sp, &cp);
            const Real* e = a + (size_t)c * 8;
            Real jr = e[0] - e[2], ji = e[1] - e[3];
            Real mr = e[4] - e[6], mi = e[5] - e[7];
            if (ia) {
                const Real* q = ia + (size_t)c * 8;
                jr += q[0] - q[2]; ji += q[1] - q[3];
                mr += q[4] - q[6]; mi += q[5] - q[7];
            }
            const int face = faces[at];
            const Real wt = (face == 0 || face == 2) ? -sphi : cphi;
            Nr -= jr * cp - ji * sp;
            Ni -= jr * sp + ji * cp;
            Lr += wt * (mr * cp - mi * sp);
            Li += wt * (mr * sp + mi * cp);
        }
        for (int o = 16; o > 0; o >>= 1) {
            Nr += __shfl_xor_sync(0xffffffffu, Nr, o);
            Ni += __shfl_xor_sync(0xffffffffu, Ni, o);
            Lr += __shfl_xor_sync(0xffffffffu, Lr, o);
            Li += __shfl_xor_sync(0xffffffffu, Li, o);
        }
        if (lane == 0 && mine) {
            const double eta = setup[0], k = setup[1], prad = setup[2];
            const double Er = ((double)Lr + eta * (double)Nr) * dl, Ei = ((double)Li + eta * (double)Ni) * dl;
            const size_t o = ((size_t)s * nfreq + f) * nang + ai;
            D[o] = (float)(k * k * (Er * Er + Ei * Ei) / (8 * kPiD * eta * prad));
            P[o] = (float)atan2(Ei, Er);
        }
    }
}

// ---------------------------------------------------------------------------
// Trace misfit: num = sum (s - t)^2 per solve and den = sum t^2 per transmitter.
//
// The samples of a solve are cut into chunks of kMisfitChunk, summed one by one
// and added in order, whether one block takes all chunks of a solve or every
// chunk has a block of its own: the result does not depend on the batch.
//
// FP64 sums were bound by the FP64 units (two lanes a clock and SM, five
// operations a sample: 596 us for 49 M samples, 5% of HBM; now 97 us, bound by
// some 40 FP32 operations a sample).  FP32 traces are summed in FP32 without
// their rounding errors instead: the difference, its square and every addition
// are split into a value and its exact error (Knuth's two-sum, an fma for a
// product), the errors and their errors are added up beside the values, and a
// chunk's sums join in FP64.  Against exact sums of 1000 to 240000 samples the
// relative error is 0.8e-16 to 1.7e-16 rms, the FP64 sums' 1.1e-16 to 1.9e-16.
// (Without the errors' errors: 1.9e-16 to 2.5e-16, in 87 us.)  A chunk's sum that
// is outside [2^-70, 2^100] -- where products would lose bits to underflow or
// overflow -- or not finite is done in FP64, num and den each for itself: only the
// first candidate's solves take den, and num must not depend on it.
constexpr int kMisfitChunk = 8192;
inline int misfit_chunks(size_t n_per_solve) { return (int)((n_per_solve + kMisfitChunk - 1) / kMisfitChunk); }

// A sum, its error and that error's error, two columns of each.
struct SplitSum {
    Two<float> sum{0.0f, 0.0f}, err{0.0f, 0.0f}, rest{0.0f, 0.0f};
    // adds -m + e + low: m the negative of a rounded product, e its error, low what e lost
    __device__ __forceinline__ void take(Two<float> m, Two<float> e, Two<float> low) {
        const Two<float> x = sub2(sum, m), bv = sub2(sum, x), av = add2(x, bv);
        const Two<float> y = add2(sub2(sum, av), sub2(bv, m));
        sum = x;
        const Two<float> f = add2(y, e), ee = sub2(f, y), ye = sub2(f, ee);
        low = add2(low, add2(sub2(y, ye), sub2(e, ee)));
        const Two<float> z = add2(err, f), fv = sub2(z, err), ev = sub2(z, fv);
        rest = add2(rest, add2(low, add2(sub2(err, ev), sub2(f, fv))));
        err = z;
    }
    // adds (a - b)^2
    __device__ __forceinline__ void square_difference(Two<float> a, Two<float> b) {
        const Two<float> d = sub2(a, b), bv = sub2(a, d), av = add2(d, bv);
        const Two<float> lo = add2(sub2(a, av), sub2(bv, b));
        const Two<float> m{__fmul_rn(-d.x, d.x), __fmul_rn(-d.y, d.y)};
        // d^2 - m and 2 d lo with its error, their sum with its error, lo^2
        const Two<float> q = fma2(d, d, m), d2 = add2(d, d), g{__fmul_rn(d2.x, lo.x), __fmul_rn(d2.y, lo.y)};
        const Two<float> gl = fma2(d2, lo, Two<float>{-g.x, -g.y}), u = add2(q, g), gv = sub2(u, q), qv = sub2(u, gv);
        take(m, u, fma2(lo, lo, add2(gl, add2(sub2(q, qv), sub2(g, gv)))));
    }
    __device__ __forceinline__ void square(Two<float> a) {
        const Two<float> m{__fmul_rn(-a.x, a.x), __fmul_rn(-a.y, a.y)};
        take(m, fma2(a, a, m), Two<float>{0.0f, 0.0f});
    }
    // The block's sum in FP64 (thread 0): lanes, then the eight warps, in three parts.
    // (In two, the few last additions of the errors would round at 2^-49 of the sum.)
    __device__ __forceinline__ double block_total(float (*part)[3]) const {
        float s = sum.x, e = err.x, r = rest.x;
        auto two_sum = [](float& a, float b) {   // a += b; returns the rounding error
            const float x = __fadd_rn(a, b), bv = __fsub_rn(x, a), av = __fsub_rn(x, bv);
            const float y = __fadd_rn(__fsub_rn(a, av), __fsub_rn(b, bv));
            a = x;
            return y;
        };
        auto add = [&](float b, float f, float g) {
            const float y = two_sum(s, b);
            r = __fadd_rn(r, __fadd_rn(g, two_sum(e, f)));
            r = __fadd_rn(r, two_sum(e, y));
        };
        auto across = [&](int o) {
            const float b = __shfl_xor_sync(0xffffffffu, s, o), f = __shfl_xor_sync(0xffffffffu, e, o),
                        g = __shfl_xor_sync(0xffffffffu, r, o);
            add(b, f, g);
        };
        add(sum.y, err.y, rest.y);
        for (int o = 16; o > 0; o >>= 1) across(o);
        __syncthreads();
        if ((threadIdx.x & 31) == 0) {
            float* q = part[threadIdx.x >> 5];
            q[0] = s; q[1] = e; q[2] = r;
        }
        __syncthreads();
        if (threadIdx.x < 32) {
            const float* q = part[threadIdx.x & 7];
            s = q[0]; e = q[1]; r = q[2];
            for (int o = 4; o > 0; o >>= 1) across(o);
        }
        return (double)s + ((double)e + (double)r);
    }
};

// Sum over the block of one value per warp, in warp order (thread 0).
__device__ __forceinline__ double misfit_join(double v, double* part) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) part[w] = v;
    __syncthreads();
    double a = 0;
    if (threadIdx.x == 0)
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) a += part[i];
    return a;
}

// One chunk in FP64, the general form: num and den, either of which may be null.
template <typename Real>
__device__ inline void misfit_chunk_fp64(const Real* tr, const float* tg, int n, double* part, double* num, double* den,
                                         int* nonfinite) {
    double a = 0, b = 0;
    int bad = 0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const double tv = (double)tg[i];
        if (num) {
            const double sv = (double)tr[i];
            if (!isfinite(sv)) bad = 1;
            a += (sv - tv) * (sv - tv);
        }
        if (den) b += tv * tv;
    }
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    bad = __any_sync(0xffffffffu, bad);
    if (bad && (threadIdx.x & 31) == 0) atomicOr(nonfinite, 1);
    if (num) *num = misfit_join(a, part);
    if (den) *den = misfit_join(b, part);
}

// One chunk of FP32 traces with split sums; which of them ask for FP64.
struct MisfitRedo {
    bool num, den;   // the same in every thread
};
__device__ inline MisfitRedo misfit_chunk_split(const float* tr, const float* tg, int n, bool aligned, double* part,
                                                double* num, double* den) {
    SplitSum d, t;
    // the same samples to the same threads whatever the alignment
    auto four = [&](const float* p, int i) {
        return aligned ? __ldg(reinterpret_cast<const float4*>(p) + i)
                       : make_float4(__ldg(p + 4 * i), __ldg(p + 4 * i + 1), __ldg(p + 4 * i + 2), __ldg(p + 4 * i + 3));
    };
    const int quads = n / 4;
#pragma unroll 4
    for (int i = threadIdx.x; i < quads; i += blockDim.x) {
        const float4 a = four(tr, i), b = four(tg, i);
        d.square_difference({a.x, a.y}, {b.x, b.y});
        d.square_difference({a.z, a.w}, {b.z, b.w});
        if (den) {
            t.square({b.x, b.y});
            t.square({b.z, b.w});
        }
    }
    for (int i = 4 * quads + threadIdx.x; i < n; i += blockDim.x) {
        d.square_difference({tr[i], 0.0f}, {tg[i], 0.0f});
        if (den) t.square({tg[i], 0.0f});
    }
    float(*const parts)[3] = reinterpret_cast<float(*)[3]>(part);
    *num = d.block_total(parts);
    if (den) *den = t.block_total(parts);
    __shared__ MisfitRedo redo;
    auto outside = [](double v) { return !(v >= 0x1p-70 && v <= 0x1p100); };
    if (threadIdx.x == 0) redo = {outside(*num), den && outside(*den)};
    __syncthreads();
    return redo;
}

// num [nsolves][parts] and den [n_tx][parts]: gridDim.y = parts blocks per solve
// (parts = the solve's chunks), or one block that adds them all up (parts = 1).
// The target's own sum is taken once, by the first candidate's solves.
template <typename Real>
__global__ void __launch_bounds__(256)
    trace_partials_kernel(const Real* __restrict__ traces, size_t tr_stride, const float* __restrict__ target,
                          int n_per_solve, int n_tx, double* __restrict__ num, double* __restrict__ den,
                          int* __restrict__ nonfinite) {
    __shared__ double part[12];   // eight warps' FP64 sums, or three floats each
    const int s = blockIdx.x, tx = s % n_tx, parts = gridDim.y, chunks = (n_per_solve + kMisfitChunk - 1) / kMisfitChunk;
    const bool with_den = s < n_tx;
    double a = 0, b = 0;
    for (int c = blockIdx.y; c < chunks; c += parts) {
        const size_t at = (size_t)c * kMisfitChunk;
        const int n = min(kMisfitChunk, n_per_solve - (int)at);
        const Real* tr = traces + (size_t)s * tr_stride + at;
        const float* tg = target + (size_t)tx * n_per_solve + at;
        double cn = 0, cd = 0;
        MisfitRedo redo{true, with_den};
        if constexpr (sizeof(Real) == 4) {
            const bool aligned = (((size_t)tr | (size_t)tg) & 15) == 0;
            redo = misfit_chunk_split(tr, tg, n, aligned, part, &cn, with_den ? &cd : nullptr);
        }
        if (redo.num || redo.den)
            misfit_chunk_fp64<Real>(tr, tg, n, part, redo.num ? &cn : nullptr, redo.den ? &cd : nullptr, nonfinite);
        a += cn;
        b += cd;
    }
    if (threadIdx.x == 0) {
        num[(size_t)s * parts + blockIdx.y] = a;
        if (with_den) den[(size_t)tx * parts + blockIdx.y] = b;
    }
}

// fitness[c] = -sum_tx num / sum_tx den: a warp per candidate, a transmitter's
// chunks in order, then the lanes' transmitters.
static __global__ void trace_fitness_kernel(const double* __restrict__ num, const double* __restrict__ den, int parts,
                                            int n_tx, int ncand, double* fitness) {
    const int c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (c >= ncand) return;
    double a = 0, b = 0;
    for (int t = lane; t < n_tx; t += 32) {
        double p = 0, q = 0;
#pragma unroll 8
        for (int k = 0; k < parts; ++k) {
            p += num[(size_t)(c * n_tx + t) * parts + k];
            q += den[(size_t)t * parts + k];
        }
        a += p;
        b += q;
    }
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if (lane == 0) fitness[c] = b > 0 ? -a / b : -a;
}

// Far-field misfit (FDTD_GPU.cu:1004-1022 absolute; FDTD_CPU.cxx:841-845 relative).
// D is [cand][n_exc][nfreq][nang] which matches the reference's index
// Phi_index*A*F + freq_index*A + angle.
static __global__ void ff_fitness_kernel(const float* __restrict__ D, const float* __restrict__ meas, int n_per_cand,
                                  double norm, int relative, double* fitness, int* nonfinite) {
    const int c = blockIdx.x;
    const float* d = D + (size_t)c * n_per_cand;
    double acc = 0;
    int bad = 0;
    for (int i = threadIdx.x; i < n_per_cand; i += blockDim.x) {
        const double diff = (double)d[i] - (double)meas[i];
        if (!isfinite((double)d[i])) bad = 1;
        double term = diff * diff / norm;
        if (relative) term /= (double)meas[i] * (double)meas[i];
        acc += term;
    }
    __shared__ double sa[32];
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    bad = __any_sync(0xffffffffu, bad);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) sa[w] = acc;
    if (bad && lane == 0) atomicOr(nonfinite, 1);
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0;
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) a += sa[i];
        fitness[c] = -a;
    }
}

// Traces of all solves to a packed host-layout buffer [solve][nrx][steps].
template <typename Real, typename Out>
__global__ void traces_pack_kernel(const Real* __restrict__ traces, size_t tr_stride, int n_per_solve, int nsolves,
                                   Out* __restrict__ out) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)n_per_solve * nsolves) return;
    const size_t s = i / n_per_solve, r = i % n_per_solve;
    out[i] = (Out)traces[s * tr_stride + r];
}

}  // namespace tomo
