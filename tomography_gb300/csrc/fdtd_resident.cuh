// On-chip resident FDTD kernel: one solve per thread-block cluster.
//
// The wavefront kernel (fdtd_advance.cuh) streams every field through HBM once
// per T steps and spends most of its issue slots on moving rows between time
// levels.  A solve of up to about 500^2 cells fits the shared memory and
// registers of one cluster, so here a cluster loads a solve once, advances it
// by many time steps without touching HBM, and writes it back.
//
// Layout.  The rows 1 .. ny-1 of the Ez grid are cut into one slab per block
// (SolveDesc::ys), a slab into groups of two (four) rows, one group per warp:
//  * Ez of a slab lives in shared memory, two copies (time n and n+1), with one
//    halo row below and above that the neighbouring blocks write through
//    distributed shared memory;
//  * Hx and Hy live in the registers of the warp that owns the rows.  The warp
//    also keeps Hx of the row below its own and advances it redundantly from
//    Ez, so that a time step needs one exchange instead of two;
//  * the Debye current of the material box, the material bytes and the CPML
//    psi of the rows that have them live in shared memory.
// A warp covers its whole rows: the 16 outermost columns of either side (PEC
// boundary, x-CPML) in one pass with one column per lane, the columns between
// in passes of 32 x 16 bytes.  Only the passes that meet a material, a y-CPML
// row or the source run the longer code.  Pairs of FP32 columns (rows, in the
// edge pass) use the packed f32x2 instructions: both halves round as the scalar
// ones, so every cell gets the bits of the other paths.
//
// A step ends with one block barrier; blocks wait for each other's halo rows
// only.  Then the threads of a block sample the step, the warps with the fewest
// rows first: the receivers to the traces and the NTFF contour to the staging buffer.
// A solve ends with a cluster barrier, behind the write-back: no block may overwrite
// its rows, or end, before its neighbours have taken the last one.
//
// What bounds it.  Latency and issue of few warps: 400^2 with its breast phantom on 16
// blocks issues on 36% of its slots and uses the shared memory pipe at 49%, and a step
// cannot be shorter than the slowest warp's passes (about 500 cycles
// of halo wait, 900 of edge pass, 500 to 1200 a pass, 400 of sampling).  So a
// warp holds as few rows as the registers allow: with two rows, 16 warps of 128
// registers (12 of 168 in FP64 and where 24 rows a block are enough) a step of one
// solve takes, with its share of the launches and the DFT,
//   400^2  2.5 us, against 3.6 with four rows and 8 warps of 255 registers,
//   200^2  1.9 us, against 2.5;   333 x 251  2.1 us, against 2.9,
//   FP64 200^2  15 us, against 25 (of which the FP64 pipe is busy 10.7: two lanes a
//   clock and 18 instructions a cell, and the passes' latency beside it).
// Three rows (12 warps) spill and run at 3.64 us on 400^2.  Ez of a warp's own
// rows kept in registers too: 4.19 us, the four-row passes lose the room to load ahead.
// Four rows stay where two would not hold the grid: 512 columns, tall narrow grids.
// The wavefront kernel took 14.3 ms for a 200^2 forward of 1000 steps, this one 2.1.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "cluster.cuh"
#include "fdtd_advance.cuh"
#include "packed.cuh"
#include "solve_desc.h"

namespace tomo {

constexpr int kEdge = 16;            // columns of either side in the edge pass (ncpml <= kEdge - 1)
constexpr int kRows = 4;             // most rows per warp
constexpr int kResidentWarps = 16;   // most warps per block
// The edge pass takes rows in pairs.
__host__ __device__ constexpr int resident_even(int share) { return (share + 1) / 2 * 2; }

// 16 bytes of a row: the columns of one lane in a pass.
template <typename Real>
struct alignas(16) Quad {
    static constexpr int N = 16 / (int)sizeof(Real);
    Real v[N];
};
template <typename Real>
__device__ __forceinline__ Quad<Real> ldq(const Real* p) {
    return *reinterpret_cast<const Quad<Real>*>(p);
}
template <typename Real>
__device__ __forceinline__ void stq(Real* p, const Quad<Real>& q) {
    *reinterpret_cast<Quad<Real>*>(p) = q;
}
// The same where the lane's columns, which start at x, lie left of `end`.
template <bool LAST, typename Real>
__device__ __forceinline__ void stq_until(Real* p, const Quad<Real>& q, int x, int end) {
    if (!LAST || x < end) stq<Real>(p, q);
}
// First column of the right edge: the inner columns, from kEdge on, are whole
// lanes, at least up to column nx - 16.
template <typename Real>
__host__ __device__ constexpr int resident_right(int nx) {
    return kEdge + (nx - 2 * kEdge + 1 + Quad<Real>::N - 1) / Quad<Real>::N * Quad<Real>::N;
}
template <typename Real>
__device__ __forceinline__ Two<Real> half_of(const Quad<Real>& q, int i) {
    return {q.v[2 * i], q.v[2 * i + 1]};
}

// What a warp's longer passes need beside the fields.  It lives in shared memory
// (one per warp): in registers it would push the fields out to local memory, and
// with this kernel's shared memory the first-level cache is too small for that.
template <typename Real>
struct ResidentWarp {
    int iyh[kRows + 1], iye[kRows];   // y-CPML profile indices of the Hx rows from y0-1 and the Ez rows, -1 outside
    int jr[kRows];               // row index in the material box, -1 outside
    int bx0, bx1, nc;
    int src[kRows];              // source column when the row's pass adds the source, else -1
    int hface[kRows];            // NTFF row of the row: 0 lower, 1 upper, -1 none
    bool plane;
    // y-CPML of those rows as {b, a, 1 / kappa, 1 inside a strip}; {0, 0, 1, 0} outside, where
    // the electric form below reduces to the plain one bit for bit
    alignas(16) Real hc[kRows + 1][4], ec[kRows][4];
    Real chezdx, dx, Kp, cs, wave;    // wave: source sample of this step
    int jp, gp, psy, tab, tab2, cpml, mats, pwcol;   // places in shared memory (bytes)
    // plane wave (reference modes); pw_t and pwf_t are of this step
    double pw_t, pw_row[kRows], pw_dxc0, pw_inv_tau;
    float pwf_t, pwf_row[kRows], pwf_col, pwf_xoff, pwf_reach;   // the same in units of tau, for an estimate
};

// One NTFF contour point of the sampler: where Ez of its cell lies in an Ez copy,
// the step to the other Ez of its average (1 or a row), where its H lies, its
// index on the contour and its sign.
struct ResidentPoint {
    unsigned ez : 24, row : 1, negative : 1;
    unsigned short h, contour;
};

// What the sampler needs of the solve, in shared memory for the same reason.
template <typename Real>
struct ResidentSampler {
    int C, S, nrx, total;
    Real *traces, *stage;
};

// Byte offsets of one block's shared memory.  The halo barriers and the Ez copies
// come first: they are placed alike in every block of the cluster, whose
// neighbours write into them.
constexpr int kBarBytes = 128;   // four mbarriers, the words below, padded
constexpr int kLostAt = 32;      // not 0: a halo row did not come, and the whole cluster gives up
constexpr int kIssuedAt = 36;    // rows sent to the block below, and above, by the end of a solve

struct ResidentLayout {
    int pitch;               // elements per Ez row
    int ez_rows;             // rows of one Ez copy
    int br0, br1;            // rows of the material box inside the slab
    int bx0, bx1;            // columns of it in the inner passes (multiples of 4)
    int edge_mat;            // the box meets edge columns in this slab
    int npoints;             // NTFF contour points of the slab
    int hstep;               // elements of the face H of one step: two rows, two columns
    int psi_lo, psi_hi;      // warps of the slab with y-CPML rows: [0, psi_lo) and [psi_hi, warps)
    size_t jp, gp, pwcol, ejp, psy, psx, prof, cpml, tab, tab2, hf, rx, warps, samp, points, mats, emats, total;
};

// share: rows per warp; [ya, yb): the slab; maxrow: the tallest slab of the cluster.
template <typename Real>
__host__ __device__ inline ResidentLayout resident_layout(int nx, int ny, int nc, int nmat, bool ref, int passes,
                                                          int share, int ya, int yb, int maxrow, int mx0, int mx1, int my0,
                                                          int my1, int d) {
    ResidentLayout L{};
    if (d >= 0) {   // NTFF distance, -1: none
        const int v0 = d > ya ? d : ya, v1 = ny - d < yb ? ny - d : yb;
        L.npoints = 2 * (v1 > v0 ? v1 - v0 : 0);
        if (d >= ya && d < yb) L.npoints += nx - 2 * d - 2;
        if (ny - d - 1 >= ya && ny - d - 1 < yb) L.npoints += nx - 2 * d - 2;
    }
    L.pitch = passes * 32 * Quad<Real>::N + 2 * kEdge;
    L.ez_rows = maxrow + share + 1;
    const int warps = (yb - ya + share - 1) / share;
    L.br0 = my0 > ya ? my0 : ya;
    L.br1 = my1 + 1 < yb ? my1 + 1 : yb;
    const int right = resident_right<Real>(nx);
    const int c0 = mx0 > kEdge ? mx0 : kEdge, c1 = mx1 < right - 1 ? mx1 : right - 1;
    L.bx0 = c0 & ~3;
    L.bx1 = (c1 + 4) & ~3;
    const bool box = mx0 <= mx1 && L.br0 < L.br1;
    L.edge_mat = box && (mx0 < kEdge || mx1 >= right);
    if (!box || c0 > c1) L.bx0 = L.bx1 = kEdge;
    if (!box) L.br0 = L.br1 = ya;
    const int brows = L.br1 - L.br0, bw = L.bx1 - L.bx0;
    // a warp has y-CPML rows when one from y0 - 1 to its last is in a strip
    L.psi_lo = 0;
    L.psi_hi = warps;
    if (nc > 0)
        for (int w = 0; w < warps; ++w) {
            const int y0 = ya + share * w;
            if (y0 - 1 <= nc) L.psi_lo = w + 1;
            if (y0 + share - 1 >= ny - nc && L.psi_hi == warps) L.psi_hi = w;
        }
    if (L.psi_hi < L.psi_lo) L.psi_hi = L.psi_lo;
    const int npsi = L.psi_lo + (warps - L.psi_hi);
    size_t o = kBarBytes + 2 * sizeof(Real) * (size_t)L.ez_rows * L.pitch;
    auto take = [&](size_t bytes) {
        const size_t at = o;
        o += (bytes + 15) / 16 * 16;
        return at;
    };
    const size_t cells = brows * bw > 0 ? (size_t)brows * bw : 4;   // never empty: lanes outside read a cell too
    L.jp = take(sizeof(Real) * cells);
    L.gp = take(ref ? sizeof(Real) * (size_t)brows * bw : 0);
    L.pwcol = take(ref ? sizeof(double) * (size_t)bw : 0);
    L.ejp = take(L.edge_mat ? sizeof(Real) * (size_t)brows * 32 : 0);
    L.psy = take(sizeof(Real) * (size_t)npsi * (2 * share + 1) * L.pitch);
    L.psx = take(nc > 0 ? sizeof(Real) * (size_t)warps * 2 * resident_even(share) * 32 : 0);
    L.prof = take(sizeof(Real) * 8 * 32);
    L.cpml = take(sizeof(Real) * 6 * nc);
    L.tab = take(sizeof(Real) * 4 * (size_t)nmat);
    L.tab2 = take(ref ? sizeof(Real) * 2 * (size_t)nmat : 0);
    L.hstep = 2 * L.pitch + 2 * ((maxrow + 1) & ~1);   // a multiple of 16 bytes
    L.hf = take(sizeof(Real) * 2 * (size_t)L.hstep);
    L.warps = take(sizeof(ResidentWarp<Real>) * (size_t)kResidentWarps);
    L.samp = take(sizeof(ResidentSampler<Real>));
    L.points = take(sizeof(ResidentPoint) * (size_t)L.npoints);
    L.rx = take(sizeof(int) * 2 * kMaxRx);
    L.mats = take(cells);
    L.emats = take(L.edge_mat ? (size_t)brows * 32 : 0);
    L.total = o;
    return L;
}

// What every pass needs, in registers.  end: first column of the right edge;
// nr: the warp's valid rows.
template <typename Real>
struct ResidentHot {
    Real chez, Ca0, Cb0;
    int end, nx, nr;
    bool clampnan;
};

// Zero every NaN of v[0..n): one multiply-add per pair finds out whether there
// is any (v * 0 is NaN for a NaN or an infinity), so finite fields pay half an
// instruction per value.
template <typename Real, int N>
__device__ __forceinline__ void clamp_nans(Real (&v)[N]) {
    Two<Real> s = dup2<Real>(Real(0));
#pragma unroll
    for (int i = 0; i + 1 < N; i += 2) s = fma2(Two<Real>{v[i], v[i + 1]}, dup2<Real>(Real(0)), s);
    Real t = s.x + s.y;
    if (N & 1) t += v[N - 1] * Real(0);
    if (t != t) {
#pragma unroll
        for (int i = 0; i < N; ++i)
            if (v[i] != v[i]) v[i] = Real(0);
    }
}

// Incident front exp(-((t - b) / tau)^2) at column x of row j (0 or 1) of the
// warp, the argument in FP64 as FDTD_GPU.cu:290 has it.  t: time of the step
// minus the offset.  It is bound by the FP64 units, so the part of the phase that only
// depends on the column is kept in shared memory.
template <typename Real>
__device__ __forceinline__ Real plane_front(const ResidentWarp<Real>& w, double t, int j, int x) {
    const double b = __dmul_rn(__dadd_rn(w.pw_row[j], shared_at<double>(w.pwcol)[x - w.bx0]), w.pw_dxc0);
    const Real u = (Real)__dmul_rn(__dsub_rn(t, b), w.pw_inv_tau);
    return dev_exp<Real>(-Op<Real>::mul(u, u));
}

// One inner pass: the lane's Quad of columns from x, the warp's rows
// y0 .. y0 + kRows - 1.  hx: from row y0-1; hy: from row y0; cur points at Ez(x, y0) of the
// step's old copy, nxt at the new one; left: Hy of the column before the pass
// (valid in lane 31).  YP: y-CPML rows; MAT: materials; both: the source too.
template <typename Real, int P, int MODE, int R, bool YP, bool MAT, bool LAST>
__device__ __forceinline__ void resident_pass(const ResidentWarp<Real>& w, const ResidentHot<Real>& g,
                                              Quad<Real> (&hx)[R + 1], Quad<Real> (&hy)[R],
                                              const Real (&left)[resident_even(R)],
                                              const Real* cur, Real* nxt, int x) {
    using O = Op<Real>;
    constexpr int N = Quad<Real>::N;
    constexpr bool kRef = MODE == kModeRef;
    const Two<Real> chez2 = dup2<Real>(g.chez), mchez2 = dup2<Real>(-g.chez);
    const int end = g.end;   // the columns from here on belong to the edge pass
    const int lane = threadIdx.x & 31;
    Quad<Real> e[R + 2];   // Ez rows from y0-1
#pragma unroll
    for (int i = 0; i < R + 2; ++i) e[i] = ldq<Real>(cur + (i - 1) * P);
    // materials and Debye current of the rows, loaded ahead of the first store
    Quad<Real> jp[R] = {}, gm[R] = {};
    uint32_t mb[R] = {};
    bool in[R] = {};
    int at[R] = {};
    if constexpr (MAT) {
#pragma unroll
        for (int j = 0; j < R; ++j) {
            // lanes outside the box read its first cells and drop them
            in[j] = w.jr[j] >= 0 && x >= w.bx0 && x < w.bx1;
            at[j] = in[j] ? w.jr[j] * (w.bx1 - w.bx0) + x - w.bx0 : 0;
            const Quad<Real> v = ldq<Real>(shared_at<Real>(w.jp) + at[j]);
            uint32_t m;
            if (N == 4) m = *reinterpret_cast<const uint32_t*>(shared_at<uint8_t>(w.mats) + at[j]);
            else m = *reinterpret_cast<const uint16_t*>(shared_at<uint8_t>(w.mats) + at[j]);
            mb[j] = in[j] ? m : 0u;
#pragma unroll
            for (int i = 0; i < N; ++i) jp[j].v[i] = in[j] ? v.v[i] : Real(0);
            if (kRef && w.plane && in[j]) gm[j] = ldq<Real>(shared_at<Real>(w.gp) + at[j]);
        }
    }
    // y-CPML psi of the rows, likewise
    constexpr bool kStrip = YP && !MAT;
    Quad<Real> psh[R + 1], pse[R];
    if constexpr (kStrip) {
#pragma unroll
        for (int r = 0; r < R + 1; ++r) psh[r] = ldq<Real>(shared_at<Real>(w.psy) + r * P + x);
#pragma unroll
        for (int j = 0; j < R; ++j) pse[j] = ldq<Real>(shared_at<Real>(w.psy) + (R + 1 + j) * P + x);
    }
    // H update
#pragma unroll
    for (int j = 0; j < R; ++j) {
        Real er = __shfl_down_sync(0xffffffffu, e[j + 1].v[0], 1);
        if (lane == 31) er = cur[j * P + N];
#pragma unroll
        for (int i = 0; i < N / 2; ++i) {
            Two<Real> d;
            d.x = O::sub(e[j + 1].v[2 * i + 1], e[j + 1].v[2 * i]);
            d.y = O::sub(2 * i + 2 < N ? e[j + 1].v[(2 * i + 2) % N] : er, e[j + 1].v[2 * i + 1]);
            const Two<Real> h = fma2(chez2, d, half_of(hy[j], i));
            hy[j].v[2 * i] = h.x;
            hy[j].v[2 * i + 1] = h.y;
        }
        if (kRef && g.clampnan) clamp_nans(hy[j].v);
    }
#pragma unroll
    for (int r = 0; r < R + 1; ++r) {
        const int iy = YP && MAT ? w.iyh[r] : -1;
        if constexpr (kStrip) {
            Real b, a, rk, flag;
            load_coefs(w.hc[r], b, a, rk, flag);
            const bool on = flag != Real(0);
#pragma unroll
            for (int i = 0; i < N / 2; ++i) {
                const Two<Real> d = sub2(half_of(e[r + 1], i), half_of(e[r], i)), h = half_of(hx[r], i);
                const Two<Real> ps = fma2(dup2<Real>(b), half_of(psh[r], i), mul2(dup2<Real>(a), d));
                Two<Real> hp = fma2(mul2(mchez2, d), dup2<Real>(rk), h);
                hp = fma2(dup2<Real>(-w.chezdx), ps, hp);
                const Two<Real> hn = fma2(mchez2, d, h);
                hx[r].v[2 * i] = on ? hp.x : hn.x;
                hx[r].v[2 * i + 1] = on ? hp.y : hn.y;
                psh[r].v[2 * i] = ps.x;
                psh[r].v[2 * i + 1] = ps.y;
            }
            stq_until<LAST>(shared_at<Real>(w.psy) + r * P + x, psh[r], x, end);
        } else if (YP && iy >= 0) {
            const Real b = shared_at<Real>(w.cpml)[4 * w.nc + iy], a = shared_at<Real>(w.cpml)[5 * w.nc + iy], rk = shared_at<Real>(w.cpml)[3 * w.nc + iy];
            Real* pp = shared_at<Real>(w.psy) + r * P + x;
            Quad<Real> ps = ldq<Real>(pp);
#pragma unroll
            for (int i = 0; i < N; ++i) {
                const Real d = O::sub(e[r + 1].v[i], e[r].v[i]);
                ps.v[i] = O::fma(b, ps.v[i], O::mul(a, d));
                hx[r].v[i] = O::fma(-O::mul(g.chez, d), rk, hx[r].v[i]);
                hx[r].v[i] = O::fma(-w.chezdx, ps.v[i], hx[r].v[i]);
            }
            stq_until<LAST>(pp, ps, x, end);
        } else {
#pragma unroll
            for (int i = 0; i < N / 2; ++i) {
                const Two<Real> h = fma2(mchez2, sub2(half_of(e[r + 1], i), half_of(e[r], i)), half_of(hx[r], i));
                hx[r].v[2 * i] = h.x;
                hx[r].v[2 * i + 1] = h.y;
            }
        }
        if (kRef && g.clampnan) clamp_nans(hx[r].v);
    }
    // E update
    Quad<Real> out[R], jn[R];
#pragma unroll
    for (int j = 0; j < R; ++j) {
        const Real hv = lane == 31 ? left[j] : hy[j].v[N - 1];
        const Real hl = __shfl_sync(0xffffffffu, hv, (lane + 31) & 31);
        const int iy = YP && MAT ? w.iye[j] : -1;
        Quad<Real> dHy;
#pragma unroll
        for (int i = 0; i < N; ++i) dHy.v[i] = O::sub(hy[j].v[i], i > 0 ? hy[j].v[i - 1] : hl);
        if constexpr (!MAT) {
            const Two<Real> ca = dup2<Real>(g.Ca0), cb = dup2<Real>(g.Cb0);
#pragma unroll
            for (int i = 0; i < N / 2; ++i) {
                const Two<Real> dHx = sub2(half_of(hx[j + 1], i), half_of(hx[j], i)), dy = half_of(dHy, i);
                Two<Real> t;
                if constexpr (kStrip) {
                    const Two<Real> b = dup2<Real>(w.ec[j][0]), a = dup2<Real>(w.ec[j][1]), rk = dup2<Real>(w.ec[j][2]);
                    const Two<Real> ps = fma2(b, half_of(pse[j], i), mul2(a, dHx));
                    pse[j].v[2 * i] = ps.x;
                    pse[j].v[2 * i + 1] = ps.y;
                    if (kRef) {
                        const bool on = w.ec[j][3] != Real(0);
                        const Two<Real> ez = half_of(e[j + 1], i);
                        Two<Real> o = fma2(ca, ez, mul2(mul2(cb, sub2(dy, dHx)), rk));
                        o = fma2(dup2<Real>(-O::mul(g.Cb0, w.dx)), ps, o);
                        const Real px = O::fma(g.Ca0, ez.x, O::sub(O::mul(g.Cb0, dy.x), O::mul(g.Cb0, dHx.x)));
                        const Real py = O::fma(g.Ca0, ez.y, O::sub(O::mul(g.Cb0, dy.y), O::mul(g.Cb0, dHx.y)));
                        out[j].v[2 * i] = on ? o.x : px;
                        out[j].v[2 * i + 1] = on ? o.y : py;
                        continue;
                    }
                    t = mul2(cb, fma2(dup2<Real>(w.dx), sub2(dup2<Real>(Real(0)), ps), sub2(dy, times2(dHx, rk))));
                } else if (kRef)   // scalar products: a packed one may be fused into the difference
                    t = {O::sub(O::mul(g.Cb0, dy.x), O::mul(g.Cb0, dHx.x)), O::sub(O::mul(g.Cb0, dy.y), O::mul(g.Cb0, dHx.y))};
                else t = mul2(cb, sub2(dy, dHx));
                t = fma2(ca, half_of(e[j + 1], i), t);
                out[j].v[2 * i] = t.x;
                out[j].v[2 * i + 1] = t.y;
            }
            if constexpr (kStrip) stq_until<LAST>(shared_at<Real>(w.psy) + (R + 1 + j) * P + x, pse[j], x, end);
        } else {
            Quad<Real> gp{};
            if (in[j]) {
                if (kRef && w.plane) {
                    // the front is exactly zero where it underflows: a float estimate of
                    // the argument, with a margin, saves the FP64 one there
                    if (fabsf(w.pwf_t - w.pwf_row[j] - w.pwf_col * ((float)x - w.pwf_xoff)) < w.pwf_reach) {
#pragma unroll
                        for (int i = 0; i < N; ++i) gp.v[i] = plane_front(w, w.pw_t, j, x + i);
                    }
                    stq<Real>(shared_at<Real>(w.gp) + at[j], gp);
                }
            }
            Quad<Real> psn;
            Real rk = Real(0);
            if (YP && iy >= 0) {
                const Real b = shared_at<Real>(w.cpml)[w.nc + iy], a = shared_at<Real>(w.cpml)[2 * w.nc + iy];
                rk = shared_at<Real>(w.cpml)[iy];
                Real* pp = shared_at<Real>(w.psy) + (R + 1 + j) * P + x;
                psn = ldq<Real>(pp);
#pragma unroll
                for (int i = 0; i < N; ++i)
                    psn.v[i] = O::fma(b, psn.v[i], O::mul(a, O::sub(hx[j + 1].v[i], hx[j].v[i])));
                stq_until<LAST>(pp, psn, x, end);
            }
#pragma unroll
            for (int i = 0; i < N; ++i) {
                const int mi = (mb[j] >> (8 * i)) & kMatMask;
                Real Ca, Cb, Cj, Bp;
                load_coefs(shared_at<Real>(w.tab) + 4 * mi, Ca, Cb, Cj, Bp);
                const Real ez = e[j + 1].v[i], dHx = O::sub(hx[j + 1].v[i], hx[j].v[i]), dy = dHy.v[i];
                Real o;
                if (kRef) {
                    o = O::fma(Ca, ez, O::sub(O::mul(Cb, dy), O::mul(Cb, dHx)));
                    if (w.plane) o = O::fma(shared_at<Real>(w.tab2)[2 * mi], gp.v[i], O::fma(shared_at<Real>(w.tab2)[2 * mi + 1], gm[j].v[i], o));
                } else if (YP && iy >= 0) {
                    o = O::fma(Ca, ez, O::mul(Cb, O::fma(w.dx, O::sub(Real(0), psn.v[i]), O::sub(dy, O::mul(dHx, rk)))));
                } else {
                    o = O::fma(Ca, ez, O::mul(Cb, O::sub(dy, dHx)));
                }
                o = O::fma(-Cj, jp[j].v[i], o);
                if (YP && x + i == w.src[j]) o = O::fma(w.cs, w.wave, o);
                if (kRef) jn[j].v[i] = O::fma(w.Kp, jp[j].v[i], O::mul(Bp, O::add(O::sub(o, ez), O::sub(gp.v[i], gm[j].v[i]))));
                else jn[j].v[i] = O::fma(w.Kp, jp[j].v[i], O::mul(Bp, O::sub(o, ez)));
                if (kRef && YP && iy >= 0) {   // the strip's own formula replaces the result
                    o = O::fma(Ca, ez, O::mul(O::mul(Cb, O::sub(dy, dHx)), rk));
                    o = O::fma(-O::mul(Cb, w.dx), psn.v[i], o);
                }
                out[j].v[i] = o;
            }
        }
        if (kRef && g.clampnan) clamp_nans(out[j].v);
    }
    // stores last: the loads of a row need not wait for the row before
#pragma unroll
    for (int j = 0; j < R; ++j) {
        if (j < g.nr) stq_until<LAST>(nxt + j * P, out[j], x, end);
        if (MAT && in[j]) stq<Real>(shared_at<Real>(w.jp) + at[j], jn[j]);
    }
}

// The edge pass: lanes 0..15 hold columns 0..15, lanes 16..31 columns
// nx-15..nx (the first few of them belong to the inner passes where the inner
// columns are rounded up to whole lanes; their Hy serves the next lane); a pair of
// the lane's rows makes the halves of the packed operations.  The x-CPML terms run
// on every lane: the neutral profile outside the strips leaves the electric
// update's bits as they are, the magnetic one is chosen by select.  hyl: Hy of
// column xq (nx - 16, lane 16's left neighbour), kept redundantly.  YP: y-CPML
// rows; ALL: materials and the source too.
template <typename Real, int P, int MODE, int R, bool YP, bool ALL>
__device__ __forceinline__ void resident_edge(const ResidentWarp<Real>& w, const ResidentHot<Real>& g,
                                              Real (&hx)[resident_even(R) + 1], Two<Real> (&hy)[(R + 1) / 2],
                                              Two<Real> (&hyl)[(R + 1) / 2], const Real* cur, Real* nxt, int xe, int xq,
                                              bool isxh, bool isxe, Real* psx, const Real* prof, bool cpml, bool mats,
                                              Real* ejp, const uint8_t* emats) {
    using O = Op<Real>;
    constexpr bool kRef = MODE == kModeRef;
    constexpr int kPairs = (R + 1) / 2;
    const int lane = threadIdx.x & 31;
    const bool mine = lane < kEdge || xe >= g.end;   // else an inner column: nothing of it is written here
    Real e[R + 2];
#pragma unroll
    for (int i = 0; i < R + 2; ++i) e[i] = cur[xe + (i - 1) * P];
    const Two<Real> chez2 = dup2<Real>(g.chez), ca = dup2<Real>(g.Ca0), cb = dup2<Real>(g.Cb0);
    Real rke, be, ae, rkm, bm, am, unused;
    load_coefs(prof, rke, be, ae, unused);
    load_coefs(prof + 4, rkm, bm, am, unused);
    Two<Real> ph[kPairs] = {}, pe[kPairs] = {};
    if (cpml) {
#pragma unroll
        for (int q = 0; q < kPairs; ++q) {
            ph[q] = *reinterpret_cast<const Two<Real>*>(psx + 2 * q);
            pe[q] = *reinterpret_cast<const Two<Real>*>(psx + 2 * kPairs + 2 * q);
        }
    }
    Real psh[R + 1] = {}, pse[2 * kPairs] = {};
    if constexpr (YP) {
        const Real* const psy = shared_at<Real>(w.psy) + xe;
#pragma unroll
        for (int r = 0; r < R + 1; ++r) psh[r] = psy[r * P];
#pragma unroll
        for (int j = 0; j < R; ++j) pse[j] = psy[(R + 1 + j) * P];
    }
    // Hy
#pragma unroll
    for (int q = 0; q < kPairs; ++q) {
        const Real* const c = cur + 2 * q * P;
        const Two<Real> dEy = sub2(Two<Real>{c[xe + 1], c[xe + P + 1]}, Two<Real>{e[2 * q + 1], e[2 * q + 2]});
        const Two<Real> hn = fma2(chez2, dEy, hy[q]);
        ph[q] = fma2(dup2<Real>(bm), ph[q], mul2(dup2<Real>(am), dEy));
        const Two<Real> hp = fma2(dup2<Real>(w.chezdx), ph[q], fma2(mul2(chez2, dEy), dup2<Real>(rkm), hy[q]));
        hy[q] = {isxh ? hp.x : hn.x, isxh ? hp.y : hn.y};
        hyl[q] = fma2(chez2, sub2(Two<Real>{c[xq + 1], c[xq + P + 1]}, Two<Real>{c[xq], c[xq + P]}), hyl[q]);
    }
    // Hx from row y0-1
#pragma unroll
    for (int r = 0; r < R + 1; ++r) {
        const Real dEx = O::sub(e[r + 1], e[r]), plain = O::fma(-g.chez, dEx, hx[r]);
        if constexpr (YP) {
            Real b, a, rk, on;
            load_coefs(w.hc[r], b, a, rk, on);
            psh[r] = O::fma(b, psh[r], O::mul(a, dEx));
            const Real h = O::fma(-w.chezdx, psh[r], O::fma(-O::mul(g.chez, dEx), rk, hx[r]));
            hx[r] = on != Real(0) ? h : plain;
        } else {
            hx[r] = plain;
        }
    }
    if (kRef && g.clampnan) {
        Real v[4 * kPairs];
#pragma unroll
        for (int q = 0; q < kPairs; ++q) {
            v[4 * q] = hy[q].x; v[4 * q + 1] = hy[q].y; v[4 * q + 2] = hyl[q].x; v[4 * q + 3] = hyl[q].y;
        }
        clamp_nans(v);
#pragma unroll
        for (int q = 0; q < kPairs; ++q) {
            hy[q] = {v[4 * q], v[4 * q + 1]};
            hyl[q] = {v[4 * q + 2], v[4 * q + 3]};
        }
        clamp_nans(hx);
    }
    // E
    const bool inner = xe >= 1 && xe <= g.nx - 1;
#pragma unroll
    for (int q = 0; q < kPairs; ++q) {
        Two<Real> hl{__shfl_up_sync(0xffffffffu, hy[q].x, 1), __shfl_up_sync(0xffffffffu, hy[q].y, 1)};
        if (lane == 16) hl = hyl[q];
        const Two<Real> ez{e[2 * q + 1], e[2 * q + 2]}, dHy = sub2(hy[q], hl);
        const Two<Real> dHx{O::sub(hx[2 * q + 1], hx[2 * q]), O::sub(hx[2 * q + 2], hx[2 * q + 1])};
        pe[q] = fma2(dup2<Real>(be), pe[q], mul2(dup2<Real>(ae), dHy));
        Two<Real> py{}, cy = dHx, rky = dup2<Real>(Real(1)), on{};
        if constexpr (YP) {
            Two<Real> b, a;
            load_coefs(w.ec[2 * q], b.x, a.x, rky.x, on.x);
            load_coefs(w.ec[2 * q + 1], b.y, a.y, rky.y, on.y);
            py = fma2(b, Two<Real>{pse[2 * q], pse[2 * q + 1]}, mul2(a, dHx));
            pse[2 * q] = py.x;
            pse[2 * q + 1] = py.y;
            cy = times2(dHx, rky);
        }
        Two<Real> o;
        if constexpr (!kRef && !ALL) {
            const Two<Real> cx = times2(dup2<Real>(rke), dHy);
            o = fma2(ca, ez, mul2(cb, fma2(dup2<Real>(w.dx), sub2(pe[q], py), sub2(cx, cy))));
        } else {
            Real r[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int j = 2 * q + h;
                const Real z = h ? ez.y : ez.x, dy = h ? dHy.y : dHy.x, dh = h ? dHx.y : dHx.x;
                const Real qx = h ? pe[q].y : pe[q].x, qy = h ? py.y : py.x, c_y = h ? cy.y : cy.x;
                Real Ca = g.Ca0, Cb = g.Cb0, Cj = Real(0), Bp = Real(0), jp = Real(0);
                const bool mat = ALL && mats && w.jr[j] >= 0;
                if (mat) {
                    load_coefs(shared_at<Real>(w.tab) + 4 * (emats[w.jr[j] * 32 + lane] & kMatMask), Ca, Cb, Cj, Bp);
                    jp = ejp[w.jr[j] * 32 + lane];
                }
                Real v;
                if constexpr (kRef) {   // each strip's own formula replaces the result, the rows' last
                    v = O::fma(Ca, z, O::sub(O::mul(Cb, dy), O::mul(Cb, dh)));
                    if (ALL && xe == w.src[j]) v = O::fma(w.cs, w.wave, v);
                    const Real curl = O::mul(Cb, O::sub(dy, dh)), cbdx = O::mul(Cb, w.dx);
                    if (isxe) v = O::fma(cbdx, qx, O::fma(Ca, z, O::mul(curl, rke)));
                    if (YP && (h ? on.y : on.x) != Real(0))
                        v = O::fma(-cbdx, qy, O::fma(Ca, z, O::mul(curl, h ? rky.y : rky.x)));
                } else {
                    v = O::fma(Ca, z, O::mul(Cb, O::fma(w.dx, O::sub(qx, qy), O::sub(O::mul(dy, rke), c_y))));
                    if (mat) v = O::fma(-Cj, jp, v);
                    if (xe == w.src[j]) v = O::fma(w.cs, w.wave, v);
                    if (mat && mine) ejp[w.jr[j] * 32 + lane] = O::fma(w.Kp, jp, O::mul(Bp, O::sub(v, z)));
                }
                r[h] = v;
            }
            if (kRef && g.clampnan) clamp_nans(r);
            o = {r[0], r[1]};
        }
        if (mine && 2 * q < g.nr) nxt[2 * q * P + xe] = inner ? o.x : Real(0);
        if (mine && 2 * q + 1 < g.nr) nxt[(2 * q + 1) * P + xe] = inner ? o.y : Real(0);
    }
    if (cpml) {
#pragma unroll
        for (int q = 0; q < kPairs; ++q) {
            *reinterpret_cast<Two<Real>*>(psx + 2 * q) = ph[q];
            *reinterpret_cast<Two<Real>*>(psx + 2 * kPairs + 2 * q) = pe[q];
        }
    }
    if (YP && mine) {
        Real* const psy = shared_at<Real>(w.psy) + xe;
#pragma unroll
        for (int r = 0; r < R + 1; ++r) psy[r * P] = psh[r];
#pragma unroll
        for (int j = 0; j < R; ++j) psy[(R + 1 + j) * P] = pse[j];
    }
}

// Samples time level k of this launch: the receivers of the slab to the traces,
// its part of the NTFF contour to the staging buffer.  h: H of the face rows and
// columns of this step.
template <typename Real, int P>
__device__ __forceinline__ void resident_sample(const ResidentSampler<Real>& q, const int* rx,
                                                const ResidentPoint* points, const Real* nxt, const Real* h, int k) {
    const int t = blockDim.x - 1 - threadIdx.x;   // the last warps first: they may have no rows
    if (t < q.nrx && rx[t] >= 0) q.traces[(size_t)t * q.S + k] = nxt[rx[t]];   // a block has a thread for each
    for (int i = t; i < q.total; i += blockDim.x) {
        const ResidentPoint p = points[i];
        const Real* z = nxt + p.ez;
        Two<Real> v{h[p.h], Op<Real>::mul(Op<Real>::add(z[0], p.row ? z[P] : z[1]), Real(0.5))};
        if (p.negative) v = {-v.x, -v.y};
        *reinterpret_cast<Two<Real>*>(q.stage + 2 * ((size_t)k * q.C + p.contour)) = v;
    }
}

// What a warp does in a step: two bits per inner pass, then single ones.
enum ResidentTodo : unsigned {
    kPassPlain = 0, kPassMaterial = 1, kPassStrip = 2, kPassAll = 3,
    kHasRows = 1u << 8,        // it has rows
    kEdgeAll = 1u << 9,        // the general edge pass
    kEdgeStrip = 1u << 10,     // the edge pass with y-CPML
    kBelow = 1u << 11, kAbove = 1u << 12,   // it exchanges a row with that block
    kFaceRow = 1u << 13, kFaceColumns = 1u << 14, kSource = 1u << 15, kPlane = 1u << 16, kSample = 1u << 17,
    kSourceAdd = 1u << 18      // the source goes onto the finished row
};

// Advances `count` of the listed solves, from `first` on and around the end, by up
// to nsteps time steps.  gridDim.x is a multiple of the cluster size; cluster q takes
// the solves first + q, first + q + clusters, ...
// The fields are read from and written to copy 0 (D.resident solves do not
// alternate copies).  The contour samples of step D.step + k go to staging
// level k of their half of the buffer.  *error is set when a halo row did not arrive: the
// cluster then gives up together, at the end of the solve.  The sampler reads Ez
// of the row above a horizontal NTFF face from the same block: no slab ends at one.
template <typename Real, int PASSES, int MODE, int R, int W>
__global__ void __launch_bounds__(32 * W, 1)
    fdtd_resident_kernel(const SolveDesc<Real>* __restrict__ descs, int nsolves, int first, int count, int nsteps,
                         int* __restrict__ error) {
    unsigned char* const smem = shared_at<unsigned char>(0);
    constexpr int N = Quad<Real>::N, P = 32 * N * PASSES + 2 * kEdge;
    constexpr bool kRef = MODE == kModeRef;
    constexpr int kEven = resident_even(R);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int rank = (int)cluster_rank(), nblk = (int)cluster_blocks();
    const int nclusters = gridDim.x / nblk;
    // barriers of the row below (two, used in turn) and of the row above; they count
    // on from solve to solve
    const unsigned bar0 = smem_addr(smem);
    volatile int* const lost = reinterpret_cast<volatile int*>(smem + kLostAt);
    if (threadIdx.x < 4) mbar_init(bar0 + 8 * threadIdx.x);
    if (threadIdx.x == 0) *lost = 0;
    int sent = 0;   // rows sent to (and taken from) each neighbour before this solve
    for (int task = blockIdx.x / nblk; task < count; task += nclusters) {
        const SolveDesc<Real>& D = descs[(first + task) % nsolves];
        const int nx = D.nx, ny = D.ny, nc = D.ncpml, S = D.steps_total, n0 = D.step;
        const int ns = min(nsteps, S - n0);
        if (!D.active || ns <= 0) continue;   // the same for every block of the cluster
        const int ya = D.ys[rank], yb = D.ys[rank + 1];
        int maxrow = 0;
        for (int b = 0; b < nblk; ++b) maxrow = max(maxrow, D.ys[b + 1] - D.ys[b]);
        const ResidentLayout L = resident_layout<Real>(nx, ny, nc, D.nmat, kRef, PASSES, R, ya, yb, maxrow, D.mx0, D.mx1,
                                                       D.my0, D.my1, D.nfreq > 0 ? D.nf_d : -1);
        const int pitch = D.pitch;
        Real* const ez_s = reinterpret_cast<Real*>(smem + kBarBytes);
        Real* const jp_s = reinterpret_cast<Real*>(smem + L.jp);
        Real* const gp_s = reinterpret_cast<Real*>(smem + L.gp);
        Real* const ejp_s = reinterpret_cast<Real*>(smem + L.ejp);
        Real* const psx_s = reinterpret_cast<Real*>(smem + L.psx);
        Real* const prof_s = reinterpret_cast<Real*>(smem + L.prof);
        Real* const cpml_s = reinterpret_cast<Real*>(smem + L.cpml);
        Real* const tab_s = reinterpret_cast<Real*>(smem + L.tab);
        Real* const tab2_s = reinterpret_cast<Real*>(smem + L.tab2);
        Real* const hf_s = reinterpret_cast<Real*>(smem + L.hf);
        int* const rx_s = reinterpret_cast<int*>(smem + L.rx);
        uint8_t* const mats_s = smem + L.mats;
        uint8_t* const emats_s = smem + L.emats;
        const int right = resident_right<Real>(nx);
        const int bw = L.bx1 - L.bx0, brows = L.br1 - L.br0;
        const Real* const psi_g = D.psi[0];
        const int psx_h = 0, psx_e = (ny + 1) * 2 * nc;
        const int psy_h = 2 * (ny + 1) * 2 * nc, psy_e = psy_h + 2 * nc * (nx + 1);

        // ---- load the slab
        __syncthreads();   // the previous solve's sampling is done with the shared memory
        const int nthr = blockDim.x, t = threadIdx.x;
        // rows by warps, 16 bytes a lane: the padding of the field rows is zero
        const int nwarp = nthr >> 5;
        for (int l = warp; l < L.ez_rows; l += nwarp) {
            const int y = ya - 1 + l;
            const Real* const src = D.ez[0] + (size_t)min(y, ny) * pitch;
            Real* const dst = ez_s + l * P;
#pragma unroll
            for (int i = 0; i < (P / N + 31) / 32; ++i) {
                const int x = N * (32 * i + lane);
                if (x < P) {
                    stq<Real>(dst + x, y <= ny && n0 > 0 ? ldq<Real>(src + x) : Quad<Real>{});
                    stq<Real>(dst + L.ez_rows * P + x, Quad<Real>{});
                }
            }
        }
        // the box by Quads (its columns start on a multiple of 4, rows are padded)
#pragma unroll 4
        for (int i = t; i < brows * (bw / N); i += nthr) {
            const int r = i / (bw / N), q = N * (i - r * (bw / N)), x = L.bx0 + q, y = L.br0 + r;
            Quad<Real> v = n0 > 0 ? ldq<Real>(D.jp[0] + x + (size_t)y * pitch) : Quad<Real>{};
            uchar4 m{};
            const uint8_t* const mg = D.mat + x + (size_t)y * D.mpitch;
            if (N == 4) m = *reinterpret_cast<const uchar4*>(mg);
            else { m.x = mg[0]; m.y = mg[1]; }
            // the box's columns may reach past the inner columns by up to three: those stay vacuum
            uint8_t mb[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
            for (int c = 0; c < N; ++c)
                if (x + c >= right) {
                    v.v[c] = Real(0);
                    mb[c] = 0;
                }
            stq<Real>(jp_s + r * bw + q, v);
#pragma unroll
            for (int c = 0; c < N; ++c) mats_s[r * bw + q + c] = mb[c];
        }
        if (kRef)   // the columns' part of a plane wave's phase
            for (int i = t; i < bw; i += nthr)
                reinterpret_cast<double*>(smem + L.pwcol)[i] = __dmul_rn(D.pw_kx, (double)(L.bx0 + i) - D.pw_xoff);
        if (L.edge_mat)
            for (int i = t; i < brows * 32; i += nthr) {
                const int r = i >> 5, ln = i & 31, x = ln < 16 ? ln : nx - 31 + ln, y = L.br0 + r;
                ejp_s[i] = D.jp[0][x + (size_t)y * pitch];
                emats_s[i] = D.mat[x + (size_t)y * D.mpitch];
            }
        for (int i = t; i < D.nmat * 4; i += nthr) tab_s[i] = D.mtab[(i >> 2) * kMatCoef + (i & 3)];
        if (kRef)
            for (int i = t; i < D.nmat; i += nthr) {
                tab2_s[2 * i] = D.mtab[i * kMatCoef + kCi];
                tab2_s[2 * i + 1] = D.mtab[i * kMatCoef + kCp];
            }
        for (int i = t; i < 6 * nc; i += nthr) cpml_s[i] = D.cpml[i];
        for (int i = t; i < D.nrx; i += nthr) {   // receivers of this slab: index in the Ez copy, else -1
            const int x = D.rx[2 * i], y = D.rx[2 * i + 1];
            rx_s[i] = (y >= ya && y < yb) ? (y - ya + 1) * P + x : -1;
        }
        ResidentSampler<Real>* const samp = reinterpret_cast<ResidentSampler<Real>*>(smem + L.samp);
        ResidentPoint* const points_s = reinterpret_cast<ResidentPoint*>(smem + L.points);
        if (t == 0) *samp = {D.n_contour, S, D.nrx, L.npoints, D.traces + n0, D.stage + stage_half(D, n0, nsteps)};
        {
            // vertical faces, then the lower and the upper horizontal face; the H buffer of a
            // step holds Hx of the two face rows, then Hy of the two face columns
            const int d = D.nf_d, v0 = max(d, ya), nv = max(0, min(ny - d, yb) - v0), nh = nx - 2 * d - 2;
            const bool lower = d >= ya && d < yb;
            for (int i = t; i < L.npoints; i += nthr) {
                ResidentPoint q{};
                if (i < 2 * nv) {
                    const int right = i & 1, y = v0 + (i >> 1);
                    q.ez = (y - ya + 1) * P + (right ? nx - d - 1 : d);
                    q.h = 2 * P + 2 * (y - ya) + right;
                    q.contour = right ? contour_index_xp(nx, ny, d, y) : contour_index_xn(nx, ny, d, y);
                    q.negative = !right;
                } else {
                    int x = i - 2 * nv;
                    const bool up = !lower || x >= nh;
                    if (lower && up) x -= nh;
                    x += d + 1;
                    q.ez = ((up ? ny - d - 1 : d) - ya + 1) * P + x;
                    q.h = (up ? P : 0) + x;
                    q.contour = up ? contour_index_yp(nx, ny, d, x) : contour_index_yn(nx, ny, d, x);
                    q.row = 1;
                    q.negative = up;
                }
                points_s[i] = q;
            }
        }
        // edge lanes: column, strips and profile
        const int xe = lane < 16 ? lane : nx - 31 + lane;
        const int ixh = xe < nc ? nc - 1 - xe : (xe >= nx - nc && xe < nx ? xe - nx + nc : -1);
        const int ixe = (xe >= 1 && xe <= nc) ? nc - xe : (xe >= nx - nc && xe <= nx - 1 ? xe - nx + nc : -1);
        if (t < 32) {
            const int ie = ixe >= 0 ? ixe : 0, ih = ixh >= 0 ? ixh : 0;
            for (int q = 0; q < 3; ++q) {
                // outside the strips the neutral profile (1 / kappa = 1, b = a = 0)
                const Real off = q == 0 ? Real(1) : Real(0);
                prof_s[8 * lane + q] = ixe >= 0 ? D.cpml[q * nc + ie] : off;
                prof_s[8 * lane + 4 + q] = ixh >= 0 ? D.cpml[(3 + q) * nc + ih] : off;
            }
            prof_s[8 * lane + 3] = prof_s[8 * lane + 7] = Real(0);
        }

        // ---- the warp's rows
        ResidentWarp<Real>& w = reinterpret_cast<ResidentWarp<Real>*>(smem + L.warps)[warp];
        const int y0 = ya + R * warp, l0 = y0 - ya + 1, nr = max(0, min(R, yb - y0));
        w.nc = nc;   // every lane writes the same values
        bool ypml = false;
#pragma unroll
        for (int r = 0; r < R + 1; ++r) {
            const int m = y0 - 1 + r;
            w.iyh[r] = m < nc ? nc - 1 - m : ((m >= ny - nc && m < ny) ? m - ny + nc : -1);
            ypml |= w.iyh[r] >= 0;
        }
#pragma unroll
        for (int j = 0; j < kRows; ++j) {
            const int m = y0 + j;
            w.iye[j] = j >= R ? -1 : m <= nc ? nc - m : ((m >= ny - nc && m <= ny - 1) ? m - ny + nc : -1);
            ypml |= w.iye[j] >= 0;
            w.jr[j] = (j < R && m >= L.br0 && m < L.br1) ? m - L.br0 : -1;
            const bool valid = j < nr;
            w.src[j] = -1;
            w.hface[j] = (D.nfreq > 0 && valid) ? (m == D.nf_d ? 0 : (m == ny - D.nf_d - 1 ? 1 : -1)) : -1;
        }
        w.bx0 = L.bx0;
        w.bx1 = L.bx1;
        ResidentHot<Real> g;
        g.chez = D.chez;
        g.Ca0 = D.mtab[kCa];
        g.Cb0 = D.mtab[kCb];
        g.end = right;
        g.nx = nx;
        g.nr = nr;
        g.clampnan = kRef && (D.flags & kNanClamp) != 0;
        w.dx = D.dx;
        w.chezdx = Op<Real>::mul(D.chez, D.dx);
        w.Kp = D.Kp;
        w.jp = (int)L.jp;
        w.gp = (int)L.gp;
        w.pwcol = (int)L.pwcol;
        w.tab = (int)L.tab;
        w.tab2 = (int)L.tab2;
        w.cpml = (int)L.cpml;
        w.mats = (int)L.mats;
        w.cs = w.wave = Real(0);
        const int slot = warp < L.psi_lo ? warp : warp - L.psi_hi + L.psi_lo;
        w.psy = (int)(L.psy + sizeof(Real) * (size_t)slot * (2 * R + 1) * P);
        Real* const psy = shared_at<Real>(w.psy);
        Real* const psx = psx_s + ((size_t)warp * 32 + lane) * 2 * kEven;
        const bool has_src = (D.flags & kPointSource) && D.src_y >= y0 && D.src_y < y0 + nr;
        // a source in the background is added to the finished row; among materials (the Debye
        // current takes it in) or in a strip of the reference modes the general passes do it
        bool src_all = false;
        if (has_src) {
            const int mat = D.mat[D.src_x + (size_t)D.src_y * D.mpitch] & kMatMask;
            w.cs = D.mtab[mat * kMatCoef + kCs];
            src_all = mat != 0 || kRef;
#pragma unroll
            for (int j = 0; j < R; ++j)
                if (src_all && y0 + j == D.src_y) w.src[j] = D.src_x;
        }
        w.plane = kRef && (D.flags & kPlaneWave) != 0;
        if (kRef) {
            w.pw_dxc0 = D.pw_dxc0;
            w.pw_inv_tau = D.pw_inv_tau;
#pragma unroll
            for (int j = 0; j < R; ++j) {
                w.pw_row[j] = __dmul_rn(D.pw_ky, (double)(y0 + j) - D.pw_yoff);
                w.pwf_row[j] = (float)(w.pw_row[j] * D.pw_dxc0 * D.pw_inv_tau);
            }
            // exp(-u^2) is zero past |u| = 10.2 in FP32 and 27.3 in FP64; the reach adds the
            // lane's other columns and the rounding of the estimate
            w.pwf_col = (float)(D.pw_kx * D.pw_dxc0 * D.pw_inv_tau);
            w.pwf_xoff = (float)D.pw_xoff;
            w.pwf_reach = (sizeof(Real) == 8 ? 27.6f : 10.5f) + N * fabsf(w.pwf_col) +
                          1e-5f * (float)(D.pw_inv_tau * (S * D.dt + fabs(D.pw_t0l) + (nx + ny) * D.pw_dxc0));
        }
        if (lane < R + 1) {
            const int iy = w.iyh[lane];
            w.hc[lane][0] = iy >= 0 ? D.cpml[4 * nc + iy] : Real(0);
            w.hc[lane][1] = iy >= 0 ? D.cpml[5 * nc + iy] : Real(0);
            w.hc[lane][2] = iy >= 0 ? D.cpml[3 * nc + iy] : Real(1);
            w.hc[lane][3] = iy >= 0 ? Real(1) : Real(0);
        } else if (lane < 2 * R + 1) {
            const int at = lane - R - 1, iy = w.iye[at];
            w.ec[at][0] = iy >= 0 ? D.cpml[nc + iy] : Real(0);
            w.ec[at][1] = iy >= 0 ? D.cpml[2 * nc + iy] : Real(0);
            w.ec[at][2] = iy >= 0 ? D.cpml[iy] : Real(1);
            w.ec[at][3] = iy >= 0 ? Real(1) : Real(0);
        }
        __syncwarp();
        // passes with materials, and with a source that the pass adds
        bool box_rows = false;
#pragma unroll
        for (int j = 0; j < R; ++j) box_rows |= w.jr[j] >= 0;
        unsigned matmask = 0, srcmask = 0;
#pragma unroll
        for (int c = 0; c < PASSES; ++c) {
            const int xa = kEdge + 32 * N * c, xb = xa + 32 * N;
            if (box_rows && L.bx0 < xb && L.bx1 > xa && L.bx0 < L.bx1) matmask |= 1u << c;
            if (src_all && D.src_x >= xa && D.src_x < min(xb, right)) srcmask |= 1u << c;
        }
        const bool nfaces = D.nfreq > 0, cpml = nc > 0;
        // What the warp does in every step, one bit each.  The reduction leaves the word in a
        // uniform register: the step's branches then cost no divergence handling.
        const bool edge_gen = (src_all && srcmask == 0) || (L.edge_mat && box_rows);
        const bool from_below = nr > 0 && warp == 0 && rank > 0, from_above = nr > 0 && y0 + nr == yb && rank + 1 < nblk;
        unsigned todo = 0;
#pragma unroll
        for (int c = 0; c < PASSES; ++c) {
            const bool mat = (matmask >> c) & 1u, src = (srcmask >> c) & 1u;
            const unsigned kind = src || (ypml && mat) ? kPassAll : ypml ? kPassStrip : mat ? kPassMaterial : kPassPlain;
            todo |= kind << (2 * c);
        }
        if (nr > 0) todo |= kHasRows;
        if (edge_gen) todo |= kEdgeAll;
        if (ypml) todo |= kEdgeStrip;
        if (from_below) todo |= kBelow;
        if (from_above) todo |= kAbove;
#pragma unroll
        for (int j = 0; j < R; ++j)
            if (w.hface[j] >= 0) todo |= kFaceRow;
        if (nfaces) todo |= kFaceColumns;
        if (has_src) todo |= kSource;
        if (has_src && !src_all) todo |= kSourceAdd;
        if (kRef && (D.flags & kPlaneWave)) todo |= kPlane;
        if (32 * (nwarp - 1 - warp) < max(L.npoints, (int)D.nrx)) todo |= kSample;
        todo = __reduce_or_sync(0xffffffffu, todo);

        // column whose Hy ehyl follows: the left neighbour of lane 16, and in lanes 0 and 1
        // the two NTFF face columns (inner columns, without x-CPML)
        const int xq = nfaces && lane < 2 ? (lane ? nx - D.nf_d - 1 : D.nf_d) : nx - kEdge;

        // fields of the warp's rows
        Quad<Real> hx[PASSES][R + 1], hy[PASSES][R];
        Real ehx[kEven + 1] = {};
        Two<Real> ehy[kEven / 2] = {}, ehyl[kEven / 2] = {};
        // Hx and Hy are zero from column nx and row ny on, in memory too
        const Real *const hx_g = D.hx[0], *const hy_g = D.hy[0];
        auto row_of = [&](const Real* f, int m) { return f + (size_t)min(m, ny) * pitch; };
        if (nr > 0) {
#pragma unroll
            for (int c = 0; c < PASSES; ++c) {
                const int x = kEdge + 32 * N * c + N * lane;
#pragma unroll
                for (int r = 0; r < R + 1; ++r) hx[c][r] = n0 > 0 ? ldq<Real>(row_of(hx_g, y0 - 1 + r) + x) : Quad<Real>{};
#pragma unroll
                for (int j = 0; j < R; ++j) hy[c][j] = n0 > 0 ? ldq<Real>(row_of(hy_g, y0 + j) + x) : Quad<Real>{};
            }
#pragma unroll
            for (int r = 0; r < R + 1; ++r) ehx[r] = row_of(hx_g, y0 - 1 + r)[xe];
#pragma unroll
            for (int q = 0; q < kEven / 2; ++q) {
                ehy[q] = {row_of(hy_g, y0 + 2 * q)[xe], row_of(hy_g, y0 + 2 * q + 1)[xe]};
                ehyl[q] = {row_of(hy_g, y0 + 2 * q)[xq], row_of(hy_g, y0 + 2 * q + 1)[xq]};
            }
            if (nc > 0) {
                const int xh = xe < nc ? xe : xe - (nx - nc) + nc, xq = xe <= nc ? xe - 1 : xe - (nx - nc) + nc;
#pragma unroll
                for (int j = 0; j < R; ++j) {
                    const int m = y0 + j;
                    psx[j] = (ixh >= 0 && m < ny) ? psi_g[psx_h + (size_t)m * 2 * nc + xh] : Real(0);
                    psx[kEven + j] = (ixe >= 0 && m < ny) ? psi_g[psx_e + (size_t)m * 2 * nc + xq] : Real(0);
                }
            }
            if (ypml)
#pragma unroll 4
                for (int x = lane; x < P; x += 32) {
#pragma unroll
                    for (int r = 0; r < R + 1; ++r) {
                        const int m = y0 - 1 + r, yh = m < nc ? m : m - (ny - nc) + nc;
                        psy[r * P + x] = (w.iyh[r] >= 0 && x < nx) ? psi_g[psy_h + (size_t)yh * (nx + 1) + x] : Real(0);
                    }
#pragma unroll
                    for (int j = 0; j < R; ++j) {
                        const int m = y0 + j, ye = m <= nc ? m - 1 : m - (ny - nc) + nc;
                        psy[(R + 1 + j) * P + x] =
                            (w.iye[j] >= 0 && x >= 1 && x <= nx - 1) ? psi_g[psy_e + (size_t)ye * (nx + 1) + x] : Real(0);
                    }
                }
        }
        __syncthreads();
        if (kRef && w.plane && nr > 0) {
            // the front of the previous half step, which every later step takes over
            const double t1 = __dsub_rn(__dmul_rn((double)n0 - 0.5, D.dt), D.pw_t0l);
#pragma unroll
            for (int j = 0; j < R; ++j)
                if (w.jr[j] >= 0 && j < nr)
                    for (int i = lane; i < bw; i += 32) {
                        const bool near = fabsf((float)(t1 * w.pw_inv_tau) - w.pwf_row[j] -
                                                w.pwf_col * ((float)(L.bx0 + i) - w.pwf_xoff)) < w.pwf_reach;
                        gp_s[w.jr[j] * bw + i] = near ? plane_front(w, t1, j, L.bx0 + i) : Real(0);
                    }
        }
        proxy_fence();   // the halo rows, zeroed here, are written by the neighbours' copies from now on
        __syncwarp();
        cluster_arrive();
        cluster_wait();

        // ---- time steps
        const Real* const wave = D.src_wave + n0;
        const double pw_t0l = D.pw_t0l, dt = D.dt;
        const int copy = L.ez_rows * P, below = rank > 0 ? (ya - D.ys[rank - 1] + 1) * P : 0;
        // The warp that owns the slab's first row takes the row below from that
        // block and sends it its own; likewise the last row and the block above.
        const int src_at = has_src ? (D.src_y - ya + 1) * P + D.src_x : 0;
        int until = ns;   // the step at which the warp gave up its exchange
        for (int k = 0; k < ns; ++k) {
            Real* const cur = ez_s + (k & 1) * copy;
            Real* const nxt = ez_s + (~k & 1) * copy;
            if (todo & (kBelow | kAbove)) {
                // message m goes to barrier m & 1, its phase the parity of m / 2; a
                // neighbour is at most one message ahead
                const int m = sent + k - 1;
                const unsigned parity = (m >> 1) & 1, slot8 = 8 * (unsigned)(m & 1);
                bool came = true;
                if (k > 0 && k < until) {
                    if (todo & kBelow) came = mbar_wait(bar0 + slot8, parity, lost);
                    if ((todo & kAbove) && came) came = mbar_wait(bar0 + 16 + slot8, parity, lost);
                }
                if (__any_sync(0xffffffffu, !came)) {
                    until = k;
                    *error = 1;
                    if (lane < nblk) remote_store(remote_addr(bar0 + kLostAt, lane), 1);
                }
                if (k + 1 < ns && k < until && lane == 0) {
                    const unsigned bytes = (unsigned)(P * sizeof(Real)), next8 = 8 * (unsigned)((m + 1) & 1);
                    if (todo & kBelow) mbar_arm(bar0 + next8, bytes);
                    if (todo & kAbove) mbar_arm(bar0 + 16 + next8, bytes);
                }
            }
            if (todo & kHasRows) {
                if (todo & (kSource | kPlane)) {
                    if (lane == 0) {
                        if (todo & kSource) w.wave = wave[k];
                        if (todo & kPlane) {
                            const double tn = __dsub_rn(__dmul_rn((double)(n0 + k) + 0.5, dt), pw_t0l);
                            w.pw_t = tn;
                            w.pwf_t = (float)(tn * w.pw_inv_tau);
                        }
                    }
                    __syncwarp();
                }
                const Real* const rowc = cur + l0 * P;
                Real* const rown = nxt + l0 * P;
#define TOMO_EDGE(YP, ALL)                                                                                       \
    resident_edge<Real, P, MODE, R, YP, ALL>(w, g, ehx, ehy, ehyl, rowc, rown, xe, xq, ixh >= 0, ixe >= 0, psx,     \
                                          prof_s + 8 * lane, cpml, L.edge_mat != 0, ejp_s, emats_s)
                if ((todo & kEdgeAll) && (todo & kEdgeStrip)) TOMO_EDGE(true, true);
                else if (todo & kEdgeAll) TOMO_EDGE(false, true);
                else if (todo & kEdgeStrip) TOMO_EDGE(true, false);
                else TOMO_EDGE(false, false);
#undef TOMO_EDGE
                Real left[kEven];
#pragma unroll
                for (int q = 0; q < kEven / 2; ++q) {
                    left[2 * q] = __shfl_sync(0xffffffffu, ehy[q].x, 15);
                    left[2 * q + 1] = __shfl_sync(0xffffffffu, ehy[q].y, 15);
                }
#pragma unroll
                for (int c = 0; c < PASSES; ++c) {
                    const int x = kEdge + 32 * N * c + N * lane;
                    constexpr int kLast = PASSES - 1;
                    const unsigned kind = (todo >> (2 * c)) & 3u;
#define TOMO_PASS(YP, MAT)                                                                                    \
    do {                                                                                                      \
        if (c == kLast)                                                                                       \
            resident_pass<Real, P, MODE, R, YP, MAT, true>(w, g, hx[c], hy[c], left, rowc + x, rown + x, x); \
        else                                                                                                  \
            resident_pass<Real, P, MODE, R, YP, MAT, false>(w, g, hx[c], hy[c], left, rowc + x, rown + x, x); \
    } while (0)
                    if (kind == kPassAll) TOMO_PASS(true, true);
                    else if (kind == kPassStrip) TOMO_PASS(true, false);
                    else if (kind == kPassMaterial) TOMO_PASS(false, true);
                    else TOMO_PASS(false, false);
#undef TOMO_PASS
#pragma unroll
                    for (int j = 0; j < R; ++j) left[j] = hy[c][j].v[N - 1];
                }
                if (todo & kSourceAdd) {
                    __syncwarp();
                    if (lane == 0) {
                        Real* const z = nxt + src_at;
                        *z = Op<Real>::fma(w.cs, w.wave, *z);
                    }
                }
                // H of the NTFF faces for the sampler: Hx of the face rows, Hy of the face columns
                if (todo & kFaceRow) {
#pragma unroll
                    for (int j = 0; j < R; ++j)
                        if (w.hface[j] >= 0) {
                            Real* const o = hf_s + (k & 1) * L.hstep + w.hface[j] * P;
#pragma unroll
                            for (int c = 0; c < PASSES; ++c) {
                                const int x = kEdge + 32 * N * c + N * lane;
                                if (c + 1 < PASSES) stq_until<false>(o + x, hx[c][j + 1], x, g.end);
                                else stq_until<true>(o + x, hx[c][j + 1], x, g.end);
                            }
                            o[xe] = ehx[j + 1];
                        }
                }
                if ((todo & kFaceColumns) && lane < 2) {
                    Real* const o = hf_s + (k & 1) * L.hstep + 2 * P + 2 * (y0 - ya) + lane;
#pragma unroll
                    for (int q = 0; q < kEven / 2; ++q) {
                        if (2 * q < nr) o[4 * q] = ehyl[q].x;
                        if (2 * q + 1 < nr) o[4 * q + 2] = ehyl[q].y;
                    }
                }
                // boundary rows of the slab to the neighbours' halo rows
                if ((todo & (kBelow | kAbove)) && k + 1 < ns && k < until) {
                    proxy_fence();   // the row is written by every lane, and read by the copy
                    __syncwarp();
                    if (lane == 0) {
                        const unsigned at8 = 8 * (unsigned)((sent + k) & 1), bytes = (unsigned)(P * sizeof(Real));
                        if (todo & kBelow)
                            copy_row(remote_addr(smem_addr(nxt + below), rank - 1), smem_addr(nxt + l0 * P), bytes,
                                     remote_addr(bar0 + 16, rank - 1) + at8);
                        if (todo & kAbove)
                            copy_row(remote_addr(smem_addr(nxt), rank + 1), smem_addr(nxt + (l0 + nr - 1) * P), bytes,
                                     remote_addr(bar0, rank + 1) + at8);
                    }
                }
            }
            __syncthreads();
            // ---- sample the new time level
            if (todo & kSample)
                resident_sample<Real, P>(*samp, rx_s, points_s, nxt, hf_s + (k & 1) * L.hstep, k);
        }
        // The neighbours have not answered the last row sent to them.  A block may overwrite
        // its rows, or end, once every block of the cluster has waited for its own; the
        // write-back hides the barrier.
        const int issued = sent + (until < ns ? until : ns - 1);
        if (lane == 0 && (todo & kBelow)) reinterpret_cast<int*>(smem + kIssuedAt)[0] = issued;
        if (lane == 0 && (todo & kAbove)) reinterpret_cast<int*>(smem + kIssuedAt)[1] = issued;
        __syncwarp();
        cluster_arrive();

        // ---- write the slab back
        const Real* const fin = ez_s + (ns & 1) * copy;
        for (int r = warp; r < yb - ya; r += nwarp) {
            Real* const dst = D.ez[0] + (size_t)(ya + r) * pitch;
            for (int x = N * lane; x < P; x += 32 * N) stq<Real>(dst + x, ldq<Real>(fin + (r + 1) * P + x));
        }
        for (int i = t; i < brows * (bw / N); i += nthr) {
            const int r = i / (bw / N), q = N * (i - r * (bw / N)), x = L.bx0 + q;
            stq_until<true>(D.jp[0] + x + (size_t)(L.br0 + r) * pitch, ldq<Real>(jp_s + r * bw + q), x, right);
        }
        if (L.edge_mat)
            for (int i = t; i < brows * 32; i += nthr) {
                const int ln = i & 31, x = ln < 16 ? ln : nx - 31 + ln;
                if (x >= 1 && x <= nx - 1 && (ln < 16 || x >= right)) D.jp[0][x + (size_t)(L.br0 + (i >> 5)) * pitch] = ejp_s[i];
            }
        Real* const psi_o = D.psi[0];
        auto put = [&](Real* f, int m, int x, Real v) {
            if (x < nx) f[x + (size_t)m * pitch] = v;
        };
#pragma unroll
        for (int r = 0; r < R + 1; ++r) {
            // the row below the warp's rows belongs to another warp, except row 0
            if (r == 0 ? (nr == 0 || y0 != 1) : r > nr) continue;
            const int m = y0 - 1 + r;
#pragma unroll
            for (int c = 0; c < PASSES; ++c) {
                const int x = kEdge + 32 * N * c + N * lane;
                if (x < right) stq<Real>(D.hx[0] + x + (size_t)m * pitch, hx[c][r]);
            }
            put(D.hx[0], m, xe, ehx[r]);
            if (w.iyh[r] >= 0) {
                const int yh = m < nc ? m : m - (ny - nc) + nc;
                for (int x = lane; x < nx; x += 32) psi_o[psy_h + (size_t)yh * (nx + 1) + x] = psy[r * P + x];
            }
        }
#pragma unroll
        for (int j = 0; j < R; ++j) {
            if (j >= nr) continue;
            const int m = y0 + j;
#pragma unroll
            for (int c = 0; c < PASSES; ++c) {
                const int x = kEdge + 32 * N * c + N * lane;
                if (x < right) stq<Real>(D.hy[0] + x + (size_t)m * pitch, hy[c][j]);
            }
            put(D.hy[0], m, xe, j & 1 ? ehy[j / 2].y : ehy[j / 2].x);
            if (ixh >= 0) {
                const int xh = xe < nc ? xe : xe - (nx - nc) + nc;
                psi_o[psx_h + (size_t)m * 2 * nc + xh] = psx[j];
            }
            if (ixe >= 0) {
                const int xq = xe <= nc ? xe - 1 : xe - (nx - nc) + nc;
                psi_o[psx_e + (size_t)m * 2 * nc + xq] = psx[kEven + j];
            }
            if (w.iye[j] >= 0) {
                const int ye = m <= nc ? m - 1 : m - (ny - nc) + nc;
                for (int x = 1 + lane; x <= nx - 1; x += 32)
                    psi_o[psy_e + (size_t)ye * (nx + 1) + x] = psy[(R + 1 + j) * P + x];
            }
        }
        __syncwarp();
        cluster_wait();
        if (*lost) {   // the same in every block
            // rows that are still on their way: none may arrive after its receiver has ended
            auto drain = [&](unsigned bar, unsigned theirs) {
                for (int m = sent + until - 1, end = remote_load(theirs); m < end; ++m) {
                    if (m >= issued && lane == 0) mbar_arm(bar + 8 * (unsigned)(m & 1), (unsigned)(P * sizeof(Real)));
                    __syncwarp();
                    if (!__all_sync(0xffffffffu, mbar_wait(bar + 8 * (unsigned)(m & 1), (m >> 1) & 1, nullptr))) return;
                }
            };
            if (todo & kBelow) drain(bar0, remote_addr(bar0 + kIssuedAt + 4, rank - 1));
            if (todo & kAbove) drain(bar0 + 16, remote_addr(bar0 + kIssuedAt, rank + 1));
            __syncwarp();
            cluster_arrive();
            cluster_wait();
            return;
        }
        sent += ns - 1;
    }
}

// ------------------------------------------------------------------- host side
// Warps of a block: the tallest slab's, and a thread for every receiver (slabs of four rows
// are one warp tall).  A loop over the receivers instead costs up to 0.8% (400^2, 256 candidates: 618 and 623 ms).
__host__ __device__ constexpr int resident_warps(int tall, int share, int nrx) {
    const int rows = (tall + share - 1) / share, receivers = (nrx + 31) / 32;
    return rows > receivers ? rows : receivers;
}

template <typename Real>
using ResidentFn = void (*)(const SolveDesc<Real>*, int, int, int, int, int*);
// Rows per warp and most warps of a block.
struct ResidentShape {
    int share, warps;
};
// The compiled kernel of a number of inner passes, a mode and a shape (null: none).
template <typename Real>
ResidentFn<Real> resident_kernel_for(int passes, int mode, ResidentShape shape);

}  // namespace tomo
