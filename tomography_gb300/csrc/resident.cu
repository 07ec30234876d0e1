// Host side of the resident kernel: which problems fit it, how the rows are cut
// into slabs, and the cluster launch.
#include "engine_impl.cuh"

namespace tomo {

// The shapes in the order of their speed: the first that holds a batch takes it.  Two
// rows a warp beat four wherever both hold the slabs (400^2: 2.98 against 3.60 us a step);
// 12 warps leave 168 registers, 16 leave 128 and some spills (384 rows of 400: 2.89
// against 3.17 us).  Which of them are compiled for a number of inner passes follows the
// grids in use, not a limit of the kernel: two rows on 16 warps and 16 blocks hold 512
// rows, any square of one to three passes (up to 415 columns); four rows are there for
// what two do not hold, tall grids of one pass (768 rows) and four passes, where the
// fields of two rows take 80 of 16 warps' 128 registers.  The reference modes' problem
// (401^2) takes three passes, FP64 one to three.  Other grids take the wavefront kernel.
static constexpr ResidentShape kShapes[] = {{2, 12}, {2, 16}, {4, 12}, {4, 8}};

template <typename Real>
bool resident_plan(const ProblemClass& pc, const SolveLayout& lay, int blocks, ResidentPlan& p) {
    const tomo_spec& s = pc.spec;
    const int rows = pc.ny - 1;
    // the edge pass holds the PEC columns and the x-CPML; background cells carry no Debye current
    if (pc.nc > kEdge - 1 || pc.nx < 3 * kEdge || blocks > kMaxSlabs || rows < 4 * blocks) return false;
    if (s.mode == TOMO_MODE_BREAST && s.bg_del_eps != 0) return false;
    if (pc.nfreq > 0 && s.nf2ff_d < pc.nc) return false;   // Hy of the NTFF face columns has no x-CPML
    if (s.mode != TOMO_MODE_BREAST) {
        // the reference's strips replace the whole update: patches stay clear of them
        const int r = (int)std::ceil(s.breast_radius / s.dx) + 2, clear = std::max(kEdge, pc.nc + 1);
        if (pc.nx / 2 - r < clear || pc.nx / 2 + r > pc.nx - clear - 1) return false;
    }
    const int right = resident_right<Real>(pc.nx), width = 32 * Quad<Real>::N;
    if (right > pc.nx - std::max(pc.nc, 1)) return false;   // the x-CPML and PEC columns belong to the edge pass
    p.blocks = blocks;
    p.passes = (right - kEdge + width - 1) / width;
    bool holds = false;
    for (const ResidentShape& q : kShapes)
        holds |= rows <= q.share * q.warps * blocks && resident_kernel_for<Real>(p.passes, advance_mode(s), q) != nullptr;
    if (!holds) return false;
    // staging levels in the memory of the second field copies, two halves
    p.levels = kResidentSteps;
    if (pc.nfreq > 0)
        p.levels = (int)std::min<size_t>(kResidentSteps, (4 * lay.field_elems - kPadLeft) / (4 * (size_t)pc.C));
    return p.levels >= 1;
}

// Cuts rows 1 .. ny-1 into slabs of about equal cost: the least cost of the
// dearest slab, by bisection over a greedy cut.  box: the candidate's materials.
template <typename Real>
static bool cut_slabs(const ProblemClass& pc, const ResidentPlan& p, const ResidentShape& shape, const int* box,
                      std::vector<double>& cost, int* ys, double& dearest) {
    const int most = shape.share * shape.warps, width = 32 * Quad<Real>::N;
    // Cost of a row in microseconds, fitted to the step times of 200^2, 333 x 251 and 400^2
    // grids cut in 8 to 30 ways each.  FP32 rows with materials cost up to 1.6 plain ones
    // (400^2: 2.98 us a step, against 3.6 with equal rows), y-CPML rows 1.8.  In FP64 the
    // arithmetic of the y-CPML rows and the staging of a face row count for more (200^2:
    // 14.1 us a step, against 21.2 cut with the FP32 weights).
    constexpr bool kWide = sizeof(Real) == 8;
    int mats = 0;
    for (int c = 0; c < p.passes; ++c)
        mats += box[0] < kEdge + (c + 1) * width && box[1] >= kEdge + c * width;
    const double plain = (kWide ? 0.27 : 0.022) * p.passes, strip = (kWide ? 2.0 : 1.8) * plain;
    const double mat = plain * (1.0 + (kWide ? 0.25 : 0.6) * mats / p.passes), face = kWide ? 6 * plain : 0;
    const int face0 = pc.nfreq > 0 ? pc.spec.nf2ff_d : -1, face1 = pc.nfreq > 0 ? pc.ny - pc.spec.nf2ff_d - 1 : -1;
    cost.assign(pc.ny, 0.0);
    double total = 0;
    for (int m = 1; m < pc.ny; ++m) {
        cost[m] = m <= pc.nc || m >= pc.ny - pc.nc ? strip : m >= box[2] && m <= box[3] ? mat : plain;
        if (m == face0 || m == face1) cost[m] += face;
        total += cost[m];
    }
    // a slab does not end at a horizontal NTFF face: its sample takes Ez of the row above
    auto cut = [&](double limit) {
        int m = 1;
        for (int b = 0; b < p.blocks; ++b) {
            ys[b] = m;
            const int left = p.blocks - 1 - b;
            double c = 0;
            int n = 0;
            while (m < pc.ny && pc.ny - m > 2 * left && n < most && (n < 2 || c + cost[m] <= limit)) {
                c += cost[m];
                ++m;
                ++n;
            }
            if ((m - 1 == face0 || m - 1 == face1) && left > 0) {
                if (n > 2) --m;
                else return false;
            }
        }
        ys[p.blocks] = pc.ny;
        return m == pc.ny;
    };
    double lo = 0, hi = 4 * total / p.blocks;
    if (!cut(hi)) return false;
    for (int i = 0; i < 12; ++i) {
        const double mid = 0.5 * (lo + hi);
        if (cut(mid)) hi = mid;
        else lo = mid;
    }
    if (!cut(hi)) return false;
    dearest = std::max(dearest, hi);
    for (int b = 0; b < p.blocks; ++b)
        if (ys[b + 1] - ys[b] < 2) return false;
    return true;
}

// A batch on one shape; false: it does not fit.
template <typename Real>
static bool batch_on(const ProblemClass& pc, const ResidentPlan& p, const ResidentShape& shape, const Unpacked& u,
                     ResidentBatch& b) {
    const bool ref = pc.spec.mode != TOMO_MODE_BREAST;
    const int nb = p.blocks + 1, d = pc.nfreq > 0 ? pc.spec.nf2ff_d : -1, none[4] = {1, 0, 1, 0};
    const size_t n = u.ncand + pc.extra;
    if (pc.ny - 1 > shape.share * shape.warps * p.blocks) return false;
    b.shape = shape;
    b.warps = 0;
    b.smem = 0;
    b.cost = 0;
    std::vector<double> cost;
    for (size_t c = 0; c < n; ++c) {
        const int* m = c < u.ncand ? &u.mbox[4 * c] : none;
        int* ys = &b.ys[c * nb];
        if (c > 0 && c < u.ncand && std::equal(m, m + 4, m - 4)) std::copy(ys - nb, ys, ys);
        else if (!cut_slabs<Real>(pc, p, shape, m, cost, ys, b.cost)) return false;
        int tall = 0;
        for (int k = 0; k < p.blocks; ++k) tall = std::max(tall, ys[k + 1] - ys[k]);
        b.warps = std::max(b.warps, resident_warps(tall, shape.share, pc.nrx));
        for (int k = 0; k < p.blocks; ++k)
            b.smem = std::max(b.smem, resident_layout<Real>(pc.nx, pc.ny, pc.nc, pc.nmat, ref, p.passes, shape.share, ys[k],
                                                            ys[k + 1], tall, m[0], m[1], m[2], m[3], d)
                                          .total);
    }
    b.smem = (b.smem + 4095) / 4096 * 4096;   // one captured launch serves batches of about the same boxes
    return b.smem <= kSmemPerBlock;
}

template <typename Real>
void resident_batch(const ProblemClass& pc, const ResidentPlan& p, const Unpacked& u, ResidentBatch& b) {
    b.fits = false;
    b.ys.resize((u.ncand + pc.extra) * (p.blocks + 1));
    for (const ResidentShape& q : kShapes) {
        if (!resident_kernel_for<Real>(p.passes, advance_mode(pc.spec), q)) continue;
        b.fits = batch_on<Real>(pc, p, q, u, b);
        if (b.fits) return;
    }
}

template <typename Real>
void make_resident(const ProblemClass& pc, const SolveLayout& lay, const ResidentPlan& p, const ResidentBatch& b,
                   const Unpacked& u, SolveDesc<Real>* descs, int nsolves) {
    for (int sv = 0; sv < nsolves; ++sv) {
        SolveDesc<Real>& D = descs[sv];
        Real* const f = D.ez[0];
        const size_t fe = lay.field_elems, cand = (size_t)(sv / pc.n_exc);
        D.resident = 1;
        D.ez[0] = D.ez[1] = f;
        D.hx[0] = D.hx[1] = f + fe;
        D.hy[0] = D.hy[1] = f + 2 * fe;
        D.jp[0] = D.jp[1] = f + 3 * fe;
        D.psi[1] = D.psi[0];
        D.stage = f + 4 * fe;
        D.mx0 = 1; D.mx1 = 0; D.my0 = 1; D.my1 = 0;
        if (cand < u.ncand) {
            const int* m = &u.mbox[4 * cand];
            D.mx0 = m[0]; D.mx1 = m[1]; D.my0 = m[2]; D.my1 = m[3];
        }
        const int* ys = &b.ys[std::min(cand, u.ncand + pc.extra - 1) * (p.blocks + 1)];
        std::copy(ys, ys + p.blocks + 1, D.ys);
    }
}

static cudaLaunchConfig_t cluster_config(const ResidentPlan& p, const ResidentBatch& b, int clusters, cudaStream_t st,
                                         cudaLaunchAttribute* attr) {
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(clusters * p.blocks);
    c.blockDim = dim3(32 * b.warps);
    c.dynamicSmemBytes = b.smem;
    c.stream = st;
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = p.blocks;
    attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
    c.attrs = attr;
    c.numAttrs = 1;
    return c;
}

template <typename Real>
int resident_clusters(const ResidentPlan& p, const ResidentBatch& b, int mode, int* clusters) {
    ResidentFn<Real> fn = resident_kernel_for<Real>(p.passes, mode, b.shape);
    if (!fn) return fail(TOMO_EINVAL, "no resident kernel for this grid");
    *clusters = 0;
    CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemPerBlock));
    CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchAttribute attr;
    cudaLaunchConfig_t c = cluster_config(p, b, 1, nullptr, &attr);
    if (cudaOccupancyMaxActiveClusters(clusters, fn, &c) != cudaSuccess) {
        cudaGetLastError();   // the answer to the question: no such cluster here
        *clusters = 0;
    }
    return TOMO_OK;
}

template <typename Real>
int resident_choice(const ProblemClass& pc, const SolveLayout& lay, const Unpacked& u, ResidentPlan& p,
                    ResidentBatch& b) {
    int best = -1;
    double least = 0;
    for (int blocks : kClusterSizes) {
        ResidentPlan q;
        if (!resident_plan<Real>(pc, lay, blocks, q)) continue;
        ResidentBatch c;
        resident_batch<Real>(pc, q, u, c);
        int clusters = 0;
        if (!c.fits || resident_clusters<Real>(q, c, advance_mode(pc.spec), &clusters)) continue;
        if (clusters < 1) continue;
        const double t = resident_estimate(c, (int)u.ncand * pc.n_exc, clusters);
        if (best < 0 || t < least) {
            best = blocks;
            least = t;
            p = q;
            b = c;
        }
    }
    return best;
}

template <typename Real>
int launch_resident(const ResidentPlan& p, const ResidentBatch& b, int mode, int clusters, const SolveDesc<Real>* descs,
                    int nsolves, int first, int count, int nsteps, int* error, cudaStream_t st,
                    cudaEvent_t placed) {
    ResidentFn<Real> fn = resident_kernel_for<Real>(p.passes, mode, b.shape);
    if (clusters < 1) return fail(TOMO_ECUDA, "a cluster of " + std::to_string(p.blocks) + " blocks does not fit the GPU");
    cudaLaunchAttribute attr[3];
    cudaLaunchConfig_t c = cluster_config(p, b, std::min(clusters, count), st, attr);
    // ahead of the DFT pass that runs beside it, whose blocks would hold up whole clusters
    attr[1].id = cudaLaunchAttributePriority;
    int least = 0;
    CUDA_TRY(cudaDeviceGetStreamPriorityRange(&least, &attr[1].val.priority));
    c.numAttrs = 2;
    if (placed) {
        attr[2].id = cudaLaunchAttributeLaunchCompletionEvent;
        attr[2].val.launchCompletionEvent.event = placed;
        attr[2].val.launchCompletionEvent.flags = 0;
        c.numAttrs = 3;
    }
    CUDA_TRY(cudaLaunchKernelEx(&c, fn, descs, nsolves, first, count, nsteps, error));
    return TOMO_OK;
}

#define TOMO_RESIDENT(Real)                                                                                            \
    template bool resident_plan<Real>(const ProblemClass&, const SolveLayout&, int, ResidentPlan&);                    \
    template void resident_batch<Real>(const ProblemClass&, const ResidentPlan&, const Unpacked&, ResidentBatch&);     \
    template void make_resident<Real>(const ProblemClass&, const SolveLayout&, const ResidentPlan&,                    \
                                      const ResidentBatch&, const Unpacked&, SolveDesc<Real>*, int);                   \
    template int resident_choice<Real>(const ProblemClass&, const SolveLayout&, const Unpacked&, ResidentPlan&,        \
                                       ResidentBatch&);                                                                \
    template int resident_clusters<Real>(const ResidentPlan&, const ResidentBatch&, int, int*);                        \
    template int launch_resident<Real>(const ResidentPlan&, const ResidentBatch&, int, int, const SolveDesc<Real>*,    \
                                       int, int, int, int, int*, cudaStream_t, cudaEvent_t);
TOMO_RESIDENT(float)
TOMO_RESIDENT(double)
#undef TOMO_RESIDENT

}  // namespace tomo
