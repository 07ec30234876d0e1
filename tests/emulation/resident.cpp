// Runs the resident kernel's source on host threads:
// resident <nx> <ny> <ncpml> <blocks> <steps> <receivers> <what>, with <what>
//   late    copies into block 0 come 0.1 s after they were issued; two solves in turn
//   lost    the second row sent to block 1 never comes
//   slow    it comes after the receiver's limit
//   ends    nothing of the kind: the traces end in the final field
// "late" has to give each solve's bits of a launch of its own; with "lost" and "slow" the
// launch has to end with its error word set.  Never may a copy touch a block that has ended.
#include "fdtd_resident.cuh"

#include <cstdlib>
#include <string>

using namespace tomo;
using Real = float;
constexpr int kPasses = 1, kShare = SHARE, kWarps = SHARE == 2 ? 16 : 12;

struct Solve {
    SolveDesc<Real> d{};
    std::vector<Real> fields, psi, traces, stage, mtab, cpml, wave;
    std::vector<uint8_t> mat;
    std::vector<int> rx;
};

// Random fields in a background of one material; the receivers lie in every row.
static void make(Solve& s, int nx, int ny, int nc, int blocks, int steps, int nrx, unsigned seed) {
    SolveDesc<Real>& d = s.d;
    const int pitch = (kPadLeft + nx + 1 + kPadRight + 31) / 32 * 32;
    const size_t elems = (size_t)(ny + 1) * pitch + kPadLeft;
    auto rnd = [&] { return (Real)((seed = seed * 1664525u + 1013904223u) >> 8) / (1 << 24) - Real(0.5); };
    d.nx = nx; d.ny = ny; d.pitch = d.mpitch = pitch; d.ncpml = nc;
    d.step = 1; d.steps_total = steps + 1;
    d.active = d.resident = d.nmat = 1; d.nrx = nrx;
    d.flags = kPointSource; d.src_x = nx / 2; d.src_y = ny / 2;
    d.mx0 = d.my0 = 1;
    d.chez = Real(0.4); d.Kp = Real(0.9); d.dx = Real(0.5);
    s.fields.assign(4 * elems, 0);
    Real* const f = s.fields.data() + kPadLeft;
    d.ez[0] = f; d.hx[0] = f + elems; d.hy[0] = f + 2 * elems; d.jp[0] = f + 3 * elems;
    for (int y = 1; y < ny; ++y)
        for (int x = 1; x < nx; ++x) f[x + (size_t)y * pitch] = rnd();
    s.psi.assign((size_t)4 * nc * (ny + 1 + nx + 1), 0);
    s.traces.assign((size_t)nrx * (steps + 1), 0);
    s.stage.assign(4, 0);
    s.mat.assign((size_t)(ny + 1) * pitch + kMatPadLeft, 0);
    s.mtab = {Real(0.98), Real(0.47), 0, 0, 0, 0, Real(-0.7), 0};
    for (int q = 0; q < 6; ++q)
        for (int i = 0; i < nc; ++i)
            s.cpml.push_back(q % 3 == 0 ? 1 / (1 + Real(0.1) * i) : q % 3 == 1 ? Real(0.9) - Real(0.01) * i : Real(-0.05));
    for (int n = 0; n <= steps; ++n) s.wave.push_back(rnd());
    for (int r = 0; r < nrx; ++r) {
        s.rx.push_back(2 + 7 * r % (nx - 4));
        s.rx.push_back(1 + r % (ny - 1));
    }
    d.psi[0] = s.psi.data(); d.traces = s.traces.data(); d.stage = s.stage.data(); d.mat = s.mat.data() + kMatPadLeft;
    d.mtab = s.mtab.data(); d.cpml = s.cpml.data(); d.src_wave = s.wave.data(); d.rx = s.rx.data();
    for (int b = 0; b <= blocks; ++b) d.ys[b] = 1 + (ny - 1) * b / blocks;
}

// One launch over the listed solves; returns the kernel's error word.
static int launch(std::vector<SolveDesc<Real>> descs, int blocks, std::function<double(int, int)> delay, int* faults) {
    const SolveDesc<Real>& d = descs[0];
    int tall = 0, error = 0;
    for (int b = 0; b < blocks; ++b) tall = std::max(tall, d.ys[b + 1] - d.ys[b]);
    const int threads = 32 * resident_warps(tall, kShare, d.nrx);
    HostCluster c;
    cluster = &c;
    c.blocks.resize(blocks);
    c.running.assign(blocks, threads);
    c.received.assign(blocks, 0);
    c.delay = std::move(delay);
    c.meet = std::make_unique<std::barrier<>>(blocks * threads);
    blockDim = {threads, 1, 1};
    gridDim = {blocks, 1, 1};
    for (int b = 0; b < blocks; ++b) {
        const ResidentLayout l = resident_layout<Real>(d.nx, d.ny, d.ncpml, d.nmat, false, kPasses, kShare, d.ys[b],
                                                       d.ys[b + 1], tall, d.mx0, d.mx1, d.my0, d.my1, -1);
        HostBlock& h = c.blocks[b];
        h.memory.assign(l.total + 16, 0xff);
        h.smem = (unsigned char*)(((uintptr_t)h.memory.data() + 15) / 16 * 16);
        h.meet = std::make_unique<std::barrier<>>(threads);
        h.warps = std::vector<HostWarp>(threads / 32);
    }
    std::vector<std::thread> pool;
    for (int b = 0; b < blocks; ++b)
        for (int t = 0; t < threads; ++t)
            pool.emplace_back([&, b, t] {
                threadIdx = {t, 0, 0};
                blockIdx = {b, 0, 0};
                this_block = &c.blocks[b];
                this_warp = &this_block->warps[t / 32];
                fdtd_resident_kernel<Real, kPasses, kModeBreast, kShare, kWarps>(descs.data(), (int)descs.size(), 0,
                                                                                 (int)descs.size(), 1 << 20, &error);
                std::lock_guard<std::mutex> g(c.lock);
                if (--c.running[b] == 0) std::fill(c.blocks[b].memory.begin(), c.blocks[b].memory.end(), 0xff);
            });
    for (std::thread& t : pool) t.join();
    if (!c.copies.empty()) c.fault("a copy still on its way when the launch ended");
    *faults += c.faults;
    return error;
}

int main(int argc, char** argv) {
    if (argc < 8) return 2;
    const int nx = std::atoi(argv[1]), ny = std::atoi(argv[2]), nc = std::atoi(argv[3]), blocks = std::atoi(argv[4]),
              steps = std::atoi(argv[5]), nrx = std::atoi(argv[6]);
    const std::string what = argv[7];
    int faults = 0, bad = 0;
    Solve got[2], want[2];
    std::vector<SolveDesc<Real>> both;
    for (int i = 0; i < 2; ++i) {
        make(got[i], nx, ny, nc, blocks, steps, nrx, 7 + i);
        make(want[i], nx, ny, nc, blocks, steps, nrx, 7 + i);
        both.push_back(got[i].d);
        bad += launch({want[i].d}, blocks, nullptr, &faults) != 0;
    }
    auto delay = [&](int to, int index) {
        if (what == "ends") return 0.0;
        if (what == "late") return to == 0 ? 0.1 : 0.0;
        return to == 1 && index == 1 ? (what == "lost" ? -1.0 : 2.6) : 0.0;
    };
    const int error = launch(both, blocks, delay, &faults);
    if (what == "ends") {
        for (int r = 0; r < nrx; ++r) {
            const int x = got[0].rx[2 * r], y = got[0].rx[2 * r + 1];
            bad += got[0].traces[(size_t)r * (steps + 1) + steps] != got[0].d.ez[0][x + (size_t)y * got[0].d.pitch];
        }
    } else if (what == "late") {
        bad += error != 0;
        for (int i = 0; i < 2; ++i) {
            bad += std::memcmp(got[i].fields.data(), want[i].fields.data(), sizeof(Real) * got[i].fields.size()) != 0;
            bad += std::memcmp(got[i].psi.data(), want[i].psi.data(), sizeof(Real) * got[i].psi.size()) != 0;
            bad += std::memcmp(got[i].traces.data(), want[i].traces.data(), sizeof(Real) * got[i].traces.size()) != 0;
        }
    } else {
        bad += error == 0;
    }
    std::printf("%s: error word %d, %d wrong, %d faults\n", what.c_str(), error, bad, faults);
    return bad || faults;
}
