"""The resident kernel (one solve per thread-block cluster, fields on the chip)
against the wavefront kernel at one step per launch: the same bits in receiver
traces, far field and final fields, at the sizes where its cut of the grid
changes -- the last column of a number of inner passes and the first of the
next, inner widths that are not whole lanes, slabs of few rows, launches that do
not divide the steps -- and for materials, sources and strips in every part of
the grid.  Every cell evaluates the same explicitly rounded formulas, so no
tolerance is involved.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("ez", "hx", "hy")


def _run(tomo, spec, cands, resident):
    if not resident:
        spec = spec.copy(steps_per_launch=1, cols_per_lane=1)
    with tomo.Solver(spec) as s:
        breast = spec.mode == tomo.MODE_BREAST
        out = s.forward(cands, traces=breast, traces_f64=breast, far_field=spec.nfreq > 0)
        last = len(cands) - 1, s.n_exc - 1
        out.update({f: s.field_snapshot(*last, f) for f in FIELDS})
        st = s.stats()
    if resident:
        assert st["min_blocks_per_sm"] == 1, st   # the resident kernel ran
    return out


def _same(tomo, spec, cands):
    cands = np.atleast_2d(cands)
    got, want = (_run(tomo, spec, cands, r) for r in (True, False))
    assert set(got) == set(want)
    for k in want:
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)
    assert np.abs(want["ez"]).max() > 0


def _ellipse(cx, cy, a, b, eps=12.0, deps=20.0, sig=0.3):
    return [cx, cy, a, b, 0.4, eps, deps, sig]


def _spec(tomo, nx, ny, **kw):
    base = dict(nx=nx, ny=ny, steps=121, ncpml=10, nf2ff_d=13, disc_radius=8e-3, antenna_radius=11e-3, n_antennas=5,
                n_tx=2, n_angles=12, n_ellipses=1)
    base.update(kw)
    return tomo.breast_spec(0).copy(**base)


@pytest.mark.parametrize("nx,ny", [(65, 65), (96, 131), (158, 97), (159, 96), (160, 96), (161, 95), (203, 64), (286, 90),
                                   (287, 128), (288, 77), (333, 251), (414, 129), (415, 66)])
def test_grid_cuts(tomo, nx, ny):
    _same(tomo, _spec(tomo, nx, ny), np.array(_ellipse(2e-3, -1e-3, 4e-3, 6e-3)))


@pytest.mark.parametrize("nx,ny", [(65, 70), (94, 64), (95, 66), (96, 65), (159, 80), (160, 80), (222, 70)])
def test_grid_cuts_fp64(tomo, nx, ny):
    _same(tomo, _spec(tomo, nx, ny, precision=tomo.FP64, steps=67), np.array(_ellipse(2e-3, -1e-3, 4e-3, 6e-3)))


@pytest.mark.parametrize("kw", [dict(ncpml=0, nf2ff_d=4), dict(ncpml=0, nfreq=0), dict(ncpml=1, nf2ff_d=1),
                                dict(ncpml=12, nf2ff_d=12), dict(nfreq=0), dict(steps=1), dict(steps=2),
                                dict(nf2ff_d=40), dict(disc_radius=0.0, disc_del_eps=0.0), dict(src_amp=3.0)])
def test_options(tomo, kw):
    _same(tomo, _spec(tomo, 140, 99, **kw), np.array(_ellipse(0.0, 3e-3, 4e-3, 3e-3)))


def test_materials_everywhere(tomo):
    """Candidates of one batch whose materials cover the inner columns, an edge,
    the y-CPML rows, the antennas, the whole grid, and no cell but the disc's."""
    spec = _spec(tomo, 200, 150, n_ellipses=2, antenna_radius=30e-3, n_antennas=8, n_tx=3, steps=90)
    far = _ellipse(0.0, 0.0, 1e-5, 1e-5)
    cands = [_ellipse(0, 0, 20e-3, 10e-3) + far, _ellipse(-48e-3, 0, 6e-3, 9e-3) + far,
             _ellipse(49e-3, 5e-3, 4e-3, 20e-3) + far, _ellipse(0, 36e-3, 9e-3, 5e-3) + far,
             _ellipse(30e-3, 0, 3e-3, 3e-3) + _ellipse(-48e-3, -36e-3, 7e-3, 7e-3),
             _ellipse(0, 0, 80e-3, 80e-3, 9.0, 5.0, 0.1) + far, far + far]
    _same(tomo, spec, np.array(cands))


def test_more_solves_than_clusters(tomo):
    """A cluster takes several solves in turn, and a launch boundary falls inside the run."""
    from tomography_gb300 import workloads as W

    spec = _spec(tomo, 129, 129, n_tx=5, steps=700, n_ellipses=3)
    cands = np.stack([W.candidate_params(5 + 1000 * k, 3, 8e-3) for k in range(9)])
    _same(tomo, spec, cands)


@pytest.mark.parametrize("cpu", [False, True])
def test_reference_modes(tomo, cpu):
    from tomography_gb300 import workloads as W

    spec = tomo.reference_spec(cpu).copy(steps=330)
    _same(tomo, spec, np.stack([W.reference_patch_args(7 + k, cpu) for k in range(2)]))


def test_total_field(tomo):
    from tomography_gb300 import workloads as W

    _same(tomo, tomo.reference_spec(False).copy(steps=200, total_field=1), W.reference_patch_args(3))
