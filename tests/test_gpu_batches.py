"""Batches on the resident kernel whose solves do not divide by the clusters that run at
once (launches go round the solves, the DFT of a launch runs beside the next one), the
kernel's shapes by the rows of a grid, and the wavefront sweep's background block: the
same bits as the wavefront kernel at one step and one column per launch and lane.  Every
cell evaluates the same explicitly rounded formulas, so no tolerance is involved.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _spec(tomo, nx, ny, **kw):
    base = dict(nx=nx, ny=ny, steps=121, ncpml=10, nf2ff_d=13, disc_radius=8e-3, antenna_radius=11e-3, n_antennas=5,
                n_tx=2, n_angles=12, n_ellipses=1)
    base.update(kw)
    return tomo.breast_spec(0).copy(**base)


def _cands(n):
    """n candidates with one ellipse each, of different places, sizes and materials."""
    i = np.arange(n)
    return np.stack([2e-3 - 4e-4 * i, -1e-3 + 3e-4 * i, 3e-3 + 2e-4 * i, 5e-3 - 1e-4 * i, 0.4 + 0.1 * i, 12.0 + i, 20.0 - 0.4 * i,
                     0.3 + 0.01 * i], axis=1)


def _run(tomo, spec, cands, resident=None):
    with tomo.Solver(spec) as s:
        out = s.forward(cands, traces=True, traces_f64=True, far_field=True)
        out.update({f: s.field_snapshot(len(cands) - 1, s.n_exc - 1, f) for f in ("ez", "hx", "hy")})
        if resident is not None:
            assert (s.stats()["min_blocks_per_sm"] == 1) == resident, s.stats()
    return out


def _same(tomo, spec, other, cands, resident=None):
    got, want = _run(tomo, spec, cands, resident), _run(tomo, other, cands)
    for k in want:
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)
    assert np.abs(want["ez"]).max() > 0


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("ncand,n_tx", [(1, 5), (3, 5), (4, 4), (5, 5), (11, 5), (38, 1)])
def test_solves_per_launch(tomo, ncand, n_tx, precision):
    spec = _spec(tomo, 96, 90, n_tx=n_tx, precision=tomo.FP64 if precision == 64 else tomo.FP32)
    _same(tomo, spec, spec.copy(steps_per_launch=1, cols_per_lane=1), _cands(ncand), resident=True)


@pytest.mark.parametrize("nx,ny", [(70, 513), (70, 700), (200, 385), (300, 384), (300, 385), (300, 386), (300, 510),
                                   (490, 140), (490, 420)])
def test_rows_of_the_shapes(tomo, nx, ny):
    spec = _spec(tomo, nx, ny, steps=60, n_tx=1)
    _same(tomo, spec, spec.copy(steps_per_launch=1, cols_per_lane=1), _cands(2))


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("T,cols", [(3, 1), (3, 2), (4, 1), (4, 2), (6, 1), (8, 1)])
@pytest.mark.parametrize("shape", ["centre", "corner", "band", "point"])
def test_background_block(tomo, T, cols, shape, precision):
    disc, el = {"centre": (8e-3, [2e-3, -1e-3, 4e-3, 6e-3]), "corner": (0.0, [-2e-2, 1.5e-2, 9e-3, 7e-3]),
                "band": (0.0, [0.0, 2e-3, 9e-2, 3e-3]), "point": (0.0, [1e-3, 1e-3, 2e-4, 2e-4])}[shape]
    spec = _spec(tomo, 257, 203, n_tx=1, disc_radius=disc, precision=tomo.FP64 if precision == 64 else tomo.FP32)
    cand = np.array([el + [0.4, 12.0, 20.0, 0.3]])
    try:
        other = spec.copy(steps_per_launch=T, cols_per_lane=cols)
        with tomo.Solver(other):
            pass
    except Exception as e:
        if "unsupported" not in str(e):
            raise
        pytest.skip("not a compiled blocking")
    _same(tomo, other, spec.copy(steps_per_launch=1, cols_per_lane=1), cand)
