"""Far field of grids whose vertical NTFF faces fall on the last column of a strip of the
advance kernel, were the strips all of one width: the bits of the plain path, which has no
strips, at every blocking."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("T,nx,d", [(1, 195, 15), (1, 66, 6), (2, 140, 27), (2, 121, 9), (4, 140, 23), (6, 140, 19), (8, 140, 15)])
def test_faces_at_strip_ends(tomo, T, nx, d, precision):
    spec = tomo.breast_spec(0).copy(nx=nx, ny=88, steps=200, ncpml=5, nf2ff_d=d, nfreq=2, n_angles=24, disc_radius=4e-3,
                                    antenna_radius=3e-3, n_antennas=3, n_tx=2, n_ellipses=1,
                                    precision=tomo.FP64 if precision == 64 else tomo.FP32)
    cand = np.array([[1e-3, -1e-3, 2e-3, 3e-3, 0.4, 12.0, 20.0, 0.3]])

    def run(**kw):
        with tomo.Solver(spec.copy(**kw)) as s:
            return s.forward(cand, traces=True, far_field=True)

    try:
        got = run(steps_per_launch=T, cols_per_lane=1)
    except tomo.TomoError as e:
        if "unsupported" not in str(e):
            raise
        pytest.skip("not a compiled blocking")
    want = run(plain=1)
    for k in ("traces", "D", "P"):
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)
