"""More receivers than a block of the resident kernel has threads: short wide grids, whose
slabs are one warp tall, against the wavefront kernel at one step per launch.  Every cell
evaluates the same explicitly rounded formulas, so no tolerance is involved."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_antennas", [32, 33, 64])
@pytest.mark.parametrize("nx,ny,d", [(500, 65, 5), (500, 65, None), (500, 49, 5), (420, 66, 5)])
def test_short_wide_grids(tomo, nx, ny, d, n_antennas):
    spec = tomo.breast_spec(0).copy(nx=nx, ny=ny, steps=90, ncpml=0, nf2ff_d=d or 5, nfreq=0 if d is None else 2,
                                    disc_radius=0.0, disc_del_eps=0.0, antenna_radius=11e-3, n_antennas=n_antennas,
                                    n_tx=2, n_angles=12, n_ellipses=1)
    cand = np.array([[0.0, 0.0, 1e-5, 1e-5, 0.0, 9.0, 0.0, 0.0]])   # between the cells' centres or one cell
    with tomo.Solver(spec) as s:
        got = s.forward(cand, traces=True, far_field=d is not None)["traces"]
        assert s.stats()["min_blocks_per_sm"] == 1   # the resident kernel ran
        s.set_target(np.ones(got.shape[1:], np.float32))
        served = s.wait(s.submit(cand), 1, 60.0)
    with tomo.Solver(spec.copy(steps_per_launch=1, cols_per_lane=1)) as s:
        want = s.forward(cand, traces=True, far_field=d is not None)["traces"]
        s.set_target(np.ones(got.shape[1:], np.float32))
        fitness = s.fitness_batch(cand)
    np.testing.assert_array_equal(got, want)
    np.testing.assert_array_equal(served, fitness)
    assert np.abs(want[:, :, -1]).max() > 0   # the last receiver, beside the first transmitter
