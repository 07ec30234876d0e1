"""The serving loop neither queues the resident kernel's requests behind each other nor
lets those of the wavefront kernel fall far behind them."""
from __future__ import annotations

import time

import numpy as np
import pytest

from helpers import small_breast_spec

pytestmark = pytest.mark.gpu


def _cands(W, n, seed):
    return np.stack([W.candidate_params(seed + 1000 * i, 4, disc_radius=15e-3) for i in range(n)])


def _target(spec):
    return np.ones((spec.n_tx, spec.n_antennas, spec.steps), np.float32)


def test_requests_of_both_kernels_advance_together(tomo):
    """Requests of 400 steps on the same grid; the one with 16 CPML cells streams.  A
    serving step takes the resident ones by 128 steps, the others by a third of it here."""
    from tomography_gb300 import workloads as W

    small = small_breast_spec(tomo, n_ellipses=4, steps=400)
    wide = small.copy(ncpml=16, nf2ff_d=18)
    a = _cands(W, 2, 5)
    with tomo.Solver(wide) as s:
        s.set_target(_target(wide))
        want = s.fitness_batch(a)
        assert s.stats()["min_blocks_per_sm"] > 1     # the wavefront kernel ran
    with tomo.Solver(small) as s:
        s.set_target(_target(small))
        s.set_target_for(wide, _target(wide))
        want_small = s.fitness_batch(a)
        t = s.submit(a, spec=wide)
        flow, got, steps = [s.submit(a) for _ in range(3)], None, 0
        while got is None:
            s.serve_step()
            steps += 1
            assert steps < 100
            got = s.poll(t, 2)
            for i, f in enumerate(flow):              # a steady flow of small requests
                r = s.poll(f, 2)
                if r is not None:
                    np.testing.assert_array_equal(r, want_small)
                    flow[i] = s.submit(a)
        np.testing.assert_array_equal(got, want)
        assert steps <= 16, steps                     # 400 / 42 is about 10; 50 with 8 steps each


def test_requests_share_the_gpu(tomo):
    """Sixteen requests of one solve take a cluster each, seven of which run at once: well
    below the sum of their times."""
    from tomography_gb300 import workloads as W

    spec = tomo.breast_spec(0).copy(n_tx=1)
    K = spec.n_ellipses
    c = np.stack([W.candidate_params(7 + 1000 * i, K, disc_radius=15e-3) for i in range(16)])
    with tomo.Solver(spec) as s:
        s.set_target(_target(spec))
        want = s.fitness_batch(c)

        def run(n):
            t0 = time.perf_counter()
            tickets = [s.submit(c[i:i + 1]) for i in range(n)]
            while s.serve_step():
                pass
            t1 = time.perf_counter()
            np.testing.assert_array_equal(np.concatenate([s.poll(t, 1) for t in tickets]), want[:n])
            return t1 - t0

        one, all_ = (min(run(n) for _ in range(3)) for n in (1, 16))
        assert all_ < 8 * one, (one, all_)
