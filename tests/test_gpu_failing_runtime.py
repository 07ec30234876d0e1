"""Failures of the resident kernel's launches and of its occupancy query, made on the host: a copy of the library is
linked against CUDA calls that fail on request (tests/failing_runtime).  No launch fails or
hangs on the GPU."""
from __future__ import annotations

import os
import subprocess

import numpy as np
import pytest

from helpers import small_breast_spec, small_params

pytestmark = pytest.mark.gpu

WRAPPED = ("cudaLaunchKernelExC", "cudaOccupancyMaxActiveClusters")
ECUDA = -5


@pytest.fixture(scope="module")
def failing(tomo, tmp_path_factory):
    """The package on the failing copy of the library."""
    from tomography_gb300 import build

    build.build()
    d = tmp_path_factory.mktemp("failing_runtime")
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "failing_runtime", "wraps.cu")
    obj, lib = str(d / "wraps.o"), str(d / "libfailing.so")
    subprocess.run([build.nvcc()] + build.ARCH + build.NVCC_FLAGS + ["-c", src, "-o", obj], check=True)
    objs = [os.path.join(build.OBJ_DIR, os.path.basename(s) + ".o") for s in build.SOURCES]
    wraps = [a for f in WRAPPED for a in ("-Xlinker", f"--wrap={f}")]
    subprocess.run([build.nvcc()] + build.ARCH + ["-shared", "-o", lib] + wraps + objs + [obj, "-lcudart"], check=True)
    kept = tomo.LIB_PATH, tomo._lib
    tomo.LIB_PATH, tomo._lib = lib, None
    try:
        yield tomo
    finally:
        tomo.LIB_PATH, tomo._lib = kept


def _solver(tomo, W, **kw):
    s = tomo.Solver(small_breast_spec(tomo, n_ellipses=4, steps=400, **kw))
    s.set_target(s.forward(small_params(W, 4), traces=True, far_field=False)["traces"][0])
    return s


def _cands(W, n, seed):
    return np.stack([W.candidate_params(seed + 1000 * i, 4, disc_radius=15e-3) for i in range(n)])


def _status(tomo, fn, *a):
    try:
        fn(*a)
    except tomo.TomoError as e:
        return e.status
    return 0


def test_batch(failing):
    from tomography_gb300 import workloads as W

    with _solver(failing, W) as s:
        a = _cands(W, 2, 5)
        want = s.fitness_batch(a)
        failing.library().failing_lose_row(1)
        assert _status(failing, s.fitness_batch, np.concatenate([a, a])) == ECUDA
        np.testing.assert_array_equal(s.fitness_batch(a), want)   # reported once


@pytest.mark.parametrize("launch", [1, 2, 4, 5, 7, 8])
def test_serving(failing, launch):
    """Two requests of 400 steps, four launches each, and the launch-th loses a row: its
    request fails, once, and returns its memory; the other's result is the batch's."""
    from tomography_gb300 import workloads as W

    with _solver(failing, W) as s:
        a, b = _cands(W, 2, 11), _cands(W, 1, 12)
        want = [s.fitness_batch(a), s.fitness_batch(b)]
        tickets = [s.submit(a), s.submit(b)]
        failing.library().failing_lose_row(launch)
        statuses, lost = [], (launch - 1) % 2
        for _ in range(20):
            statuses.append(_status(failing, s.serve_step))
        assert sorted(set(statuses)) == [ECUDA, 0] and statuses.count(ECUDA) == 1, statuses
        st = s.stats()
        assert st["serve_running"] == st["serve_queued"] == st["serve_bytes_in_use"] == 0, st
        for i, t in enumerate(tickets):
            if i == lost:
                assert _status(failing, s.poll, t, len(want[i])) == ECUDA
            else:
                np.testing.assert_array_equal(s.poll(t, len(want[i])), want[i])
        t = s.submit(a)                              # the slots and the words are free again
        np.testing.assert_array_equal(s.wait(t, 2, 60.0), want[0])


@pytest.mark.parametrize("error", [0, 1])
@pytest.mark.parametrize("most", [12, 5, 0])
def test_cluster_sizes_that_do_not_fit(failing, most, error):
    """Where the GPU has no room for a cluster size, a smaller one or the wavefront kernel
    serves the call, with the same bits, before and after a first choice."""
    from tomography_gb300 import workloads as W

    lib = failing.library()
    with _solver(failing, W) as s:
        a = _cands(W, 3, 21)
        want = s.fitness_batch(a)
        try:
            lib.failing_most_blocks(most, error)
            got = s.fitness_batch(a[:2])
            assert (s.stats()["min_blocks_per_sm"] == 1) == (most > 0)
            np.testing.assert_array_equal(got, want[:2])
            np.testing.assert_array_equal(s.fitness_batch(a), want)
            np.testing.assert_array_equal(s.wait(s.submit(a), 3, 60.0), want)
            with _solver(failing, W) as fresh:
                np.testing.assert_array_equal(fresh.fitness_batch(a), want)
        finally:
            lib.failing_most_blocks(1 << 30, 0)
        np.testing.assert_array_equal(s.fitness_batch(a), want)
