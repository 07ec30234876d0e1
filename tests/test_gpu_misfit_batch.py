"""The trace misfit of a candidate does not depend on its place in the batch, and at
ordinary magnitudes it is as exact as FP64 sums.

Tolerance of the latter: the split sums themselves keep more than 64 bits, so what rounds
is FP64: two roundings as a chunk's three parts join, two as three chunks are added, two as
three transmitters are, for num and for den, and the quotient; and in the reference, one
for the squares, one for the sum, for both, and the quotient: 18 roundings of 2^-53.
"""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_misfit import _exact, _misfit

pytestmark = pytest.mark.gpu

CHUNK = 8192


@pytest.mark.parametrize("m", [1, 1023, CHUNK, CHUNK + 1, 2 * CHUNK + 5])
@pytest.mark.parametrize("scale", [1.0, 1e-6, 1e6])
def test_ordinary_magnitudes(tomo, m, scale):
    rng = np.random.default_rng(m + 1)
    target = (scale * rng.standard_normal((3, m))).astype(np.float32)
    traces = (target + 0.1 * scale * rng.standard_normal((4, 3, m))).astype(np.float32)
    np.testing.assert_allclose(_misfit(tomo, traces, target), _exact(traces, target), rtol=18 * 2.0 ** -53, atol=0)


@pytest.mark.parametrize("quiet", ["zero", "faint", "loud", "match"])
def test_places_in_the_batch(tomo, quiet):
    """A chunk of the target whose own sum is done in FP64, and one that the first
    candidate matches: the others' bits stay those of every other place."""
    rng = np.random.default_rng(3)
    target = rng.standard_normal((2, 2 * CHUNK + 100)).astype(np.float32)
    traces = (target + 0.1 * rng.standard_normal((3,) + target.shape)).astype(np.float32)
    part = slice(CHUNK, 2 * CHUNK)
    if quiet == "match":
        traces[0, :, part] = target[:, part]
    else:
        target[:, part] *= {"zero": 0.0, "faint": 1e-25, "loud": 1e18}[quiet]
        traces[:, :, part] = (0.1 * rng.standard_normal(traces[:, :, part].shape)).astype(np.float32)
    got = {}
    for order in ([0, 1, 2], [1, 2, 0], [2, 0, 1]):
        for c, fit in zip(order, _misfit(tomo, traces[order], target)):
            assert got.setdefault(c, fit) == fit, (quiet, c, order)
    for c in range(3):
        assert _misfit(tomo, traces[c:c + 1], target)[0] == got[c]


@pytest.mark.parametrize("chunks,more", [(65535, 0), (65535, 1), (65536, 0), (65536, 1)])
def test_longest_solves(tomo, chunks, more):
    """Around the most chunks that one solve spreads over a grid: sums that are exact."""
    import ctypes as C

    import torch

    m = chunks * CHUNK + more
    target = torch.ones(m, dtype=torch.float32, device="cuda")
    traces = torch.full((m,), 1.5, dtype=torch.float32, device="cuda")
    fit = torch.full((1,), float("nan"), dtype=torch.float64, device="cuda")
    lib = tomo.library()
    rc = lib.tomo_trace_misfit_static(C.c_void_p(traces.data_ptr()), C.c_void_p(target.data_ptr()), 1, 1, m,
                                      C.c_void_p(fit.data_ptr()), C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0, lib.tomo_last_error()
    assert fit.item() == -0.25
