"""The trace misfit's split FP32 sums against 64-bit sums (math.fsum of the
exact squares), at the edges of its chunks and of its 4-sample loads, for
unaligned buffers, quiet and extreme traces (where a chunk falls back to FP64),
and non-finite values.

Tolerance: a term keeps 47 bits and the sums' errors are carried along, so one
fitness is within 2^-44 (5.7e-14) of the exact quotient whatever the values; it
is typically below 3e-16.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _exact(traces, target):
    den = math.fsum((target.astype(np.float64).ravel() ** 2).tolist())   # squares of floats are exact in FP64
    out = []
    for tr in traces:
        d = tr.astype(np.float64) - target.astype(np.float64)
        # (s - t) is exact unless the exponents differ by more than 29 bits; its square is rounded once
        num = math.fsum((d.astype(np.longdouble) ** 2).astype(np.float64).ravel().tolist())
        out.append(-num / den if den > 0 else -num)
    return np.array(out)


def _misfit(tomo, traces, target, offset=0):
    import torch

    n, tx, m = traces.shape
    dev = torch.device("cuda", 0)
    buf = torch.zeros(traces.size + offset, dtype=torch.float32, device=dev)
    buf[offset:] = torch.from_numpy(np.ascontiguousarray(traces).ravel()).to(dev)
    tgt = torch.from_numpy(np.ascontiguousarray(target)).to(dev)
    fit = torch.full((n,), float("nan"), dtype=torch.float64, device=dev)
    lib = tomo.library()
    rc = lib.tomo_trace_misfit_static(C.c_void_p(buf.data_ptr() + 4 * offset), C.c_void_p(tgt.data_ptr()), n, tx, m,
                                      C.c_void_p(fit.data_ptr()), C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0, lib.tomo_last_error()
    torch.cuda.synchronize()
    return fit.cpu().numpy()


@pytest.mark.parametrize("m", [1, 3, 4, 1023, 8191, 8192, 8193, 16384 + 5])
@pytest.mark.parametrize("scale", [1.0, 1e-12, 1e-25, 1e12, 1e18])
def test_sums(tomo, m, scale):
    rng = np.random.default_rng(m)
    target = (scale * rng.standard_normal((3, m))).astype(np.float32)
    traces = (target + 0.1 * scale * rng.standard_normal((2, 3, m))).astype(np.float32)
    want = _exact(traces, target)
    got = _misfit(tomo, traces, target)
    np.testing.assert_allclose(got, want, rtol=2.0 ** -44, atol=0)
    for offset in (1, 2):   # unaligned traces: the same bits
        np.testing.assert_array_equal(_misfit(tomo, traces, target, offset), got)


def test_mixed_magnitudes_and_zeros(tomo):
    rng = np.random.default_rng(1)
    target = (10.0 ** rng.uniform(-30, 3, (2, 20000))).astype(np.float32)
    traces = np.stack([target, np.zeros_like(target), (target * rng.uniform(0.5, 1.5, target.shape)).astype(np.float32)])
    want = _exact(traces, target)
    got = _misfit(tomo, traces, target)
    assert got[0] == 0
    np.testing.assert_allclose(got, want, rtol=2.0 ** -44, atol=0)
    assert np.all(_misfit(tomo, traces * np.float32(0), target * np.float32(0)) == 0)


def test_non_finite(tomo):
    target = np.ones((1, 9000), dtype=np.float32)
    traces = np.ones((3, 1, 9000), dtype=np.float32)
    traces[1, 0, 8500] = np.inf
    traces[2, 0, 3] = np.nan
    got = _misfit(tomo, traces, target)
    assert got[0] == 0 and got[1] == -np.inf and np.isnan(got[2])
