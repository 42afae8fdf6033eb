"""Interleaved systems that a CTA holds whole (csrc/columns.cuh): row counts at
the edges of its chunks (16 rows) and of its range (448 rows FP32, 224 FP64),
system counts around its 32, staged by tensor copies (FP32, a multiple of 32
systems) and by plain loads, and as the separator systems of longer ones,
against the FP64 oracle.  Tolerances: tests/parity.py."""
from __future__ import annotations

import numpy as np
import pytest

import tridiagonalsolvers_gb300 as tg
from oracle import gold
from tridiagonalsolvers_gb300 import workloads

from .parity import RES_TOL

pytestmark = pytest.mark.gpu

ROWS = [33, 34, 35, 36, 47, 48, 49, 52, 64, 65, 207, 208, 209, 223, 224, 225, 433, 447, 448, 449, 3601, 7167, 7169]


def _solve(cuda, arrs, n, m):
    import torch

    t = [torch.from_numpy(np.ascontiguousarray(v).ravel()).to(cuda) for v in arrs]
    return tg.solve_large(*t, n, m, layout="interleaved").cpu().numpy().reshape(n, m)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", ROWS)
def test_every_edge(cuda, n, dtype):
    for m in (1, 31, 32, 33, 96):
        # (what the solve may not look at: the first row's a, the last row's c)
        arrs = [v.astype(dtype) for v in workloads.weak(m, n, seed=n + m, layout=1)]
        want = _solve(cuda, arrs, n, m)
        assert gold.rel_residual(*arrs, want, layout=1).max() <= RES_TOL[dtype]
        arrs[0][0], arrs[2][-1] = np.nan, np.nan
        assert np.array_equal(_solve(cuda, arrs, n, m), want)
    assert tg.device_status() == 0


def test_plain_loads_and_tensor_copies_agree(cuda):
    """The two stagings hold the same rows: the same solution bit for bit."""
    from tridiagonalsolvers_gb300._lib import lib

    for n in (40, 300, 448):
        arrs = workloads.weak(64, n, seed=n, layout=1)
        x = _solve(cuda, arrs, n, 64)
        assert lib().tridi_set_tunable(6, 2) == 0
        try:
            assert np.array_equal(_solve(cuda, arrs, n, 64), x)
        finally:
            lib().tridi_set_tunable(6, 0)


def test_nan_system_apart(cuda):
    n, m = 300, 64
    arrs = workloads.weak(m, n, seed=4, layout=1)
    x = _solve(cuda, arrs, n, m)
    arrs = [v.copy() for v in arrs]
    arrs[3][7, 5] = np.nan
    y = _solve(cuda, arrs, n, m)
    keep = np.arange(m) != 5
    assert np.isnan(y[7, 5]) and np.array_equal(x[:, keep], y[:, keep])
