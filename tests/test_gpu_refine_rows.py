"""Refinement of contiguous systems in one kernel (csrc/refine_rows.cu) at the
edges of its shapes: lanes per system, rows a lane, warps a CTA, row counts off
the 16-byte grid, unread a[0] and c[n-1], the sweep counts around it and a
tolerance that the first solution meets.  Against the FP64 oracle: residual
1e-10 as for every refinement, forward error 1e-10 (the double-float residual
leaves some 1e-13, the systems' condition is below 10)."""
from __future__ import annotations

import numpy as np
import pytest

import tridiagonalsolvers_gb300 as tg
from oracle import gold
from tridiagonalsolvers_gb300 import workloads

pytestmark = pytest.mark.gpu


def _refine(cuda, arrs, n, m, **kw):
    import torch

    t = [torch.from_numpy(np.ascontiguousarray(v).ravel()).to(cuda) for v in arrs]
    x, sweeps, rel = tg.refine(*t, n, m, **kw)
    return x.cpu().numpy().reshape(m, n), sweeps, rel


@pytest.mark.parametrize("n", [1, 2, 3, 7, 16, 17, 33, 64, 65, 100, 129, 250, 333, 400, 544, 545, 640, 641, 897, 1000,
                               1153, 2176, 2177, 3000, 4352, 4353, 6001, 8704])
def test_every_shape(cuda, n):
    for m in (1, 6, max(1, (1 << 18) // n) | 1):
        arrs = workloads.dominant(m, n, seed=3 * n + m)
        x, sweeps, rel = _refine(cuda, arrs, n, m)
        res = gold.rel_residual(*arrs, x).max()
        x64 = gold.solve_f64(*arrs)
        assert sweeps <= 1 and res <= 1e-10 and rel <= 4 * res + 1e-13 and res <= 4 * rel + 1e-13
        assert np.abs(x - x64).max() <= 1e-10 * np.abs(x64).max()
        ends = [v.copy() for v in arrs]
        ends[0][:, 0] = np.nan
        ends[2][:, -1] = np.nan
        y, s2, _ = _refine(cuda, ends, n, m)
        assert s2 == sweeps and np.array_equal(x, y)
    assert tg.device_status() == 0


@pytest.mark.parametrize("n", [50, 300, 1500])
def test_sweep_counts(cuda, n):
    m = 9
    arrs = workloads.dominant(m, n, seed=n)
    # a tolerance the first solution meets: no correction
    x, sweeps, rel = _refine(cuda, arrs, n, m, tol=1e-5)
    assert sweeps == 0 and rel <= 1e-5
    # systems that FP32 solves exactly: residual zero before any correction
    one = [np.zeros_like(arrs[0]), np.full_like(arrs[0], 2.0), np.zeros_like(arrs[0]), arrs[3]]
    x, sweeps, rel = _refine(cuda, one, n, m)
    assert sweeps == 0 and rel == 0.0 and np.array_equal(x, one[3].astype(np.float64) / 2)
    # a zero right-hand side
    zero = [arrs[0], arrs[1], arrs[2], np.zeros_like(arrs[3])]
    x, sweeps, rel = _refine(cuda, zero, n, m)
    assert sweeps == 0 and rel == 0.0 and not x.any()
    for k in (1, 2, 3):
        with pytest.raises(tg.TridiError) as ei:
            _refine(cuda, arrs, n, m, tol=1e-30, max_sweeps=k)
        assert ei.value.status == 6


def test_nan_ends_the_refinement(cuda):
    n, m = 200, 12
    arrs = workloads.dominant(m, n, seed=4)
    arrs[3][5, 17] = np.nan
    with pytest.raises(tg.TridiError) as ei:
        _refine(cuda, arrs, n, m)
    assert ei.value.status == 6
