"""Rounding of the FP64 any-size solve (csrc/cr64.cu): no further from the
exact solution than the partition method was, whose root-mean-square relative
error on strictly dominant systems was 1.18e-16 at its best sizes (350 to 480
rows) and 1.19e-16 to 1.9e-16 elsewhere.  120000 unknowns give the figure to
about 1 %."""
from __future__ import annotations

import numpy as np
import pytest

import tridiagonalsolvers_gb300 as tg
from tridiagonalsolvers_gb300 import workloads

pytestmark = pytest.mark.gpu


def _exact(a, b, c, d):
    """Thomas in extended precision, all systems at once."""
    a, b, c, d = (np.ascontiguousarray(v.T).astype(np.longdouble) for v in (a, b, c, d))
    n = a.shape[0]
    cp, dp = c / b, d / b
    for i in range(1, n):
        den = b[i] - a[i] * cp[i - 1]
        cp[i] = c[i] / den
        dp[i] = (d[i] - a[i] * dp[i - 1]) / den
    for i in range(n - 2, -1, -1):
        dp[i] -= cp[i] * dp[i + 1]
    return dp.T


@pytest.mark.parametrize("n", [33, 64, 250, 300, 388, 480, 777, 1500, 4000, 4608])
def test_error_of_the_any_size_solve(cuda, n):
    import torch

    assert np.finfo(np.longdouble).eps < 1e-18
    arrs = workloads.dominant(max(1, 120000 // n), n, seed=n, dtype=np.float64)
    x = tg.solve(*(torch.from_numpy(v).to(cuda) for v in arrs)).cpu().numpy()
    exact = _exact(*arrs)
    err = np.sqrt(((x - exact) ** 2).sum() / (exact**2).sum())
    assert err <= 1.19e-16
