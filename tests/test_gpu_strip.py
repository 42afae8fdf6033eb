"""The FP32 any-size kernels (csrc/partition.cu on csrc/strip.cuh) and the
block passes of the contiguous large systems (csrc/large_rows.cu) where they
can go wrong: the smallest and largest of each shape (lanes per system, rows a
lane, warps a CTA), row counts off the 16-byte grid, a last tile that is not
full, pointers off the grid (no bulk copies), unread a[0] and c[n-1], and a
non-finite system beside the others.  Oracle: gold Thomas in FP64."""
from __future__ import annotations

import numpy as np
import pytest

import tridiagonalsolvers_gb300 as tg
from tridiagonalsolvers_gb300 import workloads

from .parity import check_against_oracle

pytestmark = pytest.mark.gpu


def _solve(cuda, arrs, n, offset=0):
    import torch

    views = []
    for v in (*arrs, np.zeros_like(arrs[0])):
        buf = torch.zeros(v.size + offset, dtype=torch.float32, device=cuda)
        buf[offset:] = torch.from_numpy(np.ascontiguousarray(v).ravel())
        views.append(buf[offset:])
    tg.solve(*views[:4], x=views[4], system_size=n)
    return views[4].cpu().numpy().reshape(-1, n)


@pytest.mark.parametrize("n", [1, 2, 3, 5, 16, 17, 31, 33, 64, 65, 100, 127, 129, 250, 256, 333, 500, 672, 673, 800,
                               991, 992, 993, 1153, 1664, 1665, 2176, 2177, 4352, 4353, 8703, 8704])
def test_any_size(cuda, n):
    for m in (1, 7, max(1, (1 << 19) // n) | 1):
        arrs = workloads.dominant(m, n, seed=11 * n + m)
        x = _solve(cuda, arrs, n)
        check_against_oracle(*arrs, x)
        assert np.array_equal(x, _solve(cuda, arrs, n, offset=1))  # plain loads, the same arithmetic
        other = [v.copy() for v in arrs]
        other[0][:, 0] = np.nan
        other[2][:, -1] = np.nan
        keep = np.arange(m) != m // 2
        if m > 1:
            other[1][m // 2] = np.nan
            other[3][m // 2] = np.inf
            y = _solve(cuda, other, n)
            assert np.array_equal(x[keep], y[keep])
        else:
            assert np.array_equal(x, _solve(cuda, other, n))
    assert tg.device_status() == 0


# one block and a row, whole blocks, a last block of one row; 2176 rows a
# block in FP32, 1664 in FP64; more than 32 blocks a system
@pytest.mark.parametrize("prec,n", [("f32", 8705), ("f32", 10880), ("f32", 10881), ("f32", 13055), ("f32", 69633),
                                    ("f32", 150001), ("f64", 4609), ("f64", 4992), ("f64", 4993), ("f64", 6655),
                                    ("f64", 54913)])
def test_large_contiguous(cuda, prec, n):
    import torch

    dt = np.float32 if prec == "f32" else np.float64
    tdt = torch.float32 if prec == "f32" else torch.float64
    for m in (1, 2, 5):
        arrs = workloads.dominant(m, n, seed=n + m, dtype=dt)

        def solve(arrs, offset=0):
            views = []
            for v in (*arrs, np.zeros_like(arrs[0])):
                buf = torch.zeros(v.size + offset, dtype=tdt, device=cuda)
                buf[offset:] = torch.from_numpy(np.ascontiguousarray(v).ravel())
                views.append(buf[offset:])
            tg.solve_large(*views[:4], n, m, x=views[4])
            return views[4].cpu().numpy().reshape(m, n)

        x = solve(arrs)
        check_against_oracle(*arrs, x, dtype=dt)
        assert np.array_equal(x, solve(arrs, offset=1))
        if m > 1:
            other = [v.copy() for v in arrs]
            other[0][:, 0] = np.nan
            other[2][:, -1] = np.nan
            other[1][m // 2] = np.nan
            keep = np.arange(m) != m // 2
            assert np.array_equal(x[keep], solve(other)[keep])
    assert tg.device_status() == 0
