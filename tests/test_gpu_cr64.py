"""The FP64 CR / PCR / CR-PCR kernel (csrc/cr64.cu) at the edges of its
shapes: every size and switch level, batches of one system, a partly filled
CTA and more than one tile a CTA, pointers off the 16-byte grid, and a system
of NaN and infinities beside the others (their results must not change by a
bit).  Oracle: the gold Thomas solver in FP64, the tolerances of parity.py."""
from __future__ import annotations

import numpy as np
import pytest

import tridiagonalsolvers_gb300 as tg
from tridiagonalsolvers_gb300 import workloads

from .parity import check_against_oracle

pytestmark = pytest.mark.gpu


def _solve(cuda, arrs, n, rest, offset=0):
    import torch

    views = []
    for v in (*arrs, np.zeros_like(arrs[0])):
        buf = torch.zeros(v.size + offset, dtype=torch.float64, device=cuda)
        buf[offset:] = torch.from_numpy(np.ascontiguousarray(v).ravel())
        views.append(buf[offset:])
    if rest == 2:
        tg.cr(*views[:4], x=views[4], system_size=n)
    elif rest == n:
        tg.pcr(*views[:4], x=views[4], system_size=n)
    else:
        tg.crpcr(*views[:4], rest, x=views[4], system_size=n)
    return views[4].cpu().numpy().reshape(-1, n)


@pytest.mark.parametrize("n", [2, 4, 8, 16, 32, 64, 256, 512, 1024, 2048])
def test_every_size_and_switch_level(cuda, n):
    rests = [1 << k for k in range(1, n.bit_length())]
    for rest in rests:
        for m in (1, 3, 2 * 152 * 4 * max(1, 1024 // n) + 5 if rest in (2, n) and n >= 256 else 37):
            arrs = workloads.dominant(m, n, seed=n + rest + m, dtype=np.float64)
            x = _solve(cuda, arrs, n, rest)
            check_against_oracle(*arrs, x, dtype=np.float64)
    assert tg.device_status() == 0


@pytest.mark.parametrize("n,rest", [(4, 4), (16, 2), (64, 8), (64, 32), (1024, 2), (1024, 512), (2048, 1024)])
def test_misaligned_and_isolated(cuda, n, rest):
    m = 9
    arrs = workloads.dominant(m, n, seed=3 * n + rest, dtype=np.float64)
    x = _solve(cuda, arrs, n, rest)
    assert np.array_equal(x, _solve(cuda, arrs, n, rest, offset=1))
    bad = [v.copy() for v in arrs]
    bad[1][4] = np.nan
    bad[3][4, ::2] = np.inf
    bad[0][4, 0] = bad[2][4, -1] = np.inf
    y = _solve(cuda, bad, n, rest)
    keep = np.arange(m) != 4
    assert np.array_equal(x[keep], y[keep])
    # a[0] and c[n-1] are not part of a system, whatever they hold
    ends = [v.copy() for v in arrs]
    ends[0][:, 0] = np.nan
    ends[2][:, -1] = np.nan
    assert np.array_equal(x, _solve(cuda, ends, n, rest))


@pytest.mark.parametrize("n", [1, 2, 3, 7, 8, 9, 16, 17, 63, 257, 1000, 1025, 2047, 2049, 4096, 4097, 4607, 4608])
def test_any_size(cuda, n):
    """tg.solve in FP64: the same kernel on n rows, whatever n: the sizes
    around a thread's 8 rows, a CTA's and the largest, in batches of one
    system, an odd count and more tiles than CTAs; an odd pointer offset and a
    non-finite neighbour change no bit."""
    import torch

    for m in (1, 6, 2 * 152 * 5 + 7 if n in (1, 257, 1000) else 19):
        arrs = workloads.dominant(m, n, seed=7 * n + m, dtype=np.float64)
        t = [torch.from_numpy(v).to(cuda) for v in arrs]
        x = tg.solve(*t).cpu().numpy()
        check_against_oracle(*arrs, x, dtype=np.float64)
        off = []
        for v in arrs:
            buf = torch.zeros(v.size + 1, dtype=torch.float64, device=cuda)
            buf[1:] = torch.from_numpy(v.ravel())
            off.append(buf[1:].view(m, n))
        assert np.array_equal(x, tg.solve(*off).cpu().numpy())
        if m > 1:
            bad = [v.copy() for v in arrs]
            bad[1][m // 2] = np.nan
            bad[3][m // 2] = np.inf
            y = tg.solve(*(torch.from_numpy(v).to(cuda) for v in bad)).cpu().numpy()
            keep = np.arange(m) != m // 2
            assert np.array_equal(x[keep], y[keep])
    assert tg.device_status() == 0
