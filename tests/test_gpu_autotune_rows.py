"""The rows-per-thread tuner times the kernels whose shape it chooses (the
hybrid kernels), also at the sizes where aligned arrays run a register kernel:
its time is that of cr by the hybrid kernel in the chosen shape, and it chooses
among the shapes that exist."""
from __future__ import annotations

import pytest

import tridiagonalsolvers_gb300 as tg
from tridiagonalsolvers_gb300 import _lib, autotune

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,shapes", [(256, (8, 16)), (1024, (8, 16)), (2048, (8, 16)), (4096, (16,))])
def test_times_the_hybrid_kernel(cuda, n, shapes):
    import torch

    L = _lib.lib()
    autotune.reset()
    try:
        rows, ms = autotune.tune("cr_rows", n, sample_unknowns=1 << 24)
        assert rows in shapes
        a, c, d = (torch.rand(((1 << 24) // n, n), device=cuda) - 0.5 for _ in range(3))
        b = a.abs() + c.abs() + 1
        assert L.tridi_set_tunable(10, 2) == 0  # TRIDI_TUNE_PCR_KERNEL: the hybrid kernels
        best = float("inf")
        for _ in range(12):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            tg.cr(a, b, c, d)
            e1.record()
            torch.cuda.synchronize()
            best = min(best, e0.elapsed_time(e1))
        assert 0.75 * best <= ms <= 1.33 * best
    finally:
        L.tridi_set_tunable(10, 0)
        autotune.reset()
