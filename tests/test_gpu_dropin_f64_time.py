"""The FP64 host-pointer cr on host arrays solved in place keeps the host link's
rate: it moves the bytes that crpcr moves, and takes no more than 1.25 times as
long (with eight rows a thread it took 1.6 to 1.8 times as long)."""
from __future__ import annotations

import time

import numpy as np
import pytest

from tridiagonalsolvers_gb300 import dropin, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [64, 256, 1024])
def test_cr_in_place_against_crpcr(cuda, n):
    import torch

    m = (1 << 22) // n
    pin = [torch.from_numpy(v.ravel()).pin_memory().numpy() for v in workloads.dominant(m, n, seed=n, dtype=np.float64)]
    x, y = (torch.zeros(n * m, dtype=torch.float64).pin_memory().numpy() for _ in range(2))

    def best(f):
        t = []
        for _ in range(8):
            s = time.perf_counter()
            f()
            t.append(time.perf_counter() - s)
        return min(t)

    cr = best(lambda: dropin.cr(*pin, x, n, m))
    crpcr = best(lambda: dropin.crpcr(*pin, y, n, m, n // 4))
    assert np.abs(x - y).max() <= 1e-13 * np.abs(y).max()
    assert cr <= 1.25 * crpcr
