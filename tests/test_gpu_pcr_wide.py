"""PCR and PCR-then-Thomas across the warps of a CTA (csrc/pcr_wide.cu: FP32,
2048 and 4096 unknowns) and the register PCR-then-Thomas at 32 unknowns, every
split, batches of one system, a few and more than the GPU holds at once:
against the FP64 oracle and, as the 1024-unknown kernels are, within 16 ulp of
the shared-memory kernels (TRIDI_TUNE_PCR_KERNEL = 2)."""
from __future__ import annotations

import numpy as np
import pytest

import tridiagonalsolvers_gb300 as tg
from tridiagonalsolvers_gb300 import workloads

from .parity import check_against_oracle, check_ulps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [32, 2048, 4096])
def test_every_split(cuda, n):
    import torch

    from tridiagonalsolvers_gb300._lib import lib

    L = lib()
    for m in (1, 3, 17, 2 * 152 * 4 + 1 if n > 32 else 5001):
        arrs = workloads.dominant(m, n, seed=n + m)
        t = [torch.from_numpy(v).to(cuda) for v in arrs]
        # a[0] and c[n-1] are not part of a system
        t[0][:, 0] = float("nan")
        t[2][:, -1] = float("nan")
        g = 1
        while g <= n:
            x = (tg.pcr(*t) if g == n and n > 32 else tg.pcrGauss(*t, g)).cpu().numpy()
            check_against_oracle(*arrs, x)
            if m <= 17 and g < n // 2:
                ref = [torch.from_numpy(v).to(cuda) for v in arrs]
                assert L.tridi_set_tunable(10, 2) == 0
                try:
                    xs = tg.pcrGauss(*ref, g).cpu().numpy()
                finally:
                    L.tridi_set_tunable(10, 0)
                check_ulps(x, xs, ulps=16)
            g *= 2
    assert tg.device_status() == 0


@pytest.mark.parametrize("n", [2048, 4096])
def test_systems_do_not_mix(cuda, n):
    import torch

    m = 7
    arrs = workloads.dominant(m, n, seed=n)
    for g in (64, n):
        x = tg.pcrGauss(*(torch.from_numpy(v).to(cuda) for v in arrs), g).cpu().numpy()
        bad = [v.copy() for v in arrs]
        bad[1][3] = np.nan
        bad[3][3] = np.inf
        y = tg.pcrGauss(*(torch.from_numpy(v).to(cuda) for v in bad), g).cpu().numpy()
        keep = np.arange(m) != 3
        assert np.array_equal(x[keep], y[keep])
