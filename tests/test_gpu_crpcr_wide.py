"""CR and CR-PCR across the warps of a CTA (csrc/crpcr_wide.cu: FP32, 2048 and
4096 unknowns), every switch level, batches of one system, a few and more than
the GPU holds at once: against the FP64 oracle; rest 2 (cr) bit for bit the
shared-memory CR kernel's and the hybrid kernel's results, above within 16 ulp
of the hybrid kernel (TRIDI_TUNE_PCR_KERNEL = 2)."""
from __future__ import annotations

import numpy as np
import pytest

import tridiagonalsolvers_gb300 as tg
from tridiagonalsolvers_gb300 import workloads

from .parity import check_against_oracle, check_ulps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2048, 4096])
def test_every_switch_level(cuda, n):
    import torch

    from tridiagonalsolvers_gb300._lib import lib

    L = lib()
    for m in (1, 3, 2 * 152 * 4 + 1):
        arrs = workloads.dominant(m, n, seed=n + m)
        t = [torch.from_numpy(v).to(cuda) for v in arrs]
        ends = [v.clone() for v in t]
        ends[0][:, 0] = float("nan")  # a[0] and c[n-1] are not part of a system
        ends[2][:, -1] = float("nan")
        rest = 2
        while rest <= n // 2:
            x = tg.crpcr(*t, rest).cpu().numpy()
            check_against_oracle(*arrs, x)
            assert np.array_equal(x, tg.crpcr(*ends, rest).cpu().numpy())
            if m <= 3:
                assert L.tridi_set_tunable(10, 2) == 0
                try:
                    xs = tg.crpcr(*t, rest).cpu().numpy()
                finally:
                    L.tridi_set_tunable(10, 0)
                if rest == 2:
                    assert np.array_equal(x, xs)
                    assert L.tridi_set_tunable(8, 2) == 0
                    try:
                        assert np.array_equal(x, tg.crNBC(*t).cpu().numpy())
                    finally:
                        L.tridi_set_tunable(8, 0)
                else:
                    check_ulps(x, xs, ulps=16)
            rest *= 2
    assert tg.device_status() == 0


@pytest.mark.parametrize("n", [2048, 4096])
def test_systems_do_not_mix(cuda, n):
    import torch

    m = 7
    arrs = workloads.dominant(m, n, seed=n)
    bad = [v.copy() for v in arrs]
    bad[1][3] = np.nan
    bad[3][3] = np.inf
    keep = np.arange(m) != 3
    for rest in (2, 8, n // 32):
        x = tg.crpcr(*(torch.from_numpy(v).to(cuda) for v in arrs), rest).cpu().numpy()
        y = tg.crpcr(*(torch.from_numpy(v).to(cuda) for v in bad), rest).cpu().numpy()
        assert np.array_equal(x[keep], y[keep])
