"""Refinement with the residual formed in the interleaved solver's back pass
(csrc/large_tma.cu, FP32 batches of a multiple of 32 systems): row counts at
the edges of its chunks (16 rows) and tiles (128), one and several columns of
tiles, every sweep count, against the FP64 oracle and the separate passes
(TRIDI_TUNE_LARGE_TMA = 2): both solve to the residual's own arithmetic, some
1e-13 relative, so x agrees to 1e-11."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

import tridiagonalsolvers_gb300 as tg
from oracle import gold
from tridiagonalsolvers_gb300 import workloads

pytestmark = pytest.mark.gpu


def _refine(cuda, arrs, n, m, max_sweeps):
    import torch

    from tridiagonalsolvers_gb300 import _lib

    L = _lib.lib()
    t = [torch.from_numpy(np.ascontiguousarray(v).ravel()).to(cuda) for v in arrs]
    x = torch.full((n * m,), float("nan"), dtype=torch.float64, device=cuda)
    wsb = L.tridi_refine_workspace_bytes(n, m, 1)
    ws = torch.empty(wsb, dtype=torch.uint8, device=cuda)
    sweeps, rel = ctypes.c_int(-1), ctypes.c_double(0.0)
    st = L.tridi_refine_f32(*(v.data_ptr() for v in t), x.data_ptr(), n, m, 1, 1e-30, max_sweeps, ws.data_ptr(), wsb,
                            torch.cuda.current_stream().cuda_stream, ctypes.byref(sweeps), ctypes.byref(rel))
    assert st == 6 and sweeps.value == max_sweeps
    return x.cpu().numpy().reshape(n, m), rel.value


@pytest.mark.parametrize("n", [33, 48, 127, 128, 129, 144, 145, 256, 257, 1000, 4097, 20011])
@pytest.mark.parametrize("m", [32, 96])
def test_every_edge(cuda, n, m):
    from tridiagonalsolvers_gb300._lib import lib

    L = lib()
    arrs = workloads.weak(m, n, seed=n + m, layout=1)
    for max_sweeps in (0, 1, 2):
        x, rel = _refine(cuda, arrs, n, m, max_sweeps)
        res = gold.rel_residual(*arrs, x, layout=1).max()
        assert res <= (2e-5 if max_sweeps == 0 else 1e-10)
        assert rel <= 4 * res + 1e-13 and res <= 4 * rel + 1e-13
        assert L.tridi_set_tunable(6, 2) == 0
        try:
            y, _ = _refine(cuda, arrs, n, m, max_sweeps)
        finally:
            L.tridi_set_tunable(6, 0)
        assert np.abs(x - y).max() <= (1e-4 if max_sweeps == 0 else 1e-11) * np.abs(y).max()
    assert tg.device_status() == 0


def test_nan_system_is_reported_and_apart(cuda):
    """A NaN in one system ends the refinement (its residual is not a number)
    and leaves the others' first solution as it is without it."""
    n, m = 500, 64
    arrs = workloads.weak(m, n, seed=8, layout=1)
    bad = [v.copy() for v in arrs]
    bad[3][7, 5] = np.nan
    x, _ = _refine(cuda, arrs, n, m, 0)
    y, rel = _refine(cuda, bad, n, m, 0)
    keep = np.arange(m) != 5
    assert np.isnan(rel)
    assert np.array_equal(x[:, keep], y[:, keep])


@pytest.mark.parametrize("n", [47, 49, 63, 64, 65, 79, 80, 81, 191, 192, 193, 255, 321])
def test_correction_from_the_back_pass(cuda, n):
    """The correction's separator system gets its right-hand side from the
    first sweep's back pass: row counts around its tiles (64 rows) and chunks,
    on systems whose corrections all matter (one sweep takes the residual of
    some 1e-7 to 1e-13; a wrong right-hand side in any chunk leaves it)."""
    m = 64
    arrs = workloads.weak(m, n, seed=3 * n, layout=1)
    x, _ = _refine(cuda, arrs, n, m, 1)
    assert gold.rel_residual(*arrs, x, layout=1).max() <= 1e-10
