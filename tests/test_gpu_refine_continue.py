"""Sweeps after the one-kernel correction of contiguous systems (csrc/refine.cu):
||d||^2 from a pass on x = 0, x split into pairs, the residual from a pass with a
zero correction, then sweeps that alternate between x and the workspace's copy.
A tolerance that no sweep meets makes max_sweeps the number of sweeps; x is the
last iterate (residual and forward error 1e-10 against the FP64 oracle, as for
every refinement) and the returned residual is x's."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from oracle import gold
from tridiagonalsolvers_gb300 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("make", [workloads.dominant, workloads.weak])
@pytest.mark.parametrize("n,m", [(3, 50), (50, 9), (300, 9), (512, 40), (1500, 5), (8704, 2)])
@pytest.mark.parametrize("sweeps", [1, 2, 3, 4])
def test_last_iterate(cuda, n, m, make, sweeps):
    import torch

    from tridiagonalsolvers_gb300 import _lib

    L = _lib.lib()
    arrs = make(m, n, seed=n + sweeps)
    t = [torch.from_numpy(np.ascontiguousarray(v).ravel()).to(cuda) for v in arrs]
    x = torch.full((n * m,), float("nan"), dtype=torch.float64, device=cuda)
    wsb = L.tridi_refine_workspace_bytes(n, m, 0)
    ws = torch.full((wsb,), 255, dtype=torch.uint8, device=cuda)
    done, rel = ctypes.c_int(-1), ctypes.c_double(-1.0)
    st = L.tridi_refine_f32(*(v.data_ptr() for v in t), x.data_ptr(), n, m, 0, 1e-30, sweeps, ws.data_ptr(), wsb,
                            torch.cuda.current_stream().cuda_stream, ctypes.byref(done), ctypes.byref(rel))
    assert st == 6 and done.value == sweeps
    x = x.cpu().numpy().reshape(m, n)
    res = gold.rel_residual(*arrs, x).max()
    assert res <= 1e-10 and rel.value <= 4 * res + 1e-13 and res <= 4 * rel.value + 1e-13
    x64 = gold.solve_f64(*arrs)
    assert np.abs(x - x64).max() <= 1e-10 * np.abs(x64).max()
