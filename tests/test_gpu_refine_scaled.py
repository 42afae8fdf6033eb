"""Right-hand sides of any size: the refinements' convergence tests sum squares
of residuals, which leave FP32's range long before the residuals do (a
residual of 1e-10 of a right-hand side of 1e-16 squares to zero).  Scaling d
by a power of two scales every FP32 intermediate without rounding, up to
subnormal numbers, so the sweeps and the relative residual of the scaled
system are those of the unscaled one: the residual to 1e-4 (its FP32 sums, and
the last bits of residuals near 2^-130), x to the 1e-10 of every refinement."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

import tridiagonalsolvers_gb300 as tg
from oracle import gold
from tridiagonalsolvers_gb300 import workloads

pytestmark = pytest.mark.gpu

SCALES = (-66, -53, 60, 100)  # 2^-66 = 1.4e-20, 2^100 = 1.3e30


def _refine(cuda, arrs, n, m, layout, tol=1e-10, max_sweeps=10, residual=1):
    """(status, x, sweeps, rel) of tridi_refine_f32."""
    import torch

    from tridiagonalsolvers_gb300 import _lib

    L = _lib.lib()
    t = [torch.from_numpy(np.ascontiguousarray(v).ravel()).to(cuda) for v in arrs]
    x = torch.full((n * m,), float("nan"), dtype=torch.float64, device=cuda)
    wsb = L.tridi_refine_workspace_bytes(n, m, layout)
    ws = torch.empty(wsb, dtype=torch.uint8, device=cuda)
    sweeps, rel = ctypes.c_int(-1), ctypes.c_double(-1.0)
    prev = L.tridi_get_tunable(4)  # TRIDI_TUNE_RESIDUAL
    assert L.tridi_set_tunable(4, residual) == 0
    try:
        st = L.tridi_refine_f32(*(v.data_ptr() for v in t), x.data_ptr(), n, m, layout, tol, max_sweeps, ws.data_ptr(),
                                wsb, torch.cuda.current_stream().cuda_stream, ctypes.byref(sweeps), ctypes.byref(rel))
    finally:
        L.tridi_set_tunable(4, prev)
    return st, x.cpu().numpy().reshape(np.shape(arrs[0])), sweeps.value, rel.value


def _check(cuda, k, arrs, n, m, layout, **kw):
    st1, x1, sweeps1, rel1 = _refine(cuda, arrs, n, m, layout, **kw)
    assert st1 == 0 and 0 < rel1 <= kw.get("tol", 1e-10)
    f = np.float64(2.0) ** k
    scaled = (*arrs[:3], (arrs[3] * f).astype(np.float32))
    st, x, sweeps, rel = _refine(cuda, scaled, n, m, layout, **kw)
    assert (st, sweeps) == (0, sweeps1), (st, sweeps, rel, rel1)
    assert abs(rel - rel1) <= 1e-4 * rel1, (rel, rel1)
    if sweeps:
        x64 = gold.solve_f64(*(np.ascontiguousarray(v.T) for v in arrs)).T if layout else gold.solve_f64(*arrs)
        assert np.abs(x / f - x64).max() <= 1e-10 * np.abs(x64).max()


@pytest.mark.parametrize("k", SCALES)
@pytest.mark.parametrize("n,m", [(5, 40), (64, 333), (500, 7), (1000, 20), (2200, 6), (8704, 3)])
def test_contiguous_one_kernel(cuda, n, m, k):
    """csrc/refine_rows.cu, a warp's and a CTA's systems."""
    _check(cuda, k, workloads.dominant(m, n, seed=n), n, m, 0, max_sweeps=1)


@pytest.mark.parametrize("k", SCALES)
@pytest.mark.parametrize("n,m", [(40, 64), (129, 32), (5000, 32)])
def test_interleaved_back_pass(cuda, n, m, k):
    """csrc/large_tma.cu: the residuals of its back pass and of its tiles' last rows."""
    _check(cuda, k, workloads.dominant(m, n, seed=n, layout=1), n, m, 1, max_sweeps=1)


@pytest.mark.parametrize("k", SCALES)
@pytest.mark.parametrize("residual", [1, 2])  # TRIDI_RESIDUAL_DF, TRIDI_RESIDUAL_FP64
@pytest.mark.parametrize("n,m,layout", [(300, 20, 0), (1024, 9, 0), (9001, 4, 0), (700, 31, 1)])
def test_separate_passes(cuda, n, m, layout, residual, k):
    """csrc/refine.cu's residual passes: tolerances that the first solution
    meets, native FP64 residuals, systems longer than a CTA holds, interleaved
    batches of no multiple of 32."""
    arrs = workloads.dominant(m, n, seed=n, layout=layout)
    _check(cuda, k, arrs, n, m, layout, tol=1e-5, residual=residual)
    _check(cuda, k, arrs, n, m, layout, max_sweeps=1, residual=residual)


@pytest.mark.parametrize("layout", [0, 1])
def test_no_number_is_no_convergence(cuda, layout):
    """A system whose ||d||^2 is no number is not converged (its absolute
    residual is no measure), whatever the others are."""
    n, m = 300, 9
    for bad in (np.inf, np.nan):
        arrs = [v.copy() for v in workloads.dominant(m, n, seed=2, layout=layout)]
        arrs[3] *= np.float32(2.0**-66)
        arrs[3][4, 5] = bad
        for tol in (1e-5, 1e-10):
            st, _, _, rel = _refine(cuda, arrs, n, m, layout, tol=tol, max_sweeps=1)
            assert st == 6 and np.isnan(rel)


@pytest.mark.parametrize("k", SCALES)
@pytest.mark.parametrize("residual", ["df", "fp64"])
@pytest.mark.parametrize("sweeps", [1, 2])
@pytest.mark.parametrize("big", [False, True])
def test_ragged(cuda, big, sweeps, residual, k):
    """csrc/ragged.cu: systems of a warp, a team, the CTA and (big) beyond the
    staging ring; the residual it returns, and x."""
    import torch

    from tridiagonalsolvers_gb300.ragged import RaggedPlan, RaggedRefiner, padded

    sizes = [1, 2, 33, 480, 481, 1000, 4800, 4801, 8100, 77] * 3 + ([20000] if big else [])
    a, b, c, d, off = workloads.adi(np.array(sizes), seed=7)
    total = int(off[-1])

    def solve(rhs):
        t = []
        for v in (a, b, c, rhs):
            u = torch.zeros(padded(total), dtype=torch.float32, device=cuda)
            u[:total] = torch.from_numpy(v)
            t.append(u)
        r = RaggedRefiner(RaggedPlan(off, refine=True), *t, sweeps=sweeps, graph=False, residual=residual)
        x, rel = r.run()
        return x.cpu().numpy()[:total], rel

    f = np.float64(2.0) ** k
    x1, rel1 = solve(d)
    x, rel = solve((d * f).astype(np.float32))
    assert 0 < rel1 <= 1e-10 and abs(rel - rel1) <= 1e-4 * rel1, (rel, rel1)
    assert np.abs(x / f - x1).max() <= 1e-10 * np.abs(x1).max()


def test_ragged_no_number(cuda):
    """One system's infinite right-hand side: the batch's residual is no number."""
    import torch

    from tridiagonalsolvers_gb300.ragged import RaggedPlan, RaggedRefiner, padded

    a, b, c, d, off = workloads.adi(np.array([30, 700, 5000, 60]), seed=3)
    total = int(off[-1])
    for bad in (np.inf, np.nan):
        d[35] = bad
        t = []
        for v in (a, b, c, d):
            u = torch.zeros(padded(total), dtype=torch.float32, device=cuda)
            u[:total] = torch.from_numpy(v)
            t.append(u)
        assert np.isnan(RaggedRefiner(RaggedPlan(off, refine=True), *t, sweeps=1, graph=False).run()[1])
