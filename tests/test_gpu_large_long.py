"""Long contiguous systems (csrc/large_rows.cu): their block rows are solved by a
warp up to 128 of them, by the any-size solver above, and by the block passes
again beyond its range.  Bidiagonal systems of ones carry every block's values
to the other end: with small integers on the right-hand side each operation is
exact in FP32, so the solution is the running sum, exactly."""
from __future__ import annotations

import pytest

import tridiagonalsolvers_gb300 as tg

pytestmark = pytest.mark.gpu
BLOCK = {"float32": 2176, "float64": 1664}  # rows a block


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("blocks,m", [(127, 3), (128, 2), (129, 1), (130, 5), (1000, 3), (4608, 1), (4609, 2), (8704, 1),
                                      (8705, 1)])
def test_running_sums(cuda, dtype, blocks, m):
    import torch

    dt = getattr(torch, dtype)
    for n in (blocks * BLOCK[dtype], (blocks - 1) * BLOCK[dtype] + 5):
        g = torch.Generator(device=cuda).manual_seed(n)
        d = torch.randint(-1, 2, (m, n), generator=g, device=cuda)
        one = torch.ones((m, n), dtype=dt, device=cuda)
        zero = torch.zeros_like(one)
        down = torch.cumsum(d, 1)
        assert int(down.abs().max()) < 2**24
        x = tg.solve_large(-one, one, zero, d.to(dt), n, m)
        assert torch.equal(x.view(m, n).double(), down.double())
        up = d.flip(1).cumsum(1).flip(1)
        x = tg.solve_large(zero, one, -one, d.to(dt), n, m)
        assert torch.equal(x.view(m, n).double(), up.double())
    assert tg.device_status() == 0


def test_one_long_system_streams(cuda):
    """One system of 10^8 rows takes no more than twice what a hundred of 10^6
    take, which have few block rows each (its own block rows solved by one
    warp: over six times)."""
    import torch

    rows = 10**8
    a, c, d = (torch.rand(rows, device=cuda) - 0.5 for _ in range(3))
    b = a.abs() + c.abs() + 1

    def ms(n):
        best = float("inf")
        for _ in range(4):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            tg.solve_large(a, b, c, d, n, rows // n)
            e1.record()
            torch.cuda.synchronize()
            best = min(best, e0.elapsed_time(e1))
        return best

    assert ms(rows) <= 2 * ms(10**6)
