"""FP64 division on the integer units (csrc/div64.cuh).  Its quotient is
within (1/2 + 2^-7) ulp of a / b: at most one ulp from the IEEE quotient, and
another value only where a / b lies within 2^-7 ulp of a tie (a share of at
most 2^-6 of random operands).  Zeros, subnormals, infinities, NaN and
quotients outside the normal range are the IEEE ones exactly."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
SPECIAL = np.array([0.0, -0.0, 1.0, -2.0, 3.0, np.inf, -np.inf, np.nan, 5e-324, -1e-310, 2.2250738585072014e-308,
                    1e308, 1.7976931348623157e308, 1.0 - 2.0**-53, 1.0 + 2.0**-52])


def _operands(count, seed):
    """Random significands (some with long runs of zeros or ones) and exponents."""
    g = np.random.default_rng(seed)
    out = []
    for _ in range(2):
        mant = g.integers(0, 1 << 52, count, dtype=np.uint64)
        low = (np.uint64(1) << g.integers(0, 53, count, dtype=np.uint64)) - np.uint64(1)
        kind = g.integers(0, 4, count)
        mant = np.where(kind == 0, mant & ~low, np.where(kind == 1, mant | low, mant)) & np.uint64((1 << 52) - 1)
        bits = mant | (g.integers(700, 1347, count, dtype=np.uint64) << np.uint64(52)) | (
            g.integers(0, 2, count, dtype=np.uint64) << np.uint64(63))
        out.append(bits.view(np.float64))
    return out


def _check(q, a, b):
    with np.errstate(all="ignore"):
        t = a / b
    same = (q.view(np.int64) == t.view(np.int64)) | (np.isnan(q) & np.isnan(t))
    normal = np.isfinite(t) & (np.abs(t) >= 2.0**-1021) & (np.abs(a) >= 2.0**-1022) & (np.abs(b) >= 2.0**-1022)
    assert np.all(same[~normal])
    assert np.abs(q.view(np.int64) - t.view(np.int64))[normal].max() <= 1
    assert np.mean(~same) <= 2.0**-6


def _cases():
    a, b = _operands(200000, 3)
    sa, sb = (v.ravel() for v in np.meshgrid(SPECIAL, SPECIAL))
    return np.concatenate([a, sa]), np.concatenate([b, sb])


def test_host_form(tmp_path):
    cxx = shutil.which("g++")
    inc = Path("/usr/local/cuda/include")
    if not cxx or not inc.exists():
        pytest.skip("no host compiler or CUDA headers")
    exe = tmp_path / "div64_check"
    subprocess.run([cxx, "-O2", "-std=c++17", f"-I{ROOT / 'tridiagonalsolvers_gb300' / 'csrc'}", f"-I{inc}",
                    str(ROOT / "tests" / "cpp" / "div64_check.cpp"), "-o", str(exe)], check=True)
    a, b = _cases()
    r = subprocess.run([str(exe)], input=np.stack([a, b], 1).tobytes(), capture_output=True, check=True)
    q = np.frombuffer(r.stdout, np.float64).reshape(-1, 4)
    _check(np.ascontiguousarray(q[:, 0]), a, b)
    _check(np.ascontiguousarray(q[:, 1]), a, b)
    _check(np.ascontiguousarray(q[:, 2]), -a, b)
    _check(np.ascontiguousarray(q[:, 3]), np.full_like(b, 2.0), b)


@pytest.mark.gpu
def test_device_form(cuda):
    """tridi_selfcheck_div_f64: the division as the kernels issue it."""
    import torch

    from tridiagonalsolvers_gb300 import _lib

    a, b = _cases()
    ta, tb = (torch.from_numpy(v).to(cuda) for v in (a, b))
    q = torch.empty_like(ta)
    _lib.check(_lib.lib().tridi_selfcheck_div_f64(ta.data_ptr(), tb.data_ptr(), q.data_ptr(), len(a),
                                                  torch.cuda.current_stream().cuda_stream), "selfcheck")
    _check(q.cpu().numpy(), a, b)
