"""Launches run once (csrc/runtime.h, checked_launch): an error that the calling
thread had not read does not make one run twice, and is returned after it; a
launch that fails for want of the shared-memory limit is repeated once with the
limit set.  On the CPU, against fakes of the runtime."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
BAD, OTHER = 1, 2  # cudaErrorInvalidValue, cudaErrorMemoryAllocation


def test_launches_run_once(tmp_path):
    cxx = shutil.which("g++")
    inc = Path("/usr/local/cuda/include")
    if not cxx or not inc.exists():
        pytest.skip("no host compiler or CUDA headers")
    exe = tmp_path / "launch_check"
    subprocess.run([cxx, "-O1", "-std=c++17", f"-I{ROOT / 'tridiagonalsolvers_gb300' / 'csrc'}",
                    f"-I{ROOT / 'include'}", f"-I{inc}", str(ROOT / "tests" / "cpp" / "launch_check.cpp"), "-o",
                    str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    rows = [tuple(int(v) for v in line.split()) for line in out.splitlines()]
    # launches, limits raised, status returned, error left unread
    assert rows == [
        (1, 0, 0, 0),
        (1, 0, BAD, 0),
        (1, 0, OTHER, 0),
        (2, 1, 0, 0),
        (2, 1, 0, 0),
        (2, 1, BAD, 0),
        (1, 0, BAD, 0),
        (1, 0, BAD, 0),
        (1, 0, OTHER, 0),
    ]
