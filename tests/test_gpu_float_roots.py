"""The float square roots and quotients of the 16-bit kernels' subgrid rate are
the correctly rounded ones, for every float of the ranges they are used on."""
from __future__ import annotations

import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent


def test_roots_and_quotients_of_every_float(tmp_path):
    from turbulent_lbm_multigpu_gb300 import build

    exe = tmp_path / "float_roots_check"
    subprocess.run([build.nvcc()] + build.ARCH + build.NVFLAGS + [str(ROOT / "tests/cpp/float_roots_check.cu"), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
