"""Passes that only the scalar kernels have refuse a pair plan instead of giving wrong numbers (no GPU)."""
import os
import subprocess

import pytest

from spim_registration_gb300 import _build

HERE = os.path.dirname(os.path.abspath(__file__))


def test_scalar_only_passes_refuse_pair_plans(tmp_path):
    try:
        nvcc = _build.nvcc()
    except RuntimeError:
        pytest.skip("no nvcc")
    lib = _build.build()
    exe = str(tmp_path / "scalar_only_check")
    subprocess.run([nvcc, *_build.ARCH, "-std=c++17", "-o", exe, os.path.join(HERE, "scalar_only_check.cu"), lib],
                   check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
