"""A build with a quadratic form wider than the one-launch PSO takes compiles:
that kernel is left out and the per-iteration one serves."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc not available")
def test_wide_quadratic_forms_compile(tmp_path):
    cmd = ["nvcc", "-std=c++20", "--expt-relaxed-constexpr", "-gencode",
           "arch=compute_100a,code=sm_100a", "-I", str(ROOT / "include"), "-I",
           str(ROOT / "zeus_b200" / "csrc"), "-c", str(ROOT / "tests" / "cpp" / "wide_gaussian.cu"),
           "-o", str(tmp_path / "wide.o")]
    r = subprocess.run(cmd, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr
