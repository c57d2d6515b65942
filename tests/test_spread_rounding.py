"""The exponent spread that picks a split product's precision is rounded exactly (no GPU needed)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc not on PATH")
def test_spread_is_the_nearest_integer(tmp_path):
    exe = str(tmp_path / "spread_check")
    csrc = os.path.join(ROOT, "flag4j_gb300", "csrc")
    cmd = ["nvcc", "-std=c++17", "-O2", "-gencode", "arch=compute_103a,code=sm_103a", "--expt-relaxed-constexpr",
           "-I", os.path.join(ROOT, "include"), "-o", exe, os.path.join(HERE, "native", "spread_check.cu"),
           os.path.join(csrc, "f4j_core.cu"), os.path.join(csrc, "f4j_dense.cu"), os.path.join(csrc, "f4j_config.cu")]
    subprocess.run(cmd, check=True, capture_output=True, timeout=600)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout[-2000:]
