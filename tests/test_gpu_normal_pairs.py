"""The FP32 noise's packed pairs equal the scalar ones for every uniform."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu


def test_packed_pairs_equal_scalar_pairs_for_every_uniform(cuda, tmp_path):
    from libbi_b200 import build

    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cpp", "normal_pair_test.cu")
    exe = str(tmp_path / "normal_pair_test")
    flags = [f for f in build.NVCC_FLAGS if f not in ("-Xcompiler", "-fPIC")]
    subprocess.run([build.nvcc()] + flags + [src, "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "0\n", r.stdout + r.stderr
