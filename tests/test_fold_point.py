"""The guard folds in closed form (fold_point): a host harness
(tests/fold_point_check.cu, built with nvcc, no GPU needed) compares every
element with the slab operations run one after the other."""
import os
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.mark.skipif(shutil.which("nvcc") is None and not os.path.exists("/usr/local/cuda/bin/nvcc"),
                    reason="nvcc not found")
def test_fold_point_is_the_operations_in_order(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = tmp_path / "fold_point_check"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O1", "-I",
                    str(ROOT / "include"), "-I", str(ROOT / "ctca_b200" / "csrc"),
                    str(ROOT / "tests" / "fold_point_check.cu"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
    assert out.stdout.startswith("ok")
