"""A dry tile with an extreme value leaves the tiles after it in their own class
(the unguarded arithmetic for moderate ones)."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "native", "dry_tile_class_check.cu")
OUT = os.path.join(HERE, "native", "_build", "dry_tile_class_check")


def test_dry_tile_leaves_no_extreme_behind():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                    "--fmad=false", "-prec-div=true", "-prec-sqrt=true",
                    "--expt-relaxed-constexpr", SRC, "-o", OUT], check=True)
    r = subprocess.run([OUT], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
