"""Faces with a dry or very thin side, unguarded (hf::wb_face_moderate), equal
the guarded hf::wb_face bit for bit."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "native", "partial_face_check.cu")
OUT = os.path.join(HERE, "native", "_build", "partial_face_check")


@pytest.mark.parametrize("faces", [1, 1 << 26])
def test_partial_faces_match_guarded(faces):
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
    r = subprocess.run([OUT, str(faces)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "mismatches moderate 0, wet 0" in r.stdout
