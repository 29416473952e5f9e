"""The unguarded arithmetic of moderate tiles (hfa::recip_rn, quo_keep,
quo_plus, sqrt_rn_moderate, hf::wb_face_wet) equals the guarded one bit for
bit, and a tile that holds a value outside the moderate range takes the
guarded form: stages on states with tiny, huge, negative or all-ones values
equal the oracle's."""
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "native", "moderate_math_check.cu")
OUT = os.path.join(HERE, "native", "_build", "moderate_math_check")


@pytest.fixture(scope="module")
def torch():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def test_moderate_operations_match_ieee(torch):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                    "--fmad=false", "-prec-div=true", "-prec-sqrt=true",
                    "--expt-relaxed-constexpr", SRC, "-o", OUT], check=True)
    r = subprocess.run([OUT, str(1 << 28)], capture_output=True, text=True, timeout=300)
    print(r.stdout)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.count("mismatches") == 4


def _state(kind, shape, seed):
    rng = np.random.default_rng(seed)
    z = rng.uniform(0.0, 2.0, shape)
    h = rng.uniform(0.05, 1.5, shape)
    h[rng.random(shape) < 0.15] = 0.0
    hu, hv = h * rng.normal(0, 0.5, shape), h * rng.normal(0, 0.5, shape)
    at = (shape[0] // 2, shape[1] // 2)
    if kind == "tiny momentum":
        hu[at], hv[at[0] + 1, at[1]] = 1.0e-250, 5.0e-324
    elif kind == "huge bed":
        z[at] = 1.0e35
    elif kind == "negative depth":
        h[at] = -1.0e-3
    elif kind == "tiny depth":
        h[at] = 1.0e-310
    elif kind == "large momentum":
        hu[at] = 1.0e40
    elif kind == "all ones":  # significands of all ones, quotients of powers of two
        h[:] = np.where(h > 0, np.nextafter(1.0, 0.0), 0.0)
        z[:], hu[:], hv[:] = 0.0, np.where(h > 0, 0.5, 0.0), 0.0
    return z, h, hu, hv


@pytest.mark.parametrize("shape", [(9, 33), (40, 72), (330, 350)])
@pytest.mark.parametrize("kind", ["plain", "tiny momentum", "huge bed", "negative depth",
                                  "tiny depth", "large momentum", "all ones"])
def test_stage_with_extreme_values_equals_the_oracle(torch, kind, shape):
    from hydroflux_b200 import abi, sim, step
    from oracle import oracle
    z, h, hu, hv = _state(kind, shape, 3)
    n = np.full(shape, 0.03)
    bcs = sim.Boundaries2D(sim.Boundary.wall(), sim.Boundary.transmissive(), sim.Boundary.wall(),
                           sim.Boundary.transmissive())
    m = step.DeviceMesh(z, 1.0, 2.0, n)
    dev = [torch.tensor(a, device="cuda") for a in (h, hu, hv)]
    dt = 0.01
    step.ssprk2_step(*dev, m, bcs, dt)
    step.manning_friction_step(*dev, m, dt, 1.0e-6)
    ref = oracle.ssprk2_step(z, 1.0, 2.0, h, hu, hv, bcs.to_c(), dt, n)
    ref = oracle.manning_friction_step(n, *ref, dt, 1.0e-6)
    for name, a, b in zip(("h", "hu", "hv"), dev, ref):
        assert np.array_equal(a.cpu().numpy(), b, equal_nan=True), (kind, name)
