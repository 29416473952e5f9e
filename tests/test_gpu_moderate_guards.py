"""What keeps the unguarded arithmetic of moderate tiles safe from outside the
state: a side whose ghost cell is not moderate beside cells that are (tiny, huge
and subnormal discharges and depths), and a spacing whose reciprocal the
unguarded division by it does not take (an all-ones low word, an exponent beyond
2^40 or below 2^-40), or does, but inexactly. Stages and the CFL bound equal the
oracle's bit for bit."""
import struct

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def all_ones(hi):
    """The double of the high word hi whose low word is all ones."""
    return struct.unpack("<d", struct.pack("<II", 0xffffffff, hi))[0]


def _compare(oracle, sides, dx, dy, shape, dt):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from hydroflux_b200 import sim, step
    rng = np.random.default_rng(5)
    z = rng.uniform(0.0, 2.0, shape)
    h = rng.uniform(0.05, 1.5, shape)
    h[rng.random(shape) < 0.15] = 0.0
    hu, hv = h * rng.normal(0, 0.5, shape), h * rng.normal(0, 0.5, shape)
    n = np.full(shape, 0.03)
    bcs = sim.Boundaries2D(*[getattr(sim.Boundary, k)(*v) for k, *v in sides])
    m = step.DeviceMesh(z, dx, dy, n)
    dev = [torch.tensor(a, device="cuda") for a in (h, hu, hv)]
    bound = step.cfl_time_step_with_bcs(*dev, m, bcs, 0.45)
    assert bound == oracle.cfl_time_step(z, dx, dy, h, hu, hv, 0.45, bcs.to_c(), n)
    step.ssprk2_step(*dev, m, bcs, dt)
    ref = oracle.ssprk2_step(z, dx, dy, h, hu, hv, bcs.to_c(), dt, n)
    for name, a, b in zip(("h", "hu", "hv"), dev, ref):
        assert np.array_equal(a.cpu().numpy(), b, equal_nan=True), name


@pytest.mark.parametrize("shape", [(9, 33), (40, 72), (330, 350)])
@pytest.mark.parametrize("kind,value", [("discharge", 1.0e-250), ("discharge", -5.0e-324),
                                        ("discharge", 1.0e40), ("depth", 1.0e-310),
                                        ("depth", 1.0e40)])
def test_extreme_ghosts_equal_the_oracle(oracle, kind, value, shape):
    _compare(oracle, [(kind, value), ("wall",), (kind, value), ("transmissive",)], 1.1, 0.7,
             shape, 0.01)


@pytest.mark.parametrize("shape", [(9, 33), (40, 72), (330, 350)])
@pytest.mark.parametrize("dx,dy", [(0.3, 0.7), (all_ones(0x3ff80000), 1.3),
                                   (1.3, all_ones(0x40012345)), (3.0 * 2.0**41, 1.3),
                                   (1.3, 1.7 * 2.0**-43)])
def test_spacings_equal_the_oracle(oracle, dx, dy, shape):
    _compare(oracle, [("wall",), ("transmissive",), ("discharge", 0.3), ("depth", 0.4)], dx, dy,
             shape, 0.01 * min(dx, dy))
