"""The CTAs that the automatic choice takes on grids that leave SMs idle (32 x 4
tiles by 512 threads, 32 x 8 by 768 and 384) and the 32 x 8 tiles by 256
threads, on grids several tiles wide with partial last tiles both ways: every
set of sides and both integrators against the oracle bit for bit."""
import numpy as np
import pytest

from tests.gpu_util import exact_fraction
from tests.test_gpu_parity import BC_SETS, random_case

pytestmark = pytest.mark.gpu


# 66 tiles of 32 x 4; 287 of those and 147 of 32 x 8; 171, 363 and 400 of 32 x 8
@pytest.mark.parametrize("integrator", [0, 1])
@pytest.mark.parametrize("bc", sorted(BC_SETS))
@pytest.mark.parametrize("kind,shape", [("auto", (131, 35)), ("auto", (161, 200)),
                                        ("auto", (150, 257)), ("auto", (259, 321)),
                                        ("tile", (199, 481))])
def test_small_ctas_against_oracle(oracle, kind, shape, bc, integrator):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from hydroflux_b200 import sim
    z, n, h, hu, hv = random_case(*shape, seed=sum(shape) + len(bc))
    cfg = sim.SimulationConfig(cfl=0.45, max_dt=0.5, integrator=sim.Integrator(integrator),
                               boundaries=sim.Boundaries2D(
                                   *[sim.Boundary(k, v) for k, v in BC_SETS[bc]]))
    with sim.Simulation(sim.Mesh2D(z, 2.0, 1.5, n), (h, hu, hv), cfg) as s:
        s.set_stage_kernel(kind)
        s.run_steps(6)
        got, t = s.states(), s.time()
    r = oracle.sim_run(z, n, 2.0, 1.5, h, hu, hv, cfg.to_c(), float("inf"), stop_after=6)
    assert r["status"] == 0 and r["steps"] == 6 and r["t"] == t
    assert exact_fraction(got, (r["h"], r["hu"], r["hv"])) == 1.0
