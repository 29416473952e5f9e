"""The tile kernels' CTAs on grids at the limits of their rule: 148 and 149
tiles of 32 x 4 (512 threads, then 768 per 32 x 8 tile), 148 and 149 of 32 x 8
(then 384 threads), 296 and 297 (then 256 threads), with point sources in both
halves of an 8-row source bucket, against the oracle bit for bit."""
import numpy as np
import pytest

from tests.gpu_util import exact_fraction

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(4, 33), (588, 33), (296, 64), (592, 32), (593, 32), (1184, 32),
                                   (1185, 32), (2368, 32), (2369, 32), (296, 200)])
def test_geometry_limits_against_oracle(oracle, shape):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from hydroflux_b200 import sim
    from oracle.oracle import Forcing
    nr, nc = shape
    rng = np.random.default_rng(nr + nc)
    z = 0.05 * np.abs(np.arange(nc) - nc / 2)[None, :] + rng.uniform(0, 0.2, shape)
    n = rng.choice([0.025, 0.05], size=shape)
    h = np.where(rng.random(shape) < 0.7, rng.uniform(0, 0.5, shape), 0.0)
    hu, hv = h * rng.normal(0, 0.3, shape), h * rng.normal(0, 0.3, shape)
    bcs = sim.Boundaries2D(sim.Boundary.wall(), sim.Boundary.transmissive(), sim.Boundary.wall(),
                           sim.Boundary.depth(0.4))
    cfg = sim.SimulationConfig(cfl=0.45, boundaries=bcs)
    cells = [(0, 0), (3, nc - 1), (nr - 1, 5), (nr // 2 // 8 * 8, 7),
             (min(nr // 2 // 8 * 8 + 4, nr - 1), 7)]
    with sim.Simulation(sim.Mesh2D(z, 1.0, 2.0, n), (h, hu, hv), cfg, device=0) as s:
        s.set_rain(1.0e-4)
        s.set_point_sources([sim.PointSource(r, c, 0.5) for r, c in cells])
        s.run_steps(4)
        got = s.states()
    f = Forcing(rain=(np.array([0.0]), np.array([1.0e-4])),
                sources=[(r, c, np.array([0.0]), np.array([0.5])) for r, c in cells])
    r = oracle.sim_run(z, n, 1.0, 2.0, h, hu, hv, cfg.to_c(), float("inf"), forcing=f,
                       stop_after=4)
    assert r["status"] == 0
    assert exact_fraction(got, (r["h"], r["hu"], r["hv"])) == 1.0
