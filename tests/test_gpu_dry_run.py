"""Runs of dry tiles (stage_dry_run): a dry grid with a few wet patches, so that
each CTA's tiles start and end such runs, in its tiles' order or in the last
tile, with rain and a source that wet a dry tile, against the oracle bit for
bit. Even and odd column counts (copies of pairs and of single columns)."""
import numpy as np
import pytest

from tests.gpu_util import exact_fraction

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,shape", [("tile32", (900, 704)), ("tile32", (896, 705)),
                                        ("tile", (480, 1600)), ("tile", (483, 1601))])
@pytest.mark.parametrize("rain", [0.0, 1.0e-7])
def test_dry_runs_against_oracle(oracle, kind, shape, rain):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from hydroflux_b200 import sim
    from oracle.oracle import Forcing
    nr, nc = shape
    rng = np.random.default_rng(nc)
    z = 0.1 * np.abs(np.arange(nr) - nr / 3)[:, None] + rng.uniform(0, 0.1, shape)
    h = np.where(rng.random(shape) < 0.5, 0.0, 5.0e-7)
    for r, c in ((40, 40), (300, 333), (400, nc - 50), (nr - 20, 500)):
        h[r:r + 9, c:c + 12] = 0.5
    hu, hv = 0.1 * h, -0.05 * h
    n = np.full(shape, 0.03)
    cfg = sim.SimulationConfig(cfl=0.45, boundaries=sim.Boundaries2D(
        sim.Boundary.wall(), sim.Boundary.transmissive(), sim.Boundary.transmissive(),
        sim.Boundary.wall()))
    at = (nr // 2, nc // 2)
    with sim.Simulation(sim.Mesh2D(z, 1.0, 1.5, n), (h, hu, hv), cfg, device=0) as s:
        s.set_stage_kernel(kind)
        s.set_rain(rain)
        s.set_point_sources([sim.PointSource(*at, 0.2)])
        s.run_steps(5)
        got = s.states()
    f = Forcing(rain=(np.array([0.0]), np.array([rain])),
                sources=[(*at, np.array([0.0]), np.array([0.2]))])
    r = oracle.sim_run(z, n, 1.0, 1.5, h, hu, hv, cfg.to_c(), float("inf"), forcing=f,
                       stop_after=5)
    assert r["status"] == 0
    assert exact_fraction(got, (r["h"], r["hu"], r["hv"])) == 1.0
