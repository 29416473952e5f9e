"""The tangent stage on both its CTAs: with as many lanes as fill the SMs one
tile each (512 threads) and one lane more (256 threads), every common lane has
the same tangent bit for bit."""
import numpy as np
import pytest

from tests.test_gpu_calib import directions, observations, problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["inflow"])
@pytest.mark.parametrize("steps", [1, 9])
def test_lane_counts_around_one_wave(name, steps):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from hydroflux_b200 import calib, workloads
    s, _, gauges = problem(workloads, name)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    lanes = max(sms // (-(-s.shape[0] // 8) * -(-s.shape[1] // 32)), 1)
    rng = np.random.default_rng(5)
    ds = [directions(rng, s) for _ in range(lanes + 1)]
    got = []
    with calib.Calibration(s, steps, gauges) as cal:
        observations(cal, s, steps, len(gauges), 11)
        for m in (lanes, lanes + 1):
            J, dJ = cal.tangent_lanes(s.manning, **{k: np.stack([d[k] for d in ds[:m]])
                                                    for k in ds[0]})
            got.append((J, dJ, [cal.lane_state(q) for q in range(lanes)], cal.final_state()))
    (Ja, da, la, fa), (Jb, db, lb, fb) = got
    assert Ja == Jb and np.array_equal(da, db[:lanes])
    for a, b in zip(la, lb):
        assert all(np.array_equal(a[k], b[k]) for k in ("dh", "dhu", "dhv"))
    assert all(np.array_equal(fa[k], fb[k]) for k in ("h", "hu", "hv"))
