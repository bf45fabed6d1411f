"""The debugging calls (interactions per group, the trace of one group) run the
walk that gravity itself runs: forces bit for bit, counts that add up to the
device counter, and a trace of as many entries as its group has interactions."""
import numpy as np
import pytest

from astraea_gb300 import engine, scenarios

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 33, 1000, 20_011])
@pytest.mark.parametrize("theta", [0.0, 0.5, 0.7])
def test_debugging_calls_run_the_production_walk(n, theta):
    m = max(n, 64)
    st, _ = scenarios.two_granite_spheres(n_target=m - m // 4, n_impactor=m // 4, seed=7)
    st = {k: v[:n].copy() for k, v in st.items()}
    st["originalId"] = np.arange(n, dtype=np.uint32)
    p, alt, bvh = engine.DeviceParticles(n), engine.DeviceParticles(n), engine.TorchBvh(n)
    p.upload(st)
    alt.count = n
    engine.sort_and_build_bvh(p, alt, bvh)
    fields = ["accX", "accY", "accZ", "phiGrav"]
    engine.reset_device_status()
    engine.gravity_barnes_hut(p, bvh, theta)
    flags, counters = engine.read_device_status()
    a = p.download(fields)
    counts = engine.gravity_group_counts(p, bvh, theta)
    b = p.download(fields)
    group = (n + 31) // 32 - 1
    trace = engine.gravity_group_trace(p, bvh, group, theta, capacity=1 << 20)
    c = p.download(fields)
    assert flags == 0
    assert counters["gravity_interactions"] == int(counts.astype(np.int64).sum())
    members = n - 32 * group
    leaves = np.asarray(trace) < 0
    own = np.isin(~np.asarray(trace)[leaves], np.arange(32 * group, n)).sum()
    assert len(trace) * members - own == int(counts[group])
    for f in fields:
        assert np.array_equal(a[f], b[f]) and np.array_equal(a[f], c[f]), f
