"""Gravity beside the neighbour lists, pass 1 and the EOS, in the far-field modes
whose walk runs there: the fused step against itself with timed stages (which run
one after the other), and a relaxation's initial forces against the stage calls."""
import numpy as np
import pytest

from astraea_gb300 import engine, scenarios
from conftest import rel_rms

pytestmark = pytest.mark.gpu


def state(n):
    m = max(n, 64)
    st, _ = scenarios.two_granite_spheres(n_target=m - m // 4, n_impactor=m // 4, seed=42)
    st = {k: v[:n].copy() for k, v in st.items()}
    st["originalId"] = np.arange(n, dtype=np.uint32)
    return st


@pytest.fixture(params=[0, 1, 3])
def mode(request):
    engine.set_far_field(request.param)
    yield request.param
    engine.set_far_field(0)


@pytest.mark.parametrize("n", [2, 33, 4097, (1 << 19) + 1])
def test_step_equals_step_with_timed_stages(mode, n):
    st = state(n)
    out = []
    for timed in (False, True):
        sim = engine.Simulation(n)
        sim.p.upload(st)
        sim.alt.count = n
        sim.evaluate_initial_forces(0.7)
        engine.set_stage_timing(timed)
        try:
            dts = [sim.step(5.0e-3, 0.7) for _ in range(3)]
        finally:
            engine.set_stage_timing(False)
        out.append((dts, sim.p.download()))
    assert out[0][0] == out[1][0]
    for f in out[0][1]:
        assert np.array_equal(out[0][1][f], out[1][1][f], equal_nan=out[0][1][f].dtype.kind == "f"), f


@pytest.mark.parametrize("n", [2, 33, 4097, 60_001])
def test_relaxation_forces_equal_the_stage_calls(mode, n):
    """No damped steps: the initial forces alone.  The walk's own result, the
    potential, bit for bit; pass 2 takes its lists from pass 1's radii here and
    from its own in the stage call, so its sums agree within the parity bound."""
    st = state(n)
    a, alt, bvh = engine.DeviceParticles(n), engine.DeviceParticles(n), engine.TorchBvh(n)
    a.upload(st)
    alt.count = n
    engine.relax_single_body(a, alt, bvh, None, 1.0, 0)
    b, alt2, bvh2 = engine.DeviceParticles(n), engine.DeviceParticles(n), engine.TorchBvh(n)
    b.upload(st)
    alt2.count = n
    engine.clear_stats(b)
    engine.sort_and_build_bvh(b, alt2, bvh2)
    engine.sph_pass1_neighbors(b, bvh2)
    engine.evaluate_eos(b)
    engine.gravity_barnes_hut(b, bvh2, 0.5)
    engine.sph_pass2_forces(b, bvh2)
    g, c = a.download(), b.download()
    for f in ("originalId", "phiGrav", "h", "shepardC", "divV"):
        assert np.array_equal(g[f], c[f]), f
    for f in ("accX", "accY", "accZ", "drhoDt", "duDt"):
        assert rel_rms(g[f], c[f]) < 1e-5 or np.allclose(g[f], c[f], atol=1e-12), f
