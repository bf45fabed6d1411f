"""A call that is refused leaves the fused step as it was."""
import numpy as np
import pytest

from astraea_gb300 import abi, engine, scenarios

pytestmark = pytest.mark.gpu


def scene_with_long_lists():
    st, _ = scenarios.two_granite_spheres(n_target=6000, n_impactor=2000, seed=42)
    st["h"][::500] *= 4.0                                # their lists are kept in the shared pool
    return st


def refuse_gravity_without_moments(sim):
    engine.set_far_field(1)
    with pytest.raises(abi.AstraeaError):
        engine.gravity_barnes_hut(sim.p, sim.bvh, 0.5)


def refuse_learned_gravity(sim):
    engine.ff_init(1)
    engine.set_far_field(2)
    engine.ff_configure(pairs_per_group=1 << 31)         # more pairs than 2^32
    with pytest.raises(abi.AstraeaError):
        engine.gravity_barnes_hut(sim.p, sim.bvh, 0.5)


def refuse_collect(sim):
    engine.ff_configure(pairs_per_group=1 << 31)
    with pytest.raises(abi.AstraeaError):
        engine.ff_collect(sim.p, sim.bvh, 0.5, capacity=1024)


@pytest.mark.parametrize("mode,refused", [(0, refuse_gravity_without_moments), (1, refuse_learned_gravity),
                                          (1, refuse_collect)])
def test_refused_call_between_steps_changes_nothing(mode, refused):
    st = scene_with_long_lists()
    n = len(st["posX"])
    out = []
    try:
        for disturb in (False, True):
            engine.set_far_field(mode)
            sim = engine.Simulation(n)
            sim.p.upload(st)
            sim.alt.count = n
            sim.evaluate_initial_forces(0.5)
            engine.reset_device_status()
            dts = [sim.step(5.0e-3, 0.5) for _ in range(2)]
            flags, counters = engine.read_device_status()
            assert flags == abi.DEVFLAG_NEIGHBOR_OVERFLOW and counters["fallback_walks"] == 0
            if disturb:
                try:
                    refused(sim)
                finally:
                    engine.ff_configure()
                    engine.set_far_field(mode)
            dts += [sim.step(5.0e-3, 0.5) for _ in range(2)]
            out.append((dts, sim.p.download()))
    finally:
        engine.set_far_field(0)
    assert out[0][0] == out[1][0]
    for f in out[0][1]:
        assert np.array_equal(out[0][1][f], out[1][1][f], equal_nan=out[0][1][f].dtype.kind == "f"), f
