"""Tree walks at the ends of their scratch: deep, wide trees against the walks'
stacks, and more long neighbour lists than the shared pool holds.

A scene is given by its particles' 63-bit Morton codes: coordinates are whole
numbers of 2^-17 between 0 and 2^21 - 1, so the codes are reproduced exactly and
the tree is the one the codes spell.  `spines` spells 2^bits paths of `levels`
right turns with a balanced clump of 2^leg particles beside each: every level of
it leaves a batched walk with nodes it has yet to come back to.
"""
import numpy as np
import pytest
import torch
from scipy.spatial import cKDTree

import oracle
from astraea_gb300 import abi, engine, scenarios
from conftest import rel_rms

pytestmark = pytest.mark.gpu
CELL = 2.0 ** -17


def spines(bits, levels, leg):
    out = []
    for c in range(1 << bits):
        for k in range(levels):
            path = (c << (k + 1)) | (((1 << k) - 1) << 1)
            used = bits + k + 1 + leg
            out += [((path << leg) | x) << (63 - used) for x in range(1 << leg)]
        out.append((c << (63 - bits)) | ((1 << (63 - bits)) - 1))
    return sorted(out)


def scene(codes):
    n = len(codes)
    c = np.array(codes, np.uint64)
    st = scenarios.empty_state(n)
    for k, f in enumerate(("posX", "posY", "posZ")):
        q = np.zeros(n, np.uint64)
        for b in range(21):
            q |= ((c >> np.uint64(3 * b + 2 - k)) & np.uint64(1)) << np.uint64(b)
        st[f][:] = q.astype(np.float32) * np.float32(CELL)
    st["mass"][:] = 1.0 / n
    st["h"][:] = st["h0"][:] = 1.0e-5
    st["rho"][:] = 1.0e-3
    st["materialId"][:] = 1
    st["originalId"][:] = np.arange(n, dtype=np.uint32)
    return st


def device_setup(st):
    n = len(st["posX"])
    p, alt, bvh = engine.DeviceParticles(n), engine.DeviceParticles(n), engine.TorchBvh(n)
    p.upload(st)
    alt.count = n
    return p, alt, bvh


@pytest.mark.parametrize("mode", [0, 1, 2, 3])
@pytest.mark.parametrize("bits,levels", [(5, 20), (5, 57), (0, 60)])
def test_gravity_walks_open_everything_on_deep_trees(mode, bits, levels):
    """At opening angle 0 every node is opened, whatever the tree leaves on the
    stack (a group that runs out of it takes nodes as monopoles instead): exactly
    n (n - 1) interactions.  The learned mode may still take nodes that are tiny
    against their distance; it only must not run out."""
    st = scene(spines(bits, levels, 1))
    n = len(st["posX"])
    p, alt, bvh = device_setup(st)
    try:
        engine.set_far_field(mode)
        engine.set_far_field_expansion(0, 0.3)
        if mode == 2:
            engine.ff_init(1)
            engine.ff_configure(theta_far=1.0e-6, gamma=0.3)
        engine.sort_and_build_bvh(p, alt, bvh)
        engine.reset_device_status()
        engine.gravity_barnes_hut(p, bvh, 0.0)
        flags, counters = engine.read_device_status()
    finally:
        engine.set_far_field(0)
        engine.set_far_field_expansion(16, 0.3)
        engine.ff_configure()
    assert flags == 0
    if mode != 2:
        assert counters["gravity_interactions"] == n * (n - 1)


@pytest.mark.parametrize("mode", [1, 3])
def test_gravity_small_opening_angle(mode):
    """A million particles at opening angle 0.1: no group runs out of stack, and
    the quadrupole walk's forces on sampled particles are within the error that
    angle has (below 1e-4; a group out of stack puts it above 1e-3)."""
    n = 1 << 20
    rng = np.random.default_rng(3)
    st = scenarios.empty_state(n)
    r = (rng.uniform(1.0e-6, 0.999, n) ** (-2.0 / 3.0) - 1.0) ** -0.5          # Plummer sphere
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    for k, f in enumerate(("posX", "posY", "posZ")):
        st[f][:] = r * u[:, k]
    st["mass"][:] = 1.0 / n
    st["h"][:] = st["h0"][:] = 0.01
    st["rho"][:] = 1.0e-3
    p, alt, bvh = device_setup(st)
    try:
        engine.set_far_field(mode)
        engine.sort_and_build_bvh(p, alt, bvh)
        engine.reset_device_status()
        engine.gravity_barnes_hut(p, bvh, 0.1)
        flags, counters = engine.read_device_status()
    finally:
        engine.set_far_field(0)
    g = p.download(["accX", "accY", "accZ"])
    sel = rng.choice(n, 512, replace=False).astype(np.uint32)
    ref = engine.direct_gravity_f64(p, torch.from_numpy(sel.astype(np.int64)))[0].cpu().numpy()
    a = np.stack([g[f][sel] for f in ("accX", "accY", "accZ")], 1)
    assert flags == 0
    if mode == 1:                                       # mode 3 adds its expansion's error
        assert rel_rms(a, ref) < 3e-4


@pytest.mark.parametrize("bits,levels,leg", [(1, 40, 6), (0, 24, 10), (0, 24, 12)])
def test_long_lists_of_deep_trees_are_whole(bits, levels, leg):
    """One particle reaches the whole scene: the group walk and the walk that
    fills its list in the pool open every node of a tree that leaves more on their
    stacks than those hold.  Every pair within range is visited, by count."""
    st = scene(spines(bits, levels, leg))
    n = len(st["posX"])
    big = n // 3
    st["h"][big] = st["h0"][big] = 40.0
    p, alt, bvh = device_setup(st)
    engine.sort_and_build_bvh(p, alt, bvh)
    engine.reset_device_status()
    engine.sph_pass1_neighbors(p, bvh)
    flags, counters = engine.read_device_status()
    o = oracle.Oracle(st)
    o.sort_and_build()
    o.pass1()
    g, c = p.download(), o.state()
    i = int(np.flatnonzero(g["originalId"] == big)[0])
    assert flags == abi.DEVFLAG_NEIGHBOR_OVERFLOW
    assert counters["fallback_walks"] == 0
    assert g["h"][i] == c["h"][i]
    x = np.stack([c[f] for f in ("posX", "posY", "posZ")], 1).astype(np.float64)
    assert np.linalg.norm(x - x[i], axis=1).max() < 2.0 * 40.0
    near = cKDTree(x).query_pairs(2.0e-5, output_type="ndarray")             # 2 h of all others
    pairs = n - 1 + 2 * len(near) - int(np.count_nonzero(near == i))
    assert engine.read_device_counters()["pass1_pairs"] == pairs
    for f in ("h", "shepardC", "surfFactor"):
        assert rel_rms(g[f], c[f]) < 1e-5, f


@pytest.mark.parametrize("n,every", [(2000, 33), (4000, 10)])
def test_lists_that_do_not_fit_the_pool(n, every):
    """More long lists than the pool has words for (61 of 1,999 entries; it has
    73,536) or places (all 4,000 particles, each within reach of 400 long ones; it
    has 506): no particle's sums may then depend on which of them came first, so
    all of them are walked, and runs agree bit for bit."""
    rng = np.random.default_rng(n)
    st = scenarios.empty_state(n)
    for f in ("posX", "posY", "posZ"):
        st[f][:] = rng.uniform(-1.0, 1.0, n)
    st["mass"][:] = 1.0 / n
    st["h"][:] = st["h0"][:] = 0.02
    st["h"][::every] = st["h0"][::every] = 3.0
    st["rho"][:] = rng.uniform(1.0e-3, 2.0e-3, n)
    st["originalId"][:] = np.arange(n, dtype=np.uint32)
    for f in ("velX", "velY", "velZ"):
        st[f][:] = rng.normal(size=n)
    heavy = len(range(0, n, every)) if n // every < 100 else n
    outs = []
    for _ in range(4):
        p, alt, bvh = device_setup(st)
        engine.sort_and_build_bvh(p, alt, bvh)
        engine.reset_device_status()
        engine.sph_pass1_neighbors(p, bvh)
        flags, counters = engine.read_device_status()
        assert flags == abi.DEVFLAG_NEIGHBOR_OVERFLOW
        assert counters["fallback_walks"] == heavy
        walks = counters["fallback_walks"]
        g = p.download(["h", "shepardC", "surfFactor", "divV", "curlVX"])
        outs.append((walks, g))
    for walks, g in outs[1:]:
        assert walks == outs[0][0]
        for f in g:
            assert np.array_equal(g[f], outs[0][1][f]), f
    o = oracle.Oracle(st)
    o.sort_and_build()
    o.pass1()
    c = o.state()
    for f in ("h", "shepardC", "surfFactor", "divV"):
        assert rel_rms(outs[0][1][f], c[f]) < 1e-5, f
