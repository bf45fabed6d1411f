"""GB300 kernels against the oracle, stage by stage, through the C-ABI.

Inputs are the seeded scenes of astraea_gb300.scenarios; both sides start
from the same host state.  Integer and index results (Morton codes, sorted
permutation, tree topology, dt) must be bit-identical; floating-point fields
must agree within a norm-relative RMS of 1e-5 (the parity bound for
accelerations, densities, du/dt and stress rates).
"""
import ctypes

import numpy as np
import pytest
import torch

import oracle
from astraea_gb300 import abi, engine, scenarios
from conftest import rel_rms

pytestmark = pytest.mark.gpu
TOL = 1e-5


def c1_state(n_t=12288, n_i=4096, seed=42):
    st, _ = scenarios.two_granite_spheres(n_target=n_t, n_impactor=n_i, seed=seed)
    return st


def gpu_setup(st, packed=True):
    n = len(st["posX"])
    p, alt = engine.DeviceParticles(n), engine.DeviceParticles(n)
    p.upload(st)
    alt.count = n
    bvh = engine.TorchBvh(n, packed=packed)
    return p, alt, bvh


def tnp(t, n, dtype=None):
    a = t[:n].cpu().numpy()
    return a.view(dtype) if dtype is not None else a


def report(tag, gpu, cpu, fields):
    errs = {f: rel_rms(gpu[f], cpu[f]) for f in fields}
    print("%s %s" % (tag, " ".join("%s=%.2e" % kv for kv in errs.items())))
    return errs


@pytest.mark.parametrize("packed", [True, False])
def test_sort_and_build_bit_exact(packed):
    st = c1_state()
    n = len(st["posX"])
    p, alt, bvh = gpu_setup(st, packed)
    engine.sort_and_build_bvh(p, alt, bvh)
    torch.cuda.synchronize()
    o = oracle.Oracle(st)
    o.sort_and_build()
    b = o.bvh.a
    assert np.array_equal(tnp(bvh.t["mortonCodesSorted"], n, np.uint64), b["mortonCodesSorted"])
    assert np.array_equal(tnp(bvh.t["indicesSorted"], n, np.uint32), b["indicesSorted"])
    assert np.array_equal(tnp(bvh.t["leftChild"], n - 1), b["leftChild"][: n - 1])
    assert np.array_equal(tnp(bvh.t["rightChild"], n - 1), b["rightChild"][: n - 1])
    assert np.array_equal(tnp(bvh.t["parent"], 2 * n - 1), b["parent"])
    g, c = p.download(), o.state()
    for f in abi.FIELD_NAMES:                      # 56-field permutation, bit for bit
        assert np.array_equal(g[f], c[f]), f
    for f in ("aabbMinX", "aabbMinY", "aabbMinZ", "aabbMaxX", "aabbMaxY", "aabbMaxZ", "nodeMaxH"):
        assert np.array_equal(tnp(bvh.t[f], 2 * n - 1), b[f]), f
    for f in ("nodeMass", "comX", "comY", "comZ"):  # exact moment sums vs FP32 refit
        assert rel_rms(tnp(bvh.t[f], 2 * n - 1), b[f]) < 1e-6, f
    if packed:
        assert np.array_equal(tnp(bvh.t["sceneBoundsFloat"], 6), o.bounds)
        ncm = tnp(bvh.t["nodeComMass"], 4 * (2 * n - 1)).reshape(-1, 4)
        assert rel_rms(ncm[:, 3], b["nodeMass"]) < 1e-6


def test_refit_moments_against_exact_sums():
    """Node mass and COM against exact rational sums over each node's leaves.

    The refit sums m and m x as 64-bit fixed-point integers (exact products,
    one rounding to the unit each) and divides once: every node mass is
    within one float ulp of the exact sum, every COM within one ulp plus the
    fixed-point floor (2^-40 of the scene's largest coordinate).
    """
    from fractions import Fraction
    st = c1_state()
    n = len(st["posX"])
    p, alt, bvh = gpu_setup(st, True)
    engine.sort_and_build_bvh(p, alt, bvh)
    torch.cuda.synchronize()
    g = p.download()
    lc, rc = tnp(bvh.t["leftChild"], n - 1), tnp(bvh.t["rightChild"], n - 1)
    first, last = np.zeros(n - 1, np.int64), np.zeros(n - 1, np.int64)
    order, stack = [], [0]
    while stack:
        v = stack.pop()
        order.append(v)
        stack += [int(c) for c in (lc[v], rc[v]) if c >= 0]
    for v in reversed(order):
        first[v] = ~lc[v] if lc[v] < 0 else first[lc[v]]
        last[v] = ~rc[v] if rc[v] < 0 else last[rc[v]]
    m = [Fraction(float(v)) for v in g["mass"]]
    pm, acc = [Fraction(0)], Fraction(0)
    for v in m:
        acc += v
        pm.append(acc)
    gm = tnp(bvh.t["nodeMass"], n - 1)
    X = max(float(np.abs(g[k]).max()) for k in ("posX", "posY", "posZ"))
    for f in ("nodeMass", "comX", "comY", "comZ"):
        assert np.all(np.isfinite(tnp(bvh.t[f], n - 1))), f
    for v in range(n - 1):
        s = pm[last[v] + 1] - pm[first[v]]
        assert abs(float(gm[v]) - float(s)) <= np.spacing(np.float32(float(s))), v
    for k, f in (("posX", "comX"), ("posY", "comY"), ("posZ", "comZ")):
        px, acc = [Fraction(0)], Fraction(0)
        for mi, xi in zip(m, g[k]):
            acc += mi * Fraction(float(xi))
            px.append(acc)
        gc = tnp(bvh.t[f], n - 1)
        for v in range(n - 1):
            c = float((px[last[v] + 1] - px[first[v]]) / (pm[last[v] + 1] - pm[first[v]]))
            assert abs(float(gc[v]) - c) <= np.spacing(np.float32(abs(c))) + 2.0 ** -40 * X, (f, v)


@pytest.mark.parametrize("n,end_bit", [(1, 64), (5, 64), (4096, 63), (4097, 64), (300001, 64), (1 << 20, 63)])
def test_radix_sort_pairs_stable(n, end_bit):
    rng = np.random.Generator(np.random.PCG64(n))
    hi = rng.integers(0, 7, n).astype(np.uint64) << np.uint64(min(end_bit, 63) - 3)
    keys = (hi | rng.integers(0, 1 << 20, n).astype(np.uint64) * np.uint64(rng.integers(0, 2, n) == 1)).astype(np.uint64)
    if end_bit == 64:
        keys |= (rng.integers(0, 2, n).astype(np.uint64) << np.uint64(63))
    vals = np.arange(n, dtype=np.uint32)
    kt = torch.from_numpy(keys.view(np.int64)).cuda()
    vt = torch.from_numpy(vals.view(np.int32)).cuda()
    ks, vs = engine.radix_sort_pairs(kt, vt, end_bit)
    torch.cuda.synchronize()
    mask = np.uint64((1 << end_bit) - 1) if end_bit < 64 else np.uint64(0xFFFFFFFFFFFFFFFF)
    order = np.argsort(keys & mask, kind="stable")
    assert np.array_equal(vs.cpu().numpy().view(np.uint32), vals[order])
    assert np.array_equal(ks.cpu().numpy().view(np.uint64), keys[order])


def test_pass1_eos_gravity_pass2_parity():
    st = c1_state()
    p, alt, bvh = gpu_setup(st)
    o = oracle.Oracle(st)
    engine.clear_stats(p)
    o.clear_stats()
    engine.sort_and_build_bvh(p, alt, bvh)
    o.sort_and_build()
    engine.sph_pass1_neighbors(p, bvh)
    o.pass1()
    g, c = p.download(), o.state()
    e = report("pass1", g, c, ["h", "shepardC", "surfFactor", "divV", "curlVX", "curlVY", "curlVZ"])
    assert max(e.values()) < TOL
    engine.evaluate_eos(p)
    o.eos()
    g, c = p.download(), o.state()
    e = report("eos", g, c, ["pressure", "soundSpeed", "tempK"])
    assert max(e.values()) < TOL
    # the phase is an integer output: the FP32 EOS classifies on the engine's
    # FP64 temperature wherever the FP32 one lies near a threshold, and on exact
    # float thresholds for rho and u, so every particle agrees
    assert np.array_equal(g["phaseId"], c["phaseId"])
    engine.reset_device_status()
    engine.gravity_barnes_hut(p, bvh, 0.5)
    _, counters = engine.read_device_status()
    assert counters["gravity_interactions"] == o.gravity(0.5)       # the same interaction set
    g, c = p.download(), o.state()
    e = report("gravity", g, c, ["accX", "accY", "accZ", "phiGrav"])
    assert max(e.values()) < TOL
    engine.sph_pass2_forces(p, bvh)
    o.pass2()
    g, c = p.download(), o.state()
    e = report("pass2", g, c, ["accX", "accY", "accZ", "drhoDt", "duDt", "radPowerW", "dSXX", "dSYY", "dSZZ",
                               "dSXY", "dSXZ", "dSYZ", "dDamageCbrtDt"])
    assert max(e.values()) < TOL


def test_eos_kernel_vs_reference_golden(golden_dir):
    """The FP32 EOS kernel against the reference's own FP64 EOS outputs."""
    g = np.load(golden_dir + "/eos_reference.npz")
    n = len(g["rho"])
    st = scenarios.empty_state(n)
    st["materialId"][:], st["rho"][:], st["u"][:], st["damage"][:] = g["mat"], g["rho"], g["u"], g["dmg"]
    p = engine.DeviceParticles(n)
    p.upload(st)
    engine.evaluate_eos(p)
    out = p.download(["pressure", "soundSpeed", "tempK", "phaseId"])
    for m in range(5):
        sel = g["mat"] == m
        e = {k: rel_rms(out[f][sel], g[k][sel]) for f, k in (("pressure", "P"), ("soundSpeed", "cs"), ("tempK", "T"))}
        agree = np.mean(out["phaseId"][sel] == g["phase"][sel])
        print("eos material %d %s phase-agree %.5f" % (m, " ".join("%s=%.2e" % kv for kv in e.items()), agree))
        assert max(e.values()) < TOL and agree == 1.0


def phase_threshold_states(seed=5, per=400):
    """States placed on the phase boundaries of classifyPhase (eos.cu:229-266):
    temperatures within 1e-6 relative of every threshold (u = u_cold(rho) +
    c_v T in FP64, rounded to float), u on the floats next to E_cv, rho on the
    floats next to the vapour densities."""
    rng = np.random.Generator(np.random.PCG64(seed))
    lib = oracle.load()
    cv = {0: 449.0e-6, 1: 790.0e-6, 2: 4184.0e-6, 3: 8260.0e-6, 4: 800.0e-6}
    rho0 = {0: 7.8e-3, 1: 2.68e-3, 2: 1.0e-3, 3: 0.178e-6, 4: 2.0e-3}
    temps = {0: [1811.0, 12000.0], 1: [1600.0, 12000.0], 2: [273.15, 647.0, 15000.0], 3: [10000.0],
             4: [1500.0, 12000.0]}
    ecv = {0: 8.67, 1: 18.0, 2: 2.68, 4: 18.0}
    mats, rhos, us = [], [], []
    for m, ts in temps.items():
        for t in ts:
            rho = (rho0[m] * rng.uniform(0.6, 1.6, per)).astype(np.float32)
            ucold = np.array([lib.oracle_cold_energy(m, float(r)) for r in rho])
            u = (ucold + cv[m] * t * (1.0 + rng.uniform(-1e-6, 1e-6, per))).astype(np.float32)
            mats += [m] * per; rhos += list(rho); us += list(u)
        if m in ecv:
            base = np.float32(ecv[m])
            u = np.array([np.nextafter(base, np.float32(k * np.inf)) if k else base for k in (-1, 0, 1)] * 4,
                         np.float32)
            rho = np.float32(0.8 * rho0[m]) * np.repeat(np.float32([0.5, 0.99999994, 1.0, 1.0000001]), 3)
            mats += [m] * len(u); rhos += list(rho); us += list(u)
    r322 = np.float32(322e-6)
    for r in (np.nextafter(r322, np.float32(0)), r322, np.nextafter(r322, np.float32(1))):
        ucold = lib.oracle_cold_energy(2, float(r))
        mats.append(2); rhos.append(r); us.append(np.float32(ucold + 4184.0e-6 * 700.0))
    return (np.array(mats, np.uint8), np.array(rhos, np.float32), np.array(us, np.float32))


def test_eos_phase_exact_on_phase_boundaries():
    """States on every threshold of the phase classification: the FP32 EOS
    must return the phase of the reference's FP64 EOS (restated by the
    oracle, bit-identical to it on the golden states) for each of them."""
    mat, rho, u = phase_threshold_states()
    n = len(mat)
    st = scenarios.empty_state(n)
    st["materialId"][:], st["rho"][:], st["u"][:] = mat, rho, u
    p = engine.DeviceParticles(n)
    p.upload(st)
    engine.evaluate_eos(p)
    out = p.download(["tempK", "phaseId"])
    _, _, T, ph = oracle.eos_batch(mat, rho, u, np.zeros(n, np.float32))
    bad = np.flatnonzero(out["phaseId"] != ph)
    print("phase-boundary states %d, phases per side %s" % (n, np.bincount(ph).tolist()))
    assert bad.size == 0, [(int(mat[i]), float(rho[i]), float(u[i]), float(T[i]), int(ph[i]), int(out["phaseId"][i]))
                           for i in bad[:10]]
    assert rel_rms(out["tempK"], T) < 1e-6


@pytest.mark.parametrize("theta", [0.5, 0.7])
def test_gravity_parity_and_ac3_error(theta):
    a, _ = scenarios._layered_body(2048, 6.417e-1, 0.3, 2200.0, 0, np.random.Generator(np.random.PCG64(42)))
    b, _ = scenarios._layered_body(2048, 3.3011e-1, 0.6, 3200.0, 1, np.random.Generator(np.random.PCG64(43)))
    a["posX"] -= np.float32(12.0)
    b["posX"] += np.float32(12.0)
    st = {k: np.concatenate([a[k], b[k]]) for k in a}
    st["originalId"] = np.arange(4096, dtype=np.uint32)
    p, alt, bvh = gpu_setup(st, packed=False)
    engine.sort_and_build_bvh(p, alt, bvh)
    engine.reset_device_status()
    engine.gravity_barnes_hut(p, bvh, theta)
    _, counters = engine.read_device_status()
    o = oracle.Oracle(st)
    o.sort_and_build()
    inter = o.gravity(theta)
    g, c = p.download(), o.state()
    e = report("gravity theta=%.1f" % theta, g, c, ["accX", "accY", "accZ", "phiGrav"])
    assert max(e.values()) < TOL
    # the same interaction set: the number of (particle, monopole or leaf) terms is an integer result
    assert counters["gravity_interactions"] == inter
    acc, _ = oracle.direct_gravity_f64(g, np.arange(4096))
    bh = np.stack([g["accX"], g["accY"], g["accZ"]], 1).astype(np.float64)
    err = np.linalg.norm(bh - acc, axis=1) / np.linalg.norm(acc, axis=1)
    print("AC-3 theta=%.1f median %.4f p99 %.4f" % (theta, np.median(err), np.sort(err)[int(0.99 * 4095)]))
    if theta == 0.5:
        assert np.median(err) < 0.015 and np.sort(err)[int(0.99 * 4095)] < 0.05


def test_kick_drift_dt_parity():
    st = c1_state()
    p, alt, bvh = gpu_setup(st)
    o = oracle.Oracle(st)
    engine.clear_stats(p); o.clear_stats()
    engine.sort_and_build_bvh(p, alt, bvh); o.sort_and_build()
    engine.sph_pass1_neighbors(p, bvh); o.pass1()
    engine.evaluate_eos(p); o.eos()
    engine.gravity_barnes_hut(p, bvh); o.gravity()
    engine.sph_pass2_forces(p, bvh); o.pass2()
    dt_g = engine.reduce_dt_psu(p, 0.0, 5e-3)
    dt_c, _ = o.reduce_dt(0.0, 5e-3)
    print("dt gpu %.9g oracle %.9g" % (dt_g, dt_c))
    # on identical inputs (the GPU's state after pass 2) the dt is the same float
    dt_same, _ = oracle.Oracle(p.download()).reduce_dt(0.0, 5e-3)
    assert dt_g == dt_same
    engine.leapfrog_kick_half(p, 0.5 * dt_c, True, False)
    o.kick(0.5 * dt_c)
    g, c = p.download(), o.state()
    e = report("kick", g, c, ["velX", "velY", "velZ", "rho", "u", "sXX", "sXY", "damage"])
    assert max(e.values()) < TOL
    engine.leapfrog_drift(p, dt_c, bvh)
    o.drift(dt_c)
    g, c = p.download(), o.state()
    e = report("drift", g, c, ["posX", "posY", "posZ"])
    assert max(e.values()) < 1e-6
    # each side on its own trajectory: the inputs of the dt differ by the
    # stages' ~1e-7, and so may the dt (by a float ulp)
    assert abs(dt_g - dt_c) <= 2e-7 * dt_c


def test_fused_step_matches_stagewise_and_oracle():
    st = c1_state(3072, 1024, seed=7)
    sim_f = engine.Simulation(len(st["posX"]))
    sim_s = engine.Simulation(len(st["posX"]))
    for s in (sim_f, sim_s):
        s.load_state(st)
        s.evaluate_initial_forces()
    o = oracle.Oracle(st)
    o.initial_forces()
    for k in range(4):
        dt_f = sim_f.step(5e-3)
        dt_s = sim_s.step_stagewise(5e-3)
        dt_o = o.step(5e-3)
        print("step %d dt fused %.9g stagewise %.9g oracle %.9g" % (k, dt_f, dt_s, dt_o))
        assert abs(dt_f - dt_s) <= 1e-6 * dt_s and abs(dt_f - dt_o) <= 1e-5 * dt_o
    gf, gs, c = sim_f.state(), sim_s.state(), o.state()
    fields = ["posX", "posY", "posZ", "velX", "velY", "velZ", "rho", "u", "h", "accX", "accY", "accZ", "duDt",
              "drhoDt", "pressure", "phiGrav"]
    ef = report("fused-vs-oracle", gf, c, fields)
    es = report("stagewise-vs-oracle", gs, c, fields)
    report("fused-vs-stagewise", gf, gs, fields)
    assert max(ef.values()) < 1e-4 and max(es.values()) < 1e-4
    assert np.array_equal(gf["originalId"], gs["originalId"])


@pytest.mark.parametrize("n", [1, 2, 33])
def test_small_counts(n):
    st = c1_state()
    small = {k: v[:n].copy() for k, v in st.items()}
    small["originalId"] = np.arange(n, dtype=np.uint32)
    p, alt, bvh = gpu_setup(small)
    o = oracle.Oracle(small)
    engine.clear_stats(p); o.clear_stats()
    engine.sort_and_build_bvh(p, alt, bvh); o.sort_and_build()
    engine.sph_pass1_neighbors(p, bvh); o.pass1()
    engine.evaluate_eos(p); o.eos()
    engine.gravity_barnes_hut(p, bvh); o.gravity()
    engine.sph_pass2_forces(p, bvh); o.pass2()
    g, c = p.download(), o.state()
    assert np.array_equal(g["originalId"], c["originalId"])
    for f in ("h", "surfFactor", "accX", "phiGrav", "duDt"):
        assert rel_rms(g[f], c[f]) < TOL or np.allclose(g[f], c[f], atol=1e-12), f


def test_coincident_particles_tie_break():
    n = 500
    st = c1_state()
    small = {k: v[:n].copy() for k, v in st.items()}
    small["posX"][:250] = small["posX"][0]
    small["posY"][:250] = small["posY"][0]
    small["posZ"][:250] = small["posZ"][0]
    small["originalId"] = np.arange(n, dtype=np.uint32)
    p, alt, bvh = gpu_setup(small)
    engine.sort_and_build_bvh(p, alt, bvh)
    o = oracle.Oracle(small)
    o.sort_and_build()
    torch.cuda.synchronize()
    assert np.array_equal(tnp(bvh.t["indicesSorted"], n, np.uint32), o.bvh.a["indicesSorted"])
    assert np.array_equal(tnp(bvh.t["leftChild"], n - 1), o.bvh.a["leftChild"][: n - 1])


def test_lookback_wait_gives_up_and_reports():
    engine.reset_device_status()
    out = ctypes.c_uint32(0)
    rc = abi.load_library().astraea_gb300_debug_lookback_probe(1000, ctypes.byref(out))
    assert rc == 4 and out.value == 2
    flags, _ = engine.read_device_status()
    assert flags & abi.DEVFLAG_LOOKBACK_TIMEOUT
    # the context stays usable; the blocking dt call reports the timeout
    st = c1_state(64, 32)
    p, alt, bvh = gpu_setup(st)
    with pytest.raises(abi.AstraeaError) as ei:
        engine.reduce_dt_psu(p, 0.0, 1e-3)
    assert ei.value.status == 4
    engine.reset_device_status()
    assert engine.reduce_dt_psu(p, 0.0, 1e-3) > 0.0


def test_capacity_error_like_engine():
    st = c1_state(64, 32)
    p, alt, bvh = gpu_setup(st)
    small = engine.TorchBvh(16)
    with pytest.raises(abi.AstraeaError) as ei:
        engine.sort_and_build_bvh(p, alt, small)
    assert ei.value.status == 2


def test_c1_twenty_steps_track_oracle():
    """The small benchmark configuration end to end: two granite spheres,
    12,288 + 4,096 particles, 20 fused KDK steps against 20 oracle steps
    (trajectory level: FP32 summation order and the race-free drift
    both enter, so the bound is wider than one step's), with momentum
    conserved on both."""
    st = c1_state()
    n = len(st["posX"])
    sim = engine.Simulation(n)
    sim.load_state(st)
    sim.evaluate_initial_forces()
    o = oracle.Oracle(st)
    o.initial_forces()
    for k in range(20):
        dt_g = sim.step(5e-3)
        dt_o = o.step(5e-3)
        assert abs(dt_g - dt_o) <= 1e-4 * dt_o, (k, dt_g, dt_o)
    g, c = sim.state(), o.state()
    assert np.array_equal(g["originalId"], c["originalId"])
    e = report("c1-20-steps", g, c, ["posX", "posY", "posZ", "velX", "velY", "velZ", "rho", "u", "h", "pressure"])
    assert max(e.values()) < 5e-4, e        # measured 7.2e-5 (h) on GB300
    for s in (g, c):
        m = s["mass"].astype(np.float64)
        mom = [np.sum(m * s[k].astype(np.float64)) for k in ("velX", "velY", "velZ")]
        scale = np.sum(m * np.sqrt(sum(s[k].astype(np.float64) ** 2 for k in ("velX", "velY", "velZ"))))
        assert max(abs(x) for x in mom) < 1e-4 * scale


@pytest.mark.gpu
@pytest.mark.parametrize("n", [31, 32, 33, 511, 1025, 16 * 1024, 16 * 1024 + 1, 50_001, 114_687, 114_688, 114_689, 4096 * 65 + 1])
@pytest.mark.parametrize("end_bit", [7, 40, 64])
def test_radix_sort_one_launch_and_tiled_sizes(n, end_bit):
    """Sizes around the one-launch sort's ends (32 and 114,688 keys), its rounds
    of 1,024 keys a block, and a tiled sort whose look-back crosses several
    windows; keys with few distinct digits, so runs of equal keys span blocks."""
    from astraea_gb300 import engine
    rng = np.random.default_rng(n + end_bit)
    keys = rng.integers(0, 2 ** 63, n, dtype=np.uint64) & np.uint64(0x8300000000050103 if n % 2 else 2 ** 64 - 1)
    vals = np.arange(n, dtype=np.int32)
    ks, vs = engine.radix_sort_pairs(torch.from_numpy(keys.view(np.int64)).cuda(), torch.from_numpy(vals).cuda(), end_bit)
    bits = min(64, (end_bit + 7) // 8 * 8)                      # whole digits of 8 bits
    part = keys if bits == 64 else keys & np.uint64(2 ** bits - 1)
    order = np.argsort(part, kind="stable")
    assert np.array_equal(vs.cpu().numpy(), vals[order])
    assert np.array_equal(ks.cpu().numpy().view(np.uint64), keys[order])


@pytest.mark.gpu
@pytest.mark.parametrize("n", [32, 700, 5000, 32_768, 40_001, 65_536, 65_537])
@pytest.mark.parametrize("far", [0.0, 60.0, 2000.0, 1.0e6])
def test_morton_sort_with_far_outliers(n, far):
    """A cloud beside a particle `far` cloud sizes away: the code's cells grow
    against the cloud, so its top digits tie in short runs, in runs across the
    blocks of the one-launch sort, and all over; some particles coincide.  The
    order is the stable order of the 63-bit codes."""
    rng = np.random.default_rng(n)
    st = scenarios.empty_state(n)
    for f in ("posX", "posY", "posZ"):
        st[f][:] = rng.normal(size=n) * 0.3
        st[f][n // 2: n // 2 + n // 16] = st[f][n // 2]
    st["posX"][n - 1] += far
    st["mass"][:] = 1.0 / n
    st["h"][:] = st["h0"][:] = 0.02
    st["rho"][:] = 1.0e-3
    st["originalId"][:] = np.arange(n, dtype=np.uint32)
    code = np.zeros(n, np.uint64)
    for k, f in enumerate(("posX", "posY", "posZ")):
        lo, hi = st[f].min(), st[f].max()
        inv = np.float32(2097151.0) / np.float32(hi - lo)
        q = np.clip((st[f] - lo) * inv, np.float32(0), np.float32(2097151)).astype(np.uint64)
        for b in range(21):
            code |= ((q >> np.uint64(b)) & np.uint64(1)) << np.uint64(3 * b + 2 - k)
    order = np.argsort(code, kind="stable")
    p, alt, bvh = engine.DeviceParticles(n), engine.DeviceParticles(n), engine.TorchBvh(n)
    p.upload(st)
    alt.count = n
    engine.sort_and_build_bvh(p, alt, bvh)
    assert np.array_equal(p.download(["originalId"])["originalId"], order)
    assert np.array_equal(bvh.t["mortonCodesSorted"].cpu().numpy().view(np.uint64), code[order])
    assert np.array_equal(bvh.t["indicesSorted"].cpu().numpy(), order)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [3, 31, 63, 97, 1000, 4111])
@pytest.mark.parametrize("shape", ["cloud", "line", "shell", "far", "clumps"])
def test_gravity_walk_sets_at_edges(n, shape):
    """Each group's interaction count equals the oracle's (short last groups,
    flat and hollow groups whose box, octant planes and extreme members bound
    them badly, groups far from the origin, coincident members), for angles on
    both sides of the inside-box rule and at 0; the forces agree with it."""
    rng = np.random.default_rng(n)
    x = rng.normal(size=(n, 3))
    if shape == "line":
        x[:, 1:] *= 1.0e-4
    elif shape == "shell":
        x /= np.linalg.norm(x, axis=1)[:, None]
    elif shape == "far":
        x = x * 0.05 + np.array([40.0, -30.0, 20.0])
    elif shape == "clumps":
        x = x[rng.integers(0, max(n // 8, 1), n)] + rng.normal(size=(n, 3)) * rng.choice([0.0, 1.0e-3], n)[:, None]
    st = scenarios.empty_state(n)
    for k, f in enumerate(("posX", "posY", "posZ")):
        st[f][:] = x[:, k]
    st["mass"][:] = rng.uniform(0.5, 1.5, n) / n
    st["h"][:] = st["h0"][:] = rng.uniform(0.01, 0.03, n)
    st["rho"][:] = 1.0e-3
    st["originalId"][:] = np.arange(n, dtype=np.uint32)
    p, alt, bvh = gpu_setup(st)
    o = oracle.Oracle(st)
    engine.set_node_rounding(1)
    try:
        engine.sort_and_build_bvh(p, alt, bvh)
    finally:
        engine.set_node_rounding(0)
    o.sort_and_build()
    for theta in (0.0, 0.3, 0.5, 0.6, 1.0):
        assert np.array_equal(engine.gravity_group_counts(p, bvh, theta), o.gravity_group_counts(theta)), theta
        engine.gravity_barnes_hut(p, bvh, theta)
        o.gravity(theta)
        g, c = p.download(), o.state()
        for f in ("accX", "accY", "accZ", "phiGrav"):
            assert rel_rms(g[f], c[f]) < TOL, (theta, f)


@pytest.mark.parametrize("n", [(1 << 20) + 1, (1 << 20) + 63])
@pytest.mark.parametrize("theta", [0.3, 0.5, 0.7])
def test_gravity_walk_of_large_scenes(n, theta):
    """The monopole walk adds its terms in another order than the general one:
    it takes the interactions of that walk, which the counting call runs, and the
    forces agree within the parity bound (they differ in rounding only)."""
    rng = np.random.default_rng(n)
    st = scenarios.empty_state(n)
    for f in ("posX", "posY", "posZ"):
        st[f][:] = rng.normal(size=n)
    st["mass"][:] = rng.uniform(0.5, 1.5, n) / n
    st["h"][:] = st["h0"][:] = rng.uniform(0.01, 0.03, n)
    st["rho"][:] = 1.0e-3
    st["originalId"][:] = np.arange(n, dtype=np.uint32)
    p, alt, bvh = gpu_setup(st)
    engine.sort_and_build_bvh(p, alt, bvh)
    engine.reset_device_status()
    engine.gravity_barnes_hut(p, bvh, theta)
    flags, counters = engine.read_device_status()
    a = p.download(["accX", "accY", "accZ", "phiGrav"])
    counts = engine.gravity_group_counts(p, bvh, theta)
    b = p.download(["accX", "accY", "accZ", "phiGrav"])
    assert flags == 0 and counters["gravity_interactions"] == int(counts.astype(np.int64).sum())
    for f in a:
        assert rel_rms(a[f], b[f]) < TOL, f


@pytest.mark.parametrize("n", [45, 19_456, 19_457, 29_185, 38_913, 58_369])
def test_sph_passes_lanes_and_long_lists(n):
    """Sizes on both sides of each change in the lanes per particle, with every
    1500th particle's h so large that its neighbours exceed a list (they are
    kept in the shared pool): pass 1, pass 2 and the drift against the oracle,
    within the parity bound."""
    st = c1_state(n_t=n - n // 4, n_i=n // 4)
    st["h"][::1500] *= 4.0
    p, alt, bvh = gpu_setup(st)
    o = oracle.Oracle(st)
    engine.reset_device_status()
    engine.clear_stats(p)
    o.clear_stats()
    engine.sort_and_build_bvh(p, alt, bvh)
    o.sort_and_build()
    engine.sph_pass1_neighbors(p, bvh)
    o.pass1()
    engine.evaluate_eos(p)
    o.eos()
    engine.sph_pass2_forces(p, bvh)
    o.pass2()
    g, c = p.download(), o.state()
    for f in ("h", "shepardC", "surfFactor", "divV", "curlVX", "accX", "accY", "accZ", "drhoDt", "duDt", "dSXX", "dSXY"):
        assert rel_rms(g[f], c[f]) < TOL or np.allclose(g[f], c[f], atol=1e-12), (f, rel_rms(g[f], c[f]))
    p.upload(c)
    engine.leapfrog_drift(p, 1.0e-2, bvh)
    o.drift(1.0e-2)
    g, d = p.download(), o.state()
    for f in ("posX", "posY", "posZ"):
        moved = d[f].astype(np.float64) - c[f]
        ulp = np.spacing(np.abs(c[f]).max())             # positions are stored in FP32
        assert np.max(np.abs((g[f].astype(np.float64) - c[f]) - moved)) <= ulp + 1e-5 * np.abs(moved).max(), f
    flags, counters = engine.read_device_status()
    assert counters["fallback_walks"] == 0
    assert bool(flags & abi.DEVFLAG_NEIGHBOR_OVERFLOW) == (n > 1000)


@pytest.mark.parametrize("n", [2, 33, 4097, 40_001, (1 << 19) + 1])
def test_step_walks_side_by_side_change_nothing(n):
    """The step runs the gravity walk beside the neighbour lists, pass 1 and the
    EOS; with stage timing on it runs them one after the other.  Same bits."""
    m = max(n, 64)
    st = {k: v[:n].copy() for k, v in c1_state(n_t=m - m // 4, n_i=m // 4).items()}
    st["originalId"] = np.arange(n, dtype=np.uint32)
    out = []
    for timed in (False, True):
        sim = engine.Simulation(n)
        sim.p.upload(st)
        sim.alt.count = n
        sim.evaluate_initial_forces(0.5)
        engine.set_stage_timing(timed)
        try:
            dts = [sim.step(5.0e-3, 0.5) for _ in range(3)]
        finally:
            engine.set_stage_timing(False)
        out.append((dts, sim.p.download()))
    assert out[0][0] == out[1][0]
    for f in out[0][1]:
        assert np.array_equal(out[0][1][f], out[1][1][f], equal_nan=out[0][1][f].dtype.kind == "f"), f


@pytest.mark.parametrize("n", [2, 255, 257, 513, 77_824, 77_825, 131_072, 131_073])
def test_permutation_and_refit_at_block_counts(n):
    """Both sides of the sizes where the permutation and the node search share
    their blocks and where the refit's scan and table share one launch: order,
    topology and boxes bit for bit, exact moment sums within 1e-6 of the FP32
    refit as in test_sort_and_build_bit_exact."""
    m = max(n, 64)
    st = {k: v[:n].copy() for k, v in c1_state(n_t=m - m // 4, n_i=m // 4).items()}
    st["originalId"] = np.arange(n, dtype=np.uint32)
    p, alt, bvh = gpu_setup(st)
    engine.sort_and_build_bvh(p, alt, bvh)
    torch.cuda.synchronize()
    o = oracle.Oracle(st)
    o.sort_and_build()
    b = o.bvh.a
    assert np.array_equal(tnp(bvh.t["indicesSorted"], n, np.uint32), b["indicesSorted"])
    assert np.array_equal(tnp(bvh.t["leftChild"], n - 1), b["leftChild"][: n - 1])
    assert np.array_equal(tnp(bvh.t["parent"], 2 * n - 1), b["parent"])
    for f in ("aabbMinX", "aabbMinY", "aabbMinZ", "aabbMaxX", "aabbMaxY", "aabbMaxZ", "nodeMaxH"):
        assert np.array_equal(tnp(bvh.t[f], 2 * n - 1), b[f]), f
    for f in ("nodeMass", "comX", "comY", "comZ"):
        assert rel_rms(tnp(bvh.t[f], 2 * n - 1), b[f]) < 1e-6, f


def test_neighbour_lists_do_not_depend_on_the_build_size():
    """The build above 2^19 particles has other registers: pass 1 of particles
    whose surroundings are the same gives the same bits on both sides of it."""
    n = (1 << 19) + 1
    st = c1_state(n_t=n - n // 4, n_i=n // 4)
    out = []
    for m in (n, n - 1):
        s = {k: v[:m].copy() for k, v in st.items()}
        p, alt, bvh = gpu_setup(s)
        engine.sort_and_build_bvh(p, alt, bvh)
        engine.sph_pass1_neighbors(p, bvh)
        g = p.download(["posX", "posY", "posZ", "h", "shepardC", "divV", "originalId"])
        out.append({f: v[np.argsort(g["originalId"])] for f, v in g.items()})
    a, b = out
    x = np.stack([a[f] for f in ("posX", "posY", "posZ")], 1).astype(np.float64)
    far = np.linalg.norm(x[: n - 1] - x[n - 1], axis=1) > 8.0 * a["h"].max()
    assert far.sum() > n // 2
    assert np.array_equal(a["h"][: n - 1][far], b["h"][far])
    for f in ("shepardC", "divV"):                  # list order may differ where groups shift by one
        assert rel_rms(a[f][: n - 1][far], b[f][far]) < TOL, f
