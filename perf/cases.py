"""The work that users of astraea_gb300 have it do, as measurable cases.

A case is one call (or the few calls that a program always makes together)
through the public entry points of astraea_gb300.engine:

  step       the fused step (engine.step): what a simulation spends its life in
  headless   the loop body of the headless runner: a step that is waited for
             and the per-step telemetry reduction of its conservation check
  stagewise  the same step as the engine's own sequence of stage calls, the
             drop-in path of the C-ABI
  build      sort + permutation + tree of a scene in load order
  pass1, pass2   one SPH stage call (its neighbour search included)
  gravity    one gravity stage call, in a far-field mode
  publish    what a server does per frame: telemetry, then the PCLS frame
  relax      damped steps of one loaded body

Scenes are made on the GPU from the seed: two bodies on lattices (uniform, or
an iron core under a granite mantle), a gas giant with a hydrogen envelope, a
Plummer sphere, or a single layered body.  They carry what a running
simulation's state carries (shear, noise, stresses, damage, temperatures,
surface tracers), not the smooth state of time zero.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "astraea-impact-sim_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from astraea_gb300 import abi, engine, scenarios  # noqa: E402

MAX_DT = 5.0e-3          # the runner's default bound, 5 s
G_PSU = scenarios.G_PSU
EXACT_PAIRS_N = 300_000  # above this the 64-bit pair sums take too long


def listed():
    return [
        # the smallest configuration of the benchmark: two granite spheres, launches and latency count
        dict(name="step_16k", kind="step", scene="spheres", n=16384, theta=0.5),
        # the benchmark's default workload
        dict(name="step_1m", kind="step", scene="impact", n=1_000_000, theta=0.5),
        # the largest configuration: gas-giant core impact
        dict(name="step_16m", kind="step", scene="gas", n=16_000_000, theta=0.5),
        # the headless runner's conservation check at its default 30,000 particles (odd count)
        dict(name="headless_30k", kind="headless", scene="impact", n=30_001, theta=0.5),
        # the presets' default size through the engine's own call sequence (ragged count)
        dict(name="stagewise_100k", kind="stagewise", scene="impact", n=100_003, theta=0.5),
        # loading a scene: particles arrive in builder order, all 56 fields move
        dict(name="build_1m", kind="build", scene="impact", n=1_000_000),
        # one SPH stage each, at a middle size with a ragged last group
        dict(name="pass1_200k", kind="pass1", scene="impact", n=200_017),
        dict(name="pass2_200k", kind="pass2", scene="impact", n=200_017),
        # plain gravity at the middle of the batched ensemble's sizes
        dict(name="gravity_60k", kind="gravity", scene="spheres", n=60_013, theta=0.5, mode=0),
        # the gravity-only benchmark with its equal-error option, the quadrupole at a larger angle
        dict(name="gravity_plummer_4m", kind="gravity", scene="plummer", n=4_000_000, theta=0.7, mode=1),
        # one frame of a served simulation
        dict(name="publish_1m", kind="publish", scene="impact", n=1_000_000),
        # relaxing one body of a preset (the presets run 80 such steps, all alike)
        dict(name="relax_25k", kind="relax", scene="body", n=25_000, steps=4),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["step", "step", "headless", "stagewise", "build", "pass1", "pass2", "gravity", "gravity",
                       "publish", "relax"])
    if kind == "step":
        scene = rng.choice(["spheres", "impact", "impact", "gas"])
        return dict(kind=kind, scene=scene, n=size(8192, 8_000_000 if scene == "gas" else 4_000_000),
                    theta=rng.choice([0.5, 0.5, 0.6]))
    if kind == "gravity":
        scene = rng.choice(["spheres", "impact", "plummer"])
        mode = rng.choice([0, 0, 1, 3])
        return dict(kind=kind, scene=scene, n=size(8192, 4_000_000), mode=mode,
                    theta=rng.choice([0.5, 0.7]) if mode == 0 else rng.choice([0.6, 0.7, 0.75]))
    if kind == "relax":
        return dict(kind=kind, scene="body", n=size(2000, 120_000), steps=rng.randint(2, 6))
    hi = {"headless": 500_000, "stagewise": 1_000_000, "build": 4_000_000, "pass1": 1_000_000, "pass2": 1_000_000,
          "publish": 4_000_000}[kind]
    case = dict(kind=kind, scene=rng.choice(["spheres", "impact"]), n=size(8192, hi))
    if kind in ("headless", "stagewise"):
        case["theta"] = 0.5
    return case


# ------------------------------------------------------------------ scenes
@functools.lru_cache(maxsize=None)
def _profile(mass_psu, core_frac):
    """Hydrostatic profile of a layered body (numpy, SI): it depends on no seed."""
    return scenarios.hydrostatic_profile(mass_psu, core_frac, samples=1000)


def _interp(x, xp, fp):
    """np.interp for tensors (xp increasing)."""
    k = torch.searchsorted(xp, x).clamp_(1, len(xp) - 1)
    x0, x1 = xp[k - 1], xp[k]
    t = ((x - x0) / (x1 - x0).clamp_min(1e-300)).clamp_(0.0, 1.0)
    return fp[k - 1] + t * (fp[k] - fp[k - 1])


def _ball(n, gen):
    """n points of a jittered cubic lattice filling the unit ball, from the centre outwards."""
    s = (4.0 / 3.0 * math.pi / n) ** (1.0 / 3.0)
    k = int(math.ceil(1.0 / s)) + 2
    ax = (torch.arange(-k, k + 1, device="cuda", dtype=torch.float64) + 0.5) * s
    r2 = ax[:, None, None] ** 2 + ax[None, :, None] ** 2 + ax[None, None, :] ** 2
    idx = torch.nonzero(r2.reshape(-1) < (1.0 + 3.0 * s) ** 2).reshape(-1)
    idx = idx[torch.argsort(r2.reshape(-1)[idx], stable=True)[:n]]
    m = 2 * k + 1
    pts = torch.stack([ax[idx // (m * m)], ax[(idx // m) % m], ax[idx % m]], 1)
    pts /= pts.norm(dim=1).max() + 0.5 * s
    return pts + (torch.rand(n, 3, device="cuda", dtype=torch.float64, generator=gen) - 0.5) * (0.2 * s)


def _blank(n):
    out = {}
    for name, dt in abi.FIELDS:
        out[name] = torch.zeros(n, device="cuda", dtype=torch.uint8 if dt == np.uint8 else
                                torch.int32 if dt in (np.uint32, np.int32) else torch.float64)
    out["tracerIndex"].fill_(-1)
    out["shepardC"].fill_(1.0)
    return out


def _put_points(st, pts):
    st["posX"], st["posY"], st["posZ"] = (pts[:, k].clone() for k in range(3))


def _uniform(n, radius, mat, body_id, gen):
    rho = scenarios._MAT[mat]["rho0"] / 1.0e6
    st = _blank(n)
    _put_points(st, _ball(n, gen) * radius)
    st["mass"].fill_(rho * 4.0 / 3.0 * math.pi * radius ** 3 / n)
    st["rho"].fill_(rho)
    st["u"].fill_(scenarios._MAT[mat]["cv"] * 300.0 / 1.0e6)
    st["tempK"].fill_(300.0)
    st["materialId"].fill_(mat)
    st["bodyId"].fill_(body_id)
    return st, radius


def _cold(mat, rho_si):
    """Cold compression energy of the Tillotson curve, J/kg."""
    c = scenarios._MAT[mat]
    eta = (rho_si / c["rho0"]).clamp_min(1.0)
    mu, le = eta - 1.0, torch.log(eta)
    return (c["A"] * (le - mu / eta) + c["B"] * (mu * (2.0 + mu) / eta - 2.0 * le)) / c["rho0"]


def _layered(n, mass_psu, core_frac, body_id, gen):
    """Iron core (core_frac of the mass) under a granite mantle, equal-mass particles on a hydrostatic profile."""
    rs, ms, rhos, _ = (torch.from_numpy(np.asarray(v, np.float64)).cuda() for v in _profile(mass_psu, core_frac))
    pts = _ball(n, gen)
    r0 = pts.norm(dim=1).clamp_min(1e-12)
    frac = r0.clamp(max=1.0) ** 3
    r = _interp(frac * ms[-1], ms, rs)
    rho = _interp(r, rs, rhos)
    iron = frac < core_frac
    st = _blank(n)
    _put_points(st, pts * (r / r0 / 1.0e6)[:, None])
    st["mass"].fill_(mass_psu / n)
    st["rho"] = rho / 1.0e6
    cv = torch.where(iron, scenarios._MAT[0]["cv"], scenarios._MAT[1]["cv"])
    st["u"] = (torch.where(iron, _cold(0, rho), _cold(1, rho)) + cv * 2000.0) / 1.0e6
    st["tempK"].fill_(2000.0)
    st["materialId"] = torch.where(iron, 0, 1).to(torch.uint8)
    st["bodyId"].fill_(body_id)
    return st, float(rs[-1]) / 1.0e6


def _envelope(n, mass_psu, r_in, r_out, gen):
    """Hydrogen-helium shell r_in..r_out with the n = 1 polytrope's density."""
    rs = torch.linspace(r_in, r_out, 4000, device="cuda", dtype=torch.float64)
    shape = torch.sin(math.pi * rs / r_out) / (math.pi * rs / r_out)
    dm = 4.0 * math.pi * rs * rs * shape
    ms = torch.cat([torch.zeros_like(rs[:1]), torch.cumsum(0.5 * (dm[1:] + dm[:-1]) * (rs[1] - rs[0]), 0)])
    pts = _ball(n, gen)
    r0 = pts.norm(dim=1).clamp_min(1e-12)
    r = _interp(r0.clamp(max=1.0) ** 3 * ms[-1], ms, rs)
    st = _blank(n)
    _put_points(st, pts * (r / r0)[:, None])
    st["mass"].fill_(mass_psu / n)
    st["rho"] = (mass_psu / ms[-1] * _interp(r, rs, shape)).clamp_min(1.0e-9)
    st["u"].fill_(8260.0 * 2000.0 / 1.0e6)
    st["tempK"].fill_(2000.0)
    st["epsFail"].fill_(1.0)
    st["materialId"].fill_(3)
    return st, r_out


def _join(parts):
    return {f: torch.cat([p[f] for p in parts]) for f in parts[0]}


def _approach(t, r_t, i, r_i, v_ratio, angle_deg):
    """The impactor close to contact, on a path of the given impact angle."""
    rc = r_t + r_i
    vc = v_ratio * math.sqrt(2.0 * G_PSU * float(t["mass"].sum() + i["mass"].sum()) / rc)
    a = math.radians(angle_deg)
    i["posX"] += 1.03 * rc * math.cos(a)
    i["posZ"] += 1.03 * rc * math.sin(a)
    i["velX"] -= vc
    return _join([t, i])


def _scene(case, seed):
    """The scene's fields (torch, on the GPU; floating ones rounded to 32 bits) in load order."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    n, scene = case["n"], case["scene"]
    earth = scenarios.M_EARTH_PSU
    if scene == "plummer":
        st = _blank(n)
        x = torch.rand(n, device="cuda", dtype=torch.float64, generator=gen).clamp(1e-10, 1.0 - 1e-10)
        r = (1.0 / torch.sqrt(x ** (-2.0 / 3.0) - 1.0)).clamp(max=100.0)
        v = torch.randn(n, 3, device="cuda", dtype=torch.float64, generator=gen)
        _put_points(st, v * (r / v.norm(dim=1).clamp_min(1e-12))[:, None])
        st["mass"].fill_((1.0 / n) / G_PSU)
        st["rho"].fill_(1.0e-3)
        st["h0"].fill_(1.0e-3 / 0.8)
        st["materialId"].fill_(1)
    elif scene == "spheres":
        n_i = n // 4
        st = _approach(*_uniform(n - n_i, 1.0, 1, 0, gen), *_uniform(n_i, 0.6, 1, 1, gen), 1.1, 45.0)
    elif scene == "impact":
        n_i = n // 5
        st = _approach(*_layered(n - n_i, earth, 0.3, 0, gen), *_layered(n_i, 0.1 * earth, 0.3, 1, gen), 1.1, 45.0)
    elif scene == "gas":
        n_i = n // 8
        n_core = max(1024, (n - n_i) // 10)
        core, r_core = _layered(n_core, earth, 0.33, 0, gen)
        env, r_env = _envelope(n - n_i - n_core, 9.0 * earth, r_core, 4.0 * r_core, gen)
        r_i = (3.0 * earth / (4.0 * math.pi * 2.0e-3)) ** (1.0 / 3.0)
        st = _approach(_join([core, env]), r_env, *_uniform(n_i, r_i, 4, 1, gen), 2.0, 30.0)
    else:
        st, _ = _layered(n, earth, 0.3, 0, gen)
    del gen
    return _lived_in(st, case, seed)


def _lived_in(st, case, seed):
    """What some hundred steps leave in a state: shear and noise in the velocities, smoothing lengths off their
    nominal value, stresses, damage, temperatures, and every derived field; surface tracers on body 0."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed) + 7919)
    n = case["n"]

    def rnd():
        return torch.rand(n, device="cuda", dtype=torch.float64, generator=gen)

    x, y, z = st["posX"], st["posY"], st["posZ"]
    if case["scene"] != "plummer":
        st["h0"] = 1.2 * (st["mass"] / st["rho"]) ** (1.0 / 3.0)
    st["h"] = st["h0"] * (0.98 + 0.04 * rnd())
    for k, (f, a, b) in enumerate((("velX", y, z), ("velY", z, x), ("velZ", x, y))):
        st[f] = st[f] + 0.3 * torch.sin(1.3 * a + 0.4 * k) * torch.cos(0.9 * b) + 0.02 * (rnd() - 0.5) + 0.05 * (k + 1)
    st["rho"] = st["rho"] * (0.99 + 0.02 * rnd())
    st["u"] = st["u"] * (1.0 + 0.05 * rnd())
    st["tempK"] = st["tempK"] * (0.7 + 1.2 * rnd())
    solid = (st["materialId"] != 3).to(torch.float64)
    diag = [2.0e-4 * solid * (rnd() - 0.5) for _ in range(3)]
    mean = (diag[0] + diag[1] + diag[2]) / 3.0
    for f, v in zip(("sXX", "sYY", "sZZ"), diag):
        st[f] = v - mean
    for f in ("sXY", "sXZ", "sYZ"):
        st[f] = 1.0e-4 * solid * (rnd() - 0.5)
    d = ((rnd() - 0.6) * 2.5).clamp(0.0, 1.0) * solid
    st["damageCbrt"], st["damage"] = d, d ** 3
    eps = torch.where(st["materialId"] == 0, 1.0e-3, 1.0e-4)
    st["epsFail"] = torch.where(st["materialId"] == 3, 1.0, eps * (1.0 + 2.0 * rnd()))
    st["originalId"] = torch.arange(n, device="cuda", dtype=torch.int32)
    # derived fields: a step recomputes them, single stages read them
    rad = torch.sqrt(x * x + y * y + z * z)
    st["pressure"] = 0.05 * torch.exp(-0.3 * rad) * rnd() - 2.0e-3 * rnd()
    st["soundSpeed"] = 3.0 + 5.0 * rnd()
    st["phaseId"] = (rnd() > 0.8).to(torch.uint8)
    for f in ("divV", "curlVX", "curlVY", "curlVZ"):
        st[f] = 0.4 * (rnd() - 0.5)
    st["shepardC"] = 0.75 + 0.3 * rnd()
    st["surfFactor"] = (1.4 * rnd() - 0.4).clamp(0.0, 1.0)
    st["radPowerW"] = 1.0e15 * rnd()
    st["phiGrav"] = -G_PSU * 6.0 / (rad + 1.0) * (1.0 + 1.0e-3 * rnd())
    for f in ("accX", "accY", "accZ", "drhoDt", "duDt", "dSXX", "dSYY", "dSZZ", "dSXY", "dSXZ", "dSYZ"):
        st[f] = 1.0e-2 * (rnd() - 0.5)
    tracers = min(1536, n // 8)                     # 6 x 16 x 16, the presets' grid
    first = int((st["bodyId"] == 0).sum()) - tracers   # the last particles of body 0 are its surface
    t = slice(first, first + tracers)
    st["tracerIndex"][t] = torch.arange(tracers, device="cuda", dtype=torch.int32)
    r = rad[t].clamp_min(1e-9)
    st["tracerRestRadiusPsu"][t] = r
    for f, c in (("tracerRestNormalX", x), ("tracerRestNormalY", y), ("tracerRestNormalZ", z)):
        st[f][t] = c[t] / r
    st["tracerIsOcean"][t] = (rnd()[t] > 0.5).to(torch.uint8)
    return {f: (v.to(torch.float32) if v.is_floating_point() else v) for f, v in st.items()}


def _fill(p, st, n):
    for f, v in st.items():
        p.arrays[f][:n].copy_(v)
    p.count = n


# ------------------------------------------------------------------- cases
class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case, s.kind, n = case, case["kind"], case["n"]
    s.theta = float(case.get("theta", 0.5))
    engine.set_far_field(int(case.get("mode", 0)))
    st = _scene(case, seed)
    if s.kind in ("step", "headless", "stagewise", "relax"):
        s.sim = engine.Simulation(n)
        _fill(s.sim.p, st, n)
        s.sim.alt.count = n
        s.dt = torch.zeros(1, dtype=torch.float32).pin_memory()
        if s.kind == "relax":
            s.anchor = st["tempK"].to(torch.float64)
            s.radius = float(torch.sqrt(st["posX"] ** 2 + st["posY"] ** 2 + st["posZ"] ** 2).max())
        else:
            s.sim.evaluate_initial_forces(s.theta)
        return s
    s.p, s.alt = engine.DeviceParticles(n), engine.DeviceParticles(n)
    _fill(s.p, st, n)
    s.alt.count = n
    if s.kind == "publish":
        s.alt = None
        s.tracers = int((st["tracerIndex"] >= 0).sum())
        s.frame = torch.zeros(engine.pcls_frame_bytes(n, s.tracers, True), dtype=torch.uint8, device="cuda")
        s.seq = 0
        return s
    # the arrays of the build's tree are outputs, so the caller owns them there
    s.bvh = engine.TorchBvh(n) if s.kind == "build" else engine.DeviceBvh(n)
    if s.kind == "build":
        s.fresh = True
        return s
    engine.sort_and_build_bvh(s.p, s.alt, s.bvh)
    s.h = s.p.arrays["h"].clone()
    s.acc = [s.p.arrays[f].clone() for f in ("accX", "accY", "accZ")]
    return s


PASS1_OUT = ("h", "shepardC", "surfFactor", "divV", "curlVX", "curlVY", "curlVZ")
PASS2_OUT = ("accX", "accY", "accZ", "drhoDt", "duDt", "radPowerW", "dSXX", "dSYY", "dSZZ", "dSXY", "dSXZ", "dSYZ",
             "dDamageCbrtDt")
HEADLESS_OUT = ("kineticPsu", "potentialPsu", "internalPsu", "radiatedPowerW", "totalMassPsu", "maxTempK")


def run(s):
    if s.kind == "step":
        engine.step(s.sim.p, s.sim.alt, s.sim.bvh, 0.0, MAX_DT, s.theta, s.dt.data_ptr())
        return {"dt": s.dt, "state": dict(s.sim.p.arrays)}
    if s.kind == "headless":
        dt = s.sim.step(MAX_DT, s.theta)
        tel = engine.reduce_telemetry(s.sim.p, 6.0, True)
        return {"dt": dt, "state": dict(s.sim.p.arrays), "tel": {f: tel[f] for f in HEADLESS_OUT}}
    if s.kind == "stagewise":
        dt = s.sim.step_stagewise(MAX_DT, s.theta)
        return {"dt": dt, "state": dict(s.sim.p.arrays)}
    if s.kind == "relax":
        v = engine.relax_single_body(s.sim.p, s.sim.alt, s.sim.bvh, s.anchor, s.radius, s.case["steps"])
        return {"vrms": v, "state": dict(s.sim.p.arrays)}
    if s.kind == "build":
        if not s.fresh:                             # the call swapped the buffers: the load order is in alt
            s.p, s.alt = s.alt, s.p
        s.fresh = False
        engine.sort_and_build_bvh(s.p, s.alt, s.bvh)
        t = s.bvh.t
        return {"state": dict(s.p.arrays),
                "tree": [t[f] for f in ("indicesSorted", "leftChild", "rightChild", "parent", "nodeComMass",
                                        "nodeMinExtent", "nodeMaxHPacked")]}
    if s.kind == "pass1":
        s.p.arrays["h"].copy_(s.h)                   # the stage updates h: every pass starts from the build's
        engine.sph_pass1_neighbors(s.p, s.bvh)
        return [s.p.arrays[f] for f in PASS1_OUT]
    if s.kind == "pass2":
        for f, a in zip(("accX", "accY", "accZ"), s.acc):   # the stage adds to gravity's acceleration
            s.p.arrays[f].copy_(a)
        engine.sph_pass2_forces(s.p, s.bvh)
        return [s.p.arrays[f] for f in PASS2_OUT]
    if s.kind == "gravity":
        engine.gravity_barnes_hut(s.p, s.bvh, s.theta)
        return [s.p.arrays[f] for f in ("accX", "accY", "accZ", "phiGrav")]
    tel = engine.reduce_telemetry(s.p, 6.0, True)
    s.seq += 1
    info = abi.PclsFrameInfo(100.0, s.seq, 0.5, s.tracers, 16, 1, 1)
    info.livingCom[:] = tel["livingComPsu"]
    info.sysCom[:] = tel["sysComPsu"]
    engine.pack_pcls_frame(s.p, info, s.frame)
    return {"frame": s.frame, "tel": tel}


def work(case):
    """Bytes: fields read once and written once.  Flops: the pair sums of the formulas and, for gravity, the
    interactions of a tree walk at theta (about 15.6 log2 n / theta^2 a particle)."""
    n, kind = case["n"], case["kind"]
    theta = float(case.get("theta", 0.5))
    gravity = 23.0 * 15.6 * math.log2(n) / theta ** 2
    if case.get("mode", 0) in (1, 3):
        gravity *= 2.0
    sph1, sph2, xsph = 57.0 * 65.0, 57.0 * 189.0, 57.0 * 41.0
    step = dict(bytes=344.0 * n, flops=n * (gravity + sph1 + sph2 + xsph + 400.0))
    if kind in ("step", "stagewise"):
        return step
    if kind == "headless":
        return dict(bytes=step["bytes"] + 53.0 * n, flops=step["flops"] + 200.0 * n)
    if kind == "relax":
        k = case["steps"] + 5.0
        return dict(bytes=k * step["bytes"], flops=k * step["flops"])
    if kind == "build":
        return dict(bytes=(2 * 212.0 + 4.0 + 16.0 + 2 * 48.0) * n, flops=60.0 * n)
    if kind == "pass1":
        return dict(bytes=(10 * 4.0 + 7 * 4.0) * n, flops=n * sph1)
    if kind == "pass2":
        return dict(bytes=(31 * 4.0 + 3.0 + 13 * 4.0) * n, flops=n * sph2)
    if kind == "gravity":
        return dict(bytes=(5 * 4.0 + 4 * 4.0) * n, flops=n * gravity)
    return dict(bytes=(53.0 + 47.0 + 21.0) * n, flops=300.0 * n)


# ------------------------------------------------------------- 64-bit values
def _morton_order(st):
    """The sorted order of a build: 21 bits an axis of the scene box (32-bit arithmetic, as the codes are defined),
    interleaved x y z, equal codes in load order."""
    code = torch.zeros(len(st["posX"]), device="cuda", dtype=torch.int64)
    for k, f in enumerate(("posX", "posY", "posZ")):
        v = st[f]
        lo, hi = v.min(), v.max()
        span = hi - lo
        inv = torch.where(span > 1.0e-6, torch.tensor(2097151.0, device="cuda") / span, torch.zeros_like(span))
        q = ((v - lo) * inv).clamp(0.0, 2097151.0).to(torch.int64)
        for b in range(21):
            code |= ((q >> b) & 1) << (3 * b + 2 - k)
    return torch.argsort(code, stable=True)


def _sorted64(st):
    order = _morton_order(st)
    return {f: (v[order].double() if v.is_floating_point() else v[order]) for f, v in st.items()}, order


def _pairs(x, H, both):
    """Pairs (i, j), j != i, with r < H_i, or r < max(H_i, H_j) when `both`; as two index tensors."""
    n = len(H)
    x32, h32 = (x - x.mean(0)).float(), H.float()
    out_i, out_j = [], []
    for a in range(0, n, 2048):
        d2 = torch.zeros(min(2048, n - a), n, device="cuda")
        for k in range(3):
            d2 += (x32[a:a + 2048, k, None] - x32[None, :, k]) ** 2
        R = torch.maximum(h32[a:a + 2048, None], h32[None, :]) if both else h32[a:a + 2048, None]
        c = torch.nonzero(d2 < R * R * 1.0001)
        out_i.append(c[:, 0] + a)
        out_j.append(c[:, 1])
    i, j = torch.cat(out_i), torch.cat(out_j)
    r = (x[i] - x[j]).norm(dim=1)
    R = torch.maximum(H[i], H[j]) if both else H[i]
    keep = (r < R) & (i != j)
    return i[keep], j[keep]


def _grad(r, H):
    """g of grad W = g (r_i - r_j), Wendland C2 of support H."""
    return torch.where(r < H, -210.0 / (math.pi * H ** 5) * (1.0 - r / H).clamp_min(0.0) ** 3, 0.0)


def _exact_pass1(st):
    f, _ = _sorted64(st)
    n = len(f["mass"])
    x = torch.stack([f["posX"], f["posY"], f["posZ"]], 1)
    v = torch.stack([f["velX"], f["velY"], f["velZ"]], 1)
    h, h0 = f["h"].clamp_min(1e-6), f["h0"].clamp_min(1e-6)
    H = 2.0 * h
    vol = f["mass"] / f["rho"].clamp_min(1e-9)
    i, j = _pairs(x, H, False)
    d = x[i] - x[j]
    r = d.norm(dim=1)
    w0 = 21.0 / (2.0 * math.pi * H ** 3)
    q = r / H[i]
    W = w0[i] * (1.0 - q) ** 4 * (1.0 + 4.0 * q)

    def add(val):
        return torch.zeros((n,) + val.shape[1:], device="cuda", dtype=torch.float64).index_add_(0, i, val)

    shep = vol * w0 + add(vol[j] * W)
    ns = add((vol[j] * W)[:, None] * d).norm(dim=1)
    G = add((vol[j] * _grad(r, H[i]))[:, None, None] * (v[j] - v[i])[:, :, None] * d[:, None, :])
    ngb = 1.0 + torch.bincount(i, minlength=n).double()
    fs = (1.6 * torch.maximum(1.0 - shep, ns / h) - 0.15).clamp(0.0, 1.0)
    fs = torch.where(ngb <= 2, 1.0, fs)
    hn = torch.minimum(6.0 * h0, torch.maximum(0.35 * h0, h * ((56.0 / ngb) ** (1.0 / 3.0)).clamp(0.92, 1.08)))
    return [hn, shep, fs, G[:, 0, 0] + G[:, 1, 1] + G[:, 2, 2], G[:, 2, 1] - G[:, 1, 2], G[:, 0, 2] - G[:, 2, 0],
            G[:, 1, 0] - G[:, 0, 1]]


def _exact_pass2(st):
    f, _ = _sorted64(st)
    n = len(f["mass"])
    x = torch.stack([f["posX"], f["posY"], f["posZ"]], 1)
    v = torch.stack([f["velX"], f["velY"], f["velZ"]], 1)
    h, rho, m = f["h"].clamp_min(1e-6), f["rho"].clamp_min(1e-9), f["mass"]
    H, cs = 2.0 * h, f["soundSpeed"].clamp_min(0.05)
    P = torch.where(f["phaseId"] != 0, f["pressure"].clamp_min(0.0), f["pressure"])
    curl = torch.sqrt(f["curlVX"] ** 2 + f["curlVY"] ** 2 + f["curlVZ"] ** 2)
    bal = f["divV"].abs() / (f["divV"].abs() + curl + 1e-4 * cs / h)
    S = torch.stack([torch.stack([f["sXX"], f["sXY"], f["sXZ"]], 1), torch.stack([f["sXY"], f["sYY"], f["sYZ"]], 1),
                     torch.stack([f["sXZ"], f["sYZ"], f["sZZ"]], 1)], 1)
    mat = f["materialId"].long()
    R = torch.where(P < 0.0, 0.3 * -P / rho ** 2, 0.0)
    vol = m / rho
    i, j = _pairs(x, H, True)
    d, dv = x[i] - x[j], v[i] - v[j]
    r = d.norm(dim=1)
    gi, gj = _grad(r, H[i]), _grad(r, H[j])
    g = (0.5 * (gi + gj))[:, None] * d
    vr, vg = (dv * d).sum(1), (dv * g).sum(1)

    def add(val):
        return torch.zeros((n,) + val.shape[1:], device="cuda", dtype=torch.float64).index_add_(0, i, val)

    drc = add(vol[j] * vg)
    same = (mat[i] == mat[j]).double()
    drd = add(same * vol[j] * 2.0 * (rho[j] - rho[i]) / (r * r + 0.01 * H[i] ** 2) * -(d * g).sum(1))
    hb, cb, rb = 0.5 * (h[i] + h[j]), 0.5 * (cs[i] + cs[j]), 0.5 * (rho[i] + rho[j])
    mu = hb * vr / (r * r + 0.01 * hb * hb)
    pi_ij = torch.where(vr < 0.0, (-cb * mu + 2.0 * mu * mu) / rb * 0.5 * (bal[i] + bal[j]), 0.0)
    Hb = 0.5 * (H[i] + H[j])
    q = (r / Hb).clamp(max=1.0)
    tens = torch.where((R[i] + R[j] > 0.0) & (r < Hb),
                       (R[i] + R[j]) * ((1.0 - q) ** 4 * (1.0 + 4.0 * q) / 0.6328125) ** 4, 0.0)
    por2 = P / rho ** 2
    Sr = S / (rho ** 2)[:, None, None]
    a = -m[j][:, None] * (por2[i] + por2[j] + pi_ij + tens)[:, None] * g
    a += m[j][:, None] * ((Sr[i] + Sr[j]) @ g[:, :, None])[:, :, 0]
    acc = add(a) + torch.stack([f["accX"], f["accY"], f["accZ"]], 1)
    dup, duav, dut = add(m[j] * vg), add(0.5 * m[j] * pi_ij * vg), add(0.5 * m[j] * tens * vg)
    dus = add(m[j] * ((S[i] @ -dv[:, :, None])[:, :, 0] * g).sum(1)) / rho ** 2
    G = add((vol[j] * gi)[:, None, None] * -dv[:, :, None] * d[:, None, :])
    surf, T, dam = f["surfFactor"], f["tempK"], f["damage"]
    diff = torch.where(f["shepardC"] > 0.85, 1.0 - surf, 0.0)
    drho = rho * drc + 0.05 * H * cs * diff * drd
    intact = bool(((f["tracerIndex"] >= 0) & (dam < 0.8)).any())
    amb = torch.where((f["bodyId"] == 0) & (dam < 0.8), 255.0, 3.0) if intact else torch.full_like(T, 3.0)
    rp = (3.0 * (m * 1e24).clamp_min(1.0) / (4.0 * math.pi * (rho * 1e6).clamp_min(1e-3))) ** (1.0 / 3.0)
    rad = surf * 0.9 * 5.670374419e-8 * math.pi * rp * rp * (T ** 4 - amb ** 4).clamp_min(0.0)
    du = por2 * dup + duav + dut + dus - rad / (m.clamp_min(1e-30) * 1e27)
    # strength rows (shear modulus, melting point, bulk modulus) of the materials of these scenes
    shear = torch.tensor([7.7e-2, 2.2e-2, 3.5e-3, 0.0, 8.0e-3], device="cuda", dtype=torch.float64)[mat]
    melt = torch.tensor([1811.0, 1600.0, 273.15, 0.0, 1500.0], device="cuda", dtype=torch.float64)[mat]
    bulk = torch.tensor([0.128, 0.018, 2.18e-3, 0.0, 0.012], device="cuda", dtype=torch.float64)[mat]
    on = (shear > 0.0) & (melt > 0.0)
    mue = (1.0 - dam) * shear * (1.0 - (T / melt.clamp_min(1e-9)) ** 2).clamp_min(0.0)
    E, W = 0.5 * (G + G.transpose(1, 2)), 0.5 * (G - G.transpose(1, 2))
    E = E - torch.eye(3, device="cuda", dtype=torch.float64) * (G.diagonal(dim1=1, dim2=2).sum(1) / 3.0)[:, None, None]
    dS = 2.0 * mue[:, None, None] * E + S @ W.transpose(1, 2) + W @ S     # Jaumann rate
    dS = torch.where(on[:, None, None], dS, 0.0)
    return acc, drho, du, rad, dS


def _exact_gravity(st):
    f, _ = _sorted64(st)
    n = len(f["mass"])
    x = torch.stack([f["posX"], f["posY"], f["posZ"]], 1)
    eps = 0.8 * f["h0"].clamp_min(1e-6)
    gm = G_PSU * f["mass"]
    out = torch.zeros(4, n, device="cuda", dtype=torch.float64)
    for a in range(0, n, 1024):
        d = x[a:a + 1024, None, :] - x[None, :, :]
        s2 = (d * d).sum(2) + (0.5 * (eps[a:a + 1024, None] + eps[None, :])) ** 2
        w = gm[None, :] * s2.rsqrt()
        w[torch.arange(len(d), device="cuda"), torch.arange(a, a + len(d), device="cuda")] = 0.0
        out[3, a:a + 1024] = -w.sum(1)
        out[:3, a:a + 1024] = -((w / s2)[:, :, None] * d).sum(1).T
    return list(out)


def _exact_telemetry(st, target_radius):
    f = {k: v.double() if v.is_floating_point() else v for k, v in st.items()}
    x = torch.stack([f["posX"], f["posY"], f["posZ"]], 1)
    v = torch.stack([f["velX"], f["velY"], f["velZ"]], 1)
    m = f["mass"]
    b0 = f["bodyId"] == 0
    M = m.sum()

    def com(sel, q):
        w = torch.where(sel, m, 0.0)
        return (w[:, None] * q).sum(0) / w.sum()

    L = torch.linalg.cross(x, v)
    every = torch.ones_like(b0)
    c0, v0 = com(b0, x), com(b0, v)
    o = dict(totalMassPsu=M, sysComPsu=com(every, x), massBody0Psu=m[b0].sum(), comBody0Psu=c0, velBody0Psu=v0,
             massOtherPsu=m[~b0].sum(), comOtherPsu=com(~b0, x), velOtherPsu=com(~b0, v), livingComPsu=c0,
             kineticPsu=(0.5 * m * (v * v).sum(1)).sum(), potentialPsu=(0.5 * m * f["phiGrav"]).sum(),
             internalPsu=(m * f["u"]).sum(), momentumPsu=(m[:, None] * v).sum(0),
             angularMomentumPsu=(m[:, None] * L).sum(0), maxTempK=f["tempK"].max(),
             maxPressureGPa=(f["pressure"] * 1000.0).max().clamp_min(0.0), maxDamage=f["damage"].max(),
             radiatedPowerW=f["radPowerW"].clamp_min(0.0).sum())
    e, ev = x - c0, v - v0
    near = b0 & ((e * e).sum(1) <= (1.5 * target_radius) ** 2)
    o["spinLPsu"] = (m * (e[:, 2] * ev[:, 0] - e[:, 0] * ev[:, 2]))[near].sum()
    o["spinIPsu"] = (m * (e[:, 0] ** 2 + e[:, 2] ** 2))[near].sum()
    seed = int(torch.argmin(f["phiGrav"]))
    c, cv = x[seed], v[seed]
    mass, radius = torch.maximum(o["massBody0Psu"], 0.5 * M), max(target_radius, 0.25)
    for _ in range(5):
        r2 = ((x - c) ** 2).sum(1)
        bound = 0.5 * ((v - cv) ** 2).sum(1) - G_PSU * mass / r2.sqrt().clamp_min(max(0.5 * radius, 0.1)) < 0.0
        mb = torch.where(bound, m, 0.0)
        mass = mb.sum()
        radius = max(0.5 * target_radius, math.sqrt(5.0 / 3.0) * math.sqrt(float((mb * r2).sum() / mass)))
        c, cv = (mb[:, None] * x).sum(0) / mass, (mb[:, None] * v).sum(0) / mass
    d, dv = x - c, v - cv
    r = d.norm(dim=1)
    mu = G_PSU * mass
    en = 0.5 * (dv * dv).sum(1) - mu / r.clamp_min(max(0.5 * radius, 0.1))
    j2 = (torch.linalg.cross(d, dv) ** 2).sum(1)
    peri = j2 / (mu * (1.0 + torch.sqrt((1.0 + 2.0 * en * j2 / mu ** 2).clamp_min(0.0))))
    disk = (en < 0.0) & (r > radius) & (peri > radius)
    o.update(remnantPsu=c, remnantVelPsu=cv, remnantMassPsu=mass, remnantRadiusPsu=radius,
             boundPlanetMassPsu=m[(en < 0.0) & ~disk].sum(), diskMassPsu=m[disk].sum(),
             ejectaMassPsu=m[en >= 0.0].sum(), impactorBoundMassPsu=m[(en < 0.0) & ~b0].sum())
    return {k: (w.tolist() if isinstance(w, torch.Tensor) else float(w)) for k, w in o.items()}


def exact(case, seed):
    kind, n = case["kind"], case["n"]
    if kind in ("step", "headless", "stagewise", "relax"):
        return None                                   # whole steps: chains of every stage
    if kind in ("pass1", "pass2") and n > EXACT_PAIRS_N:
        return None
    if kind == "gravity" and n > 150_000:
        return None
    st = _scene(case, seed)
    if kind == "pass1":
        return _exact_pass1(st)
    if kind == "pass2":
        acc, drho, du, rad, dS = _exact_pass2(st)
        # the damage rate jumps at its threshold: no 64-bit value for it
        return [acc[:, 0], acc[:, 1], acc[:, 2], drho, du, rad, dS[:, 0, 0], dS[:, 1, 1], dS[:, 2, 2], dS[:, 0, 1],
                dS[:, 0, 2], dS[:, 1, 2], None]
    if kind == "gravity":
        return _exact_gravity(st)                     # the direct sum, which the walk approximates
    if kind == "build":
        f, _ = _sorted64(st)                          # the moved fields; node records have no value here
        return {"state": f, "tree": [None] * 7}
    tel = _exact_telemetry(st, 6.0)
    return {"frame": None, "tel": tel}
