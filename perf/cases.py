"""Performance cases of the radiation solve: the calls its users make, over the sizes they make
them at.

A case names one of seven uses (``use``) and its sizes:

  solve   one runBand through the C ABI's device-resident entry point (Context.run_band), with
          the materials, sources and temperatures that RadiationModel passes on every call.
          ``entry`` is "device", "backend" (the same pass sequence call by call through the
          RayTracingBackend-shaped entry points, as the C++ drop-in is driven) or "rebuild"
          (geometry that moved: upload, tree build and solve in every pass).
  sweep   a day of suns and several bands of one scene in one launch graph (run_sweep).
  multi   the same for several small scenes at once, as a server groups them (run_sweep_multi).
  stress  leaves, disks and turbid voxels with deep scattering and the residual stop.
  glass   a canopy under a roof of translucent panes.
  camera  a solve followed by an image, pixel labels and depths.
  energy  the surface energy balance that follows a radiation solve.

Scenes and values are synthetic and seeded: ``prepare(case, seed)`` draws another geometry, sun
and set of rays for another seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from helios_gb300 import _hrt, scenes
from helios_gb300.radiation import Context, RadiationModel, run_band_through_backend

# ------------------------------------------------------------------ cases --
LEAF = {"PAR": (0.08, 0.05), "NIR": (0.45, 0.40), "RED": (0.06, 0.04), "GREEN": (0.12, 0.10), "SW": (0.10, 0.05)}


def _solve(name, scene, n, bands, direct, diffuse, depth, entry="device", periodic=False, sky=True, lai=2.0):
    """scene: canopy (square leaves), mixed (squares and triangles) or orchard (triangle trees);
    n: leaves; bands: comma-separated, LW emits; sky: an isotropic sky besides the sun."""
    return {"name": name, "use": "solve", "scene": scene, "n": n, "bands": bands, "direct": direct,
            "diffuse": diffuse, "depth": depth, "entry": entry, "periodic": periodic, "sky": sky, "lai": lai}


def listed():
    return [
        # one plant or plot section per call, thousands of calls (parameter fits): the latency of a solve
        _solve("small canopy", "canopy", 1000, "SW", 100, 100, 2),
        # the C++ RadiationModel over this backend: every pass a call with buffers going to and fro
        _solve("drop-in calls", "canopy", 2500, "NIR,PAR", 100, 300, 2, entry="backend"),
        # the reference's homogeneous-canopy configuration
        _solve("canopy 20k", "canopy", 20000, "SW", 100, 300, 3),
        # a periodic stand in four bands, as a client of the served stream asks for
        _solve("periodic stand", "mixed", 63457, "GREEN,NIR,PAR,RED", 100, 200, 1, periodic=True, lai=3.1),
        # growing plants: a new geometry every step, sunlit fractions from the direct sun alone
        _solve("moving geometry", "mixed", 200003, "PAR", 100, 50, 0, entry="rebuild", sky=False, lai=1.5),
        # the headline configuration: 1 M triangles, PAR, NIR and emitted longwave, five scatterings
        _solve("orchard 1M", "orchard", 1000000, "LW,NIR,PAR", 100, 200, 5),
        # a day in 15-minute steps over an orchard block
        {"name": "day sweep", "use": "sweep", "n": 100000, "suns": 96, "bands": "NIR,PAR", "direct": 100,
         "diffuse": 200, "depth": 5},
        # small requests for different scenes that a server admitted together
        {"name": "served group", "use": "multi", "scenes": 6, "n": 9000, "suns": 3, "bands": "GREEN,NIR,PAR",
         "direct": 100, "diffuse": 200, "depth": 1},
        # a section of the deep-scattering configuration at its density of leaves and voxels
        {"name": "voxel canopy", "use": "stress", "n": 16000, "vox": 10, "direct": 100, "diffuse": 400, "depth": 20,
         "tolerance": 1e-6},
        # a greenhouse crop: two suns and a sky through sixteen panes
        {"name": "greenhouse", "use": "glass", "n": 6000, "bands": "NIR,PAR", "direct": 64, "diffuse": 100,
         "depth": 3, "periodic": False},
        # a synthetic photograph with labels for training images
        {"name": "camera image", "use": "camera", "n": 20000, "bands": "NIR,PAR", "direct": 64, "diffuse": 64,
         "depth": 1, "width": 800, "height": 600, "samples": 9},
        # leaf temperatures of a large stand from its absorbed radiation
        {"name": "energy balance", "use": "energy", "n": 500009},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed uses, of at most the largest one's rays."""
    while True:
        use = rng.choice(["solve", "solve", "solve", "solve", "sweep", "multi", "stress", "glass", "camera", "energy"])
        if use == "solve":
            c = _solve("", rng.choice(["canopy", "mixed", "orchard"]), _log(rng, 500, 1000000),
                       rng.choice(["SW", "PAR", "NIR,PAR", "LW,NIR,PAR", "GREEN,NIR,PAR,RED"]), rng.randint(36, 144),
                       _log(rng, 50, 400), rng.randint(0, 5), rng.choice(["device", "device", "backend", "rebuild"]),
                       rng.random() < 0.3, rng.random() < 0.8, round(rng.uniform(0.5, 5.0), 2))
            if c["entry"] == "backend" and c["n"] > 50000 or c["depth"] > 0 and not c["sky"] and c["entry"] == "rebuild":
                continue
            most = 2.8e9
        elif use == "sweep":
            c = {"use": use, "n": _log(rng, 2000, 200000), "suns": _log(rng, 4, 96), "bands": rng.choice(["PAR", "NIR,PAR"]),
                 "direct": rng.randint(49, 144), "diffuse": _log(rng, 50, 400), "depth": rng.randint(1, 5)}
            most = 1.3e9
        elif use == "multi":
            c = {"use": use, "scenes": rng.randint(2, 12), "n": _log(rng, 2000, 30000), "suns": rng.randint(1, 6),
                 "bands": rng.choice(["PAR", "NIR,PAR", "GREEN,NIR,PAR", "GREEN,NIR,PAR,RED"]), "direct": 100,
                 "diffuse": _log(rng, 50, 400), "depth": rng.randint(1, 2)}
            most = 5e8
        elif use == "stress":
            c = {"use": use, "n": _log(rng, 1000, 32000), "vox": rng.randint(3, 14), "direct": rng.randint(36, 100),
                 "diffuse": _log(rng, 64, 400), "depth": rng.randint(3, 20), "tolerance": rng.choice([0.0, 1e-6, 1e-3])}
            most = 2.8e8
        elif use == "glass":
            c = {"use": use, "n": _log(rng, 300, 12000), "bands": rng.choice(["PAR", "NIR,PAR"]), "direct": rng.randint(36, 100),
                 "diffuse": _log(rng, 50, 200), "depth": rng.randint(1, 3), "periodic": rng.random() < 0.3}
            most = 1.2e7
        elif use == "camera":
            c = {"use": use, "n": _log(rng, 1000, 100000), "bands": rng.choice(["PAR", "NIR,PAR"]), "direct": 64, "diffuse": 64,
                 "depth": 1, "width": rng.randint(160, 1024), "height": rng.randint(120, 768), "samples": rng.choice([1, 4, 9, 16])}
            most = 1e8
        else:
            c = {"use": use, "n": _log(rng, 1000, 1000000)}
            most = 1e9
        if use == "energy" or _rays(c) <= most:
            c.pop("name", None)
            return c


def _strata(r):
    d = int(math.sqrt(r))
    return d * (r // d)


def _rays(c):
    """Rays that a pass of the case traces at most (two faces of every leaf in a diffuse pass)."""
    dif = _strata(int(math.ceil(math.sqrt(c["diffuse"]))) ** 2)
    prims = c["n"] * c.get("scenes", 1) + (c["vox"] ** 3 if "vox" in c else 0)
    suns = c.get("suns", 2 if c["use"] == "glass" else 1)
    passes = c["depth"] + (1 if c.get("sky", True) or "LW" in c["bands"].split(",") else 0)
    rays = prims * (suns * _strata(c["direct"]) + 2 * dif * passes)
    return rays + c.get("width", 0) * c.get("height", 0) * (c.get("samples", 0) + 1)


def work(case):
    """A pass reads the primitives' transforms and its other inputs once and writes its outputs
    once.  Per ray at least: its random numbers, origin and direction (about 70 operations), one
    primitive test (about 45) and an addition per channel."""
    n = case["n"] * case.get("scenes", 1)
    if case["use"] == "energy":
        return {"bytes": n * (10 * 4 + 1 + 4 + 4 + 6 * 4), "flops": n * (5 * 40 + 40)}
    nb = len(case.get("bands", "NIR").split(","))
    channels = nb * case.get("suns", 1)
    nbytes = n * (64 + 8 * nb + 4 * channels) + case.get("width", 0) * case.get("height", 0) * (4 * nb + 8)
    return {"bytes": nbytes, "flops": _rays(case) * (115 + channels)}


# ------------------------------------------------------------------ scenes --
def _leaves(ctx, leaves, bands):
    for b in bands:
        if b == "LW":
            ctx.setPrimitiveData(leaves, "emissivity_LW", np.full(leaves.size, 0.96))
        else:
            ctx.setPrimitiveData(leaves, "reflectivity_" + b, np.full(leaves.size, LEAF[b][0]))
            ctx.setPrimitiveData(leaves, "transmissivity_" + b, np.full(leaves.size, LEAF[b][1]))


def _sun(rng):
    return scenes.sun_direction(rng.uniform(10.0, 65.0), rng.uniform(0.0, 360.0))


def _crowns(n, seed):
    """Trees of at most 5,000 leaves that hold n leaves together."""
    trees = max(1, -(-n // 5000))
    nx = int(math.ceil(math.sqrt(2 * trees))) if trees > 1 else 1
    ny = -(-trees // nx)
    return scenes.orchard(nx=nx, ny=ny, leaves_per_tree=max(1, n // (nx * ny)), side=0.03, seed=seed)


def _model(case, seed, ctx, leaves, rng):
    """The user's set-up of bands, rays and sources over the scene in ctx."""
    bands = case["bands"].split(",")
    _leaves(ctx, leaves, bands)
    n = ctx.getPrimitiveCount()
    if "LW" in bands:
        ctx.setPrimitiveData(np.arange(n), "temperature", 273.15 + rng.normal(25.0, 2.0, n))
    rad = RadiationModel(ctx)
    if case.get("periodic"):
        rad.enforcePeriodicBoundary("xy")
    suns = [rad.addCollimatedRadiationSource(_sun(rng)) for _ in range(2 if case["use"] == "glass" else 1)]
    for b in bands:
        rad.addRadiationBand(b)
        rad.setDirectRayCount(b, case["direct"])
        rad.setDiffuseRayCount(b, case["diffuse"])
        rad.setScatteringDepth(b, case["depth"])
        if b != "LW":
            rad.disableEmission(b)
            for k, s in enumerate(suns):
                rad.setSourceFlux(s, b, float(rng.uniform(300.0, 600.0)) / (1 + 3 * k))
        if case.get("sky", True):
            rad.setDiffuseRadiationFlux(b, 350.0 if b == "LW" else float(rng.uniform(30.0, 120.0)))
    rad.setSeed(seed)
    return rad, bands


def _solve_scene(case, seed):
    if case["scene"] == "canopy":
        sc = scenes.homogeneous_canopy(n_leaves=case["n"], leaf=0.1, domain=math.sqrt(case["n"] * 0.01 / case["lai"]),
                                       zlo=1.0, zhi=3.0, seed=seed)
    elif case["scene"] == "mixed":
        sc = scenes.mixed_canopy(case["n"], case["lai"], seed=seed)
    else:
        sc = _crowns(case["n"], seed)
    return sc


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    use = case["use"]
    if use == "energy":
        return _prepare_energy(case, rng)
    if use == "sweep":
        sc = _crowns(case["n"], seed)
        return {"case": case, "ctx": _built(sc), **_sweep_inputs(case, sc, seed, rng)}
    if use == "multi":
        ctxs, sweeps = [], []
        for k in range(case["scenes"]):  # uneven scenes, from a half to one and a half times case["n"] leaves
            sc = scenes.mixed_canopy(int(case["n"] * (0.5 + (k + 0.5) / case["scenes"])), rng.uniform(0.5, 5.0),
                                     seed=seed * 100 + k)
            ctxs.append(_built(sc))
            sweeps.append(_sweep_inputs(case, sc, seed + k, rng)["sweep"])
        return {"case": case, "ctxs": ctxs, "sweeps": sweeps}
    ctx = Context()
    if use == "stress":
        scale = case["n"] / 4.0e6
        n = case["n"]
        sc = scenes.deep_scatter(n_tri=3 * n // 4, n_patch=n // 8, n_disk=n // 8, vox_div=case["vox"],
                                 domain=24.0 * math.sqrt(scale), seed=seed)
        ctx.addScene(sc)
        leaves = np.arange(1, sc.n)
        rad, bands = _model({**case, "bands": "NIR", "periodic": True}, seed, ctx, leaves, rng)
        rad.setScatteringResidualTolerance(case["tolerance"])
    elif use == "glass":
        side = math.sqrt(case["n"] * 0.01 / 1.7)
        sc = scenes.homogeneous_canopy(n_leaves=case["n"], leaf=0.1, domain=side, zlo=0.5, zhi=2.0, seed=seed)
        ctx.addScene(sc)
        panes = [ctx.addPatch(((i + 0.5) * side / 4, (j + 0.5) * side / 4, 2.6 + 0.05 * ((i + j) % 2)),
                              (side / 4, side / 4), (0.08 * (i - 1.5), 0.3 * j)) for i in range(4) for j in range(4)]
        for k, u in enumerate(panes):
            for b in case["bands"].split(","):
                ctx.setPrimitiveData(u, "glass_n_" + b, 1.45 + 0.005 * k)
                ctx.setPrimitiveData(u, "glass_KL_" + b, 0.05)
        rad, bands = _model(case, seed, ctx, sc.groups["leaves"], rng)
    else:
        sc = _solve_scene(case, seed) if use == "solve" else scenes.homogeneous_canopy(
            n_leaves=case["n"], leaf=0.1, domain=math.sqrt(case["n"] * 0.01 / 2.0), zlo=0.5, zhi=2.0, seed=seed)
        ctx.addScene(sc)
        rad, bands = _model(case, seed, ctx, sc.groups["leaves"], rng)
        if use == "camera":
            side = math.sqrt(case["n"] * 0.01 / 2.0)
            rad.addRadiationCamera("cam", bands, (-0.3 * side, 0.2 * side, 2.0 + 0.8 * side),
                                   (0.5 * side, 0.5 * side, 0.5),
                                   {"camera_resolution": (case["width"], case["height"]), "HFOV": 55.0,
                                    "lens_diameter": 0.0}, case["samples"])
            rad.setCameraSkyRadiance(bands[0], 30.0)
    rad.updateGeometry()
    s = {"case": case, "ctx": rad.ctx, "desc": rad.solve_description(bands)}
    T, ty, ts = rad.geometry_arrays()
    if case.get("entry") == "backend":
        s["twosided"] = ts
    if case.get("entry") == "rebuild":
        s["geometry"] = (T, ty, ts, rad._bbox_faces(), rad.periodic)
    return s


def _built(sc):
    ctx = _hrt.Context(0)
    ctx.update_geometry(sc.T, sc.ptype, sc.twosided)
    ctx.build_accel()
    return ctx


def _sweep_inputs(case, sc, seed, rng):
    bands = case["bands"].split(",")
    if case["use"] == "sweep":
        suns, direct, diffuse, _ = scenes.day_sweep(day_of_year=int(rng.integers(120, 240)), n=case["suns"],
                                                    bands=tuple("PAR" if b == "SW" else b for b in bands))
    else:
        suns = np.stack([_sun(rng) for _ in range(case["suns"])])
        direct = rng.uniform(100.0, 600.0, (case["suns"], len(bands))).astype(np.float32)
        diffuse = rng.uniform(20.0, 150.0, (case["suns"], len(bands))).astype(np.float32)
    rho = np.tile(np.array([LEAF[b][0] for b in bands], np.float32), (sc.n, 1))
    tau = np.tile(np.array([LEAF[b][1] for b in bands], np.float32), (sc.n, 1))
    return {"sweep": {"sun_dir": suns, "direct_flux": direct, "diffuse_flux": diffuse, "rho": rho, "tau": tau,
                      "direct_rays": case["direct"], "diffuse_rays": case["diffuse"], "depth": case["depth"],
                      "seed": seed}}


def _prepare_energy(case, rng):
    n = case["n"]
    f = np.float32
    Ta = rng.uniform(275.0, 312.0, n).astype(f)
    es = 611.0 * np.exp(17.502 * (Ta - 273.15) / (Ta - 273.15 + 240.97))
    surf = {"air_temperature": Ta, "air_vapor_pressure": (rng.uniform(0.2, 0.9, n) * es).astype(f),
            "air_pressure": rng.uniform(9.0e4, 1.02e5, n).astype(f), "bl_conductance": rng.uniform(0.1, 2.0, n).astype(f),
            "moisture_conductance": np.where(rng.random(n) < 0.3, 0.0, rng.uniform(0.0, 0.5, n)).astype(f),
            "emissivity": rng.uniform(0.9, 1.0, n).astype(f), "other_flux": np.zeros(n, f),
            "heat_capacity": rng.uniform(0.0, 2000.0, n).astype(f), "surface_humidity": rng.uniform(0.7, 1.0, n).astype(f),
            "stomatal_sidedness": rng.uniform(0.0, 0.5, n).astype(f), "nsides": rng.integers(1, 3, n).astype(np.uint8),
            "dt": 0.0, "temperature_default": 300.0}
    return {"case": case, "ctx": _hrt.Context(0), "surface": surf, "R": rng.uniform(300.0, 1300.0, n).astype(f),
            "T": (Ta + rng.uniform(-2.0, 8.0, n)).astype(f)}


# --------------------------------------------------------------------- run --
def run(state):
    case, use = state["case"], state["case"]["use"]
    if use == "energy":
        T, out = state["ctx"].energy_balance(state["surface"], net_radiation=state["R"], temperature=state["T"],
                                             outputs=True)
        return {"temperature": T, "fluxes": out}
    if use == "sweep":
        return {"flux": state["ctx"].run_sweep(**state["sweep"]), "rays": state["ctx"].last_stats()["rays"]}
    if use == "multi":
        return {"flux": _hrt.run_sweep_multi(state["ctxs"], state["sweeps"])}
    ctx = state["ctx"]
    if case.get("entry") == "backend":
        return {"flux": run_band_through_backend(ctx, state["desc"], state["twosided"])}
    if case.get("entry") == "rebuild":
        ctx.update_geometry(*state["geometry"])
        ctx.build_accel()
    out = {"flux": ctx.run_band(state["desc"])}
    st = ctx.last_stats()
    out["rays"], out["iterations"] = st["rays"], st["iterations"]
    if use == "camera":
        out.update(ctx.last_cameras[0])
    return out


# ------------------------------------------------------------------- exact --
# The estimators in 64 bits on the same random numbers: every ray against every primitive.
MOST_PAIRS = 3e10


def exact(case, seed):
    if case["use"] == "energy":
        return _exact_energy(prepare(case, seed))
    if case["use"] != "solve" or case["periodic"] or _rays(case) * case["n"] > MOST_PAIRS:
        return None  # about a second for 1e10 ray-primitive pairs: hours for the large scenes
    s = prepare(case, seed)
    out = {"flux": _exact_solve(case, seed, s["desc"])}
    if case["entry"] != "backend":
        out["rays"] = out["iterations"] = None
    return out


def _philox(c0, c1, c2, k0, k1):
    """Philox4x32-10 (Salmon et al., SC'11) on int64 tensors holding 32-bit words; c3 = 0."""
    m32 = 0xFFFFFFFF

    def mul(a, b):
        lo, hi = a * (b & 0xFFFF), a * (b >> 16)
        mid = hi + (lo >> 16)
        return mid >> 16, ((mid & 0xFFFF) << 16) | (lo & 0xFFFF)

    c3 = torch.zeros_like(c0)
    c1, c2 = c1.expand_as(c0), torch.full_like(c0, c2)
    for r in range(10):
        h0, l0 = mul(0xD2511F53, c0)
        h1, l1 = mul(0xCD9E8D57, c2)
        c0, c1, c2, c3 = h1 ^ c1 ^ k0, l1, h0 ^ c3 ^ k1, l0
        k0, k1 = (k0 + 0x9E3779B9) & m32, (k1 + 0xBB67AE85) & m32
    return [(c >> 8).double() / 16777216.0 for c in (c0, c1, c2, c3)]


def _exact_solve(case, seed, d):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    sc = _solve_scene(case, seed)

    def t64(a):
        return torch.as_tensor(np.asarray(a, np.float64), device=dev)

    M = t64(sc.T).reshape(-1, 4, 4)
    tri = torch.as_tensor(sc.ptype == scenes.TRIANGLE, device=dev)
    two = torch.as_tensor(sc.twosided != 0, device=dev)
    A, B, C = M[:, :3, 0], M[:, :3, 1], M[:, :3, 3]
    P = torch.where(tri[:, None], C, C - 0.5 * A - 0.5 * B)
    cr = torch.linalg.cross(A, B)
    N = torch.nn.functional.normalize(torch.where(tri[:, None], -cr, cr), dim=1)
    n2 = (cr * cr).sum(1, keepdim=True)
    dualA, dualB = torch.linalg.cross(B, cr) / n2, torch.linalg.cross(cr, A) / n2
    n = M.shape[0]

    def closest(o, v):
        """Nearest primitive along each ray (-1: none) and whether its top face is met."""
        hit = torch.empty(o.shape[0], dtype=torch.int64, device=dev)
        top = torch.empty(o.shape[0], dtype=torch.bool, device=dev)
        step = max(1, int(2e8) // n)
        for i in range(0, o.shape[0], step):
            oo, vv = o[i:i + step], v[i:i + step]
            den = vv @ N.T
            t = ((P * N).sum(1) - oo @ N.T) / den
            a = oo @ dualA.T - (P * dualA).sum(1) + t * (vv @ dualA.T)
            b = oo @ dualB.T - (P * dualB).sum(1) + t * (vv @ dualB.T)
            ok = (t >= 1e-4) & (a >= 0) & (b <= 1) & torch.where(tri, a <= b, (a <= 1) & (b >= 0))
            t = torch.where(ok, t, math.inf)
            best, k = t.min(1)
            hit[i:i + step] = torch.where(torch.isfinite(best), k, -1)
            top[i:i + step] = den.gather(1, k[:, None])[:, 0] < 0
        return hit, top

    def origins(k, u, v):
        lo, hi = torch.minimum(u, v), torch.maximum(u, v)
        u, v = torch.where(tri[k], lo, u), torch.where(tri[k], hi, v)
        return P[k] + u[:, None] * A[k] + v[:, None] * B[k]

    labels = d["band_labels"]
    rho, tau = t64(d["rho"][0]), t64(d["tau"][0])
    nb, depth = len(labels), case["depth"]
    rin, stop, sbot = (torch.zeros(n, nb, dtype=torch.float64, device=dev) for _ in range(3))

    def deposit(gt, gb):
        nonlocal rin, stop, sbot
        rin = rin + (gt + gb) * (1 - rho - tau)
        stop, sbot = stop + gt * rho + gb * tau, sbot + gt * tau + gb * rho

    def ray_ids(keep, R):
        k = torch.arange(n, device=dev)[keep].repeat_interleave(R)
        return k, torch.arange(R, device=dev).repeat(int(keep.sum()))

    # direct pass: stratified origins (patches), the sun's strength |n . s| / R where unshadowed
    flux = t64(d["source_flux"][0])
    run_direct, sky, emits = bool((flux > 0).any()), t64(d["diffuse_flux"]), bool(d["emission"].any())
    if run_direct:
        dx = int(math.sqrt(case["direct"]))
        dy = case["direct"] // dx
        sun = torch.nn.functional.normalize(t64(np.asarray(d["sources"][0]["position"], np.float32)), dim=0)
        facing = N @ sun
        k, r = ray_ids(two | (facing > 0), dx * dy)
        u, v, _, _ = _philox(r, k, 0, seed, 0)
        u = torch.where(tri[k], u, (r % dx + u) / dx)
        v = torch.where(tri[k], v, (r // dx + v) / dy)
        hit, _ = closest(origins(k, u, v), sun.expand(k.numel(), 3))
        g = torch.zeros(n, dtype=torch.float64, device=dev).index_add_(0, k, (hit < 0).double()) / (dx * dy) * facing.abs()
        gt, gb = (torch.where(s, g, 0.0)[:, None] * flux for s in (facing > 0, facing <= 0))
        deposit(gt, gb)
    ftop, fbot = torch.zeros_like(rin), torch.zeros_like(rin)
    if depth > 0 and run_direct:
        ftop = torch.where(two[:, None], stop, stop + sbot)
        fbot = torch.where(two[:, None], sbot, stop + sbot)
        stop, sbot = torch.zeros_like(rin), torch.zeros_like(rin)

    R1 = int(math.ceil(math.sqrt(case["diffuse"])))

    def diffuse(number, top_out, bot_out, from_sky):
        G = []
        for face in (1, 0):
            k, r = ray_ids(two if face == 0 else torch.ones_like(two), R1 * R1)
            j0, j1, u, v = _philox(r, k, face, seed, number)
            Rt, ph = (r % R1 + j0) / R1, 2 * math.pi * (r // R1 + j1) / R1
            lx, ly, lz = Rt.sqrt() * ph.cos(), Rt.sqrt() * ph.sin(), (1 - Rt).sqrt()
            nn = N[k]  # orthonormal basis of Duff et al. (JCGT 2017)
            sg = torch.copysign(torch.ones_like(nn[:, 2]), nn[:, 2])
            a = -1 / (sg + nn[:, 2])
            b = nn[:, 0] * nn[:, 1] * a
            t1 = torch.stack([1 + sg * nn[:, 0] ** 2 * a, sg * b, -sg * nn[:, 0]], 1)
            t2 = torch.stack([b, sg + nn[:, 1] ** 2 * a, -nn[:, 1]], 1)
            w = t1 * lx[:, None] + t2 * ly[:, None] + nn * lz[:, None]
            hit, top = closest(origins(k, u, v), w if face else -w)
            seen = torch.where(top[:, None], top_out[hit.clamp_min(0)], bot_out[hit.clamp_min(0)])
            seen = torch.where(hit[:, None] >= 0, seen, from_sky.expand_as(seen))
            G.append(torch.zeros_like(rin).index_add_(0, k, seen) / (R1 * R1))
        deposit(*G)

    if emits or bool((sky > 0).any()):
        for b, on in enumerate(d["emission"]):
            if on:
                e = t64(d["eps"][:, b]) if depth > 0 else torch.ones(n, dtype=torch.float64, device=dev)
                out = 5.6703744e-8 * e * t64(d["temperature"]) ** 4
                ftop[:, b] += out
                fbot[:, b] += torch.where(two, out, 0.0)
        diffuse(1, ftop, fbot, sky)
        if depth > 0 and not run_direct:
            ftop, fbot, stop, sbot = stop, sbot, torch.zeros_like(rin), torch.zeros_like(rin)
    for it in range(depth if emits or run_direct or bool((sky > 0).any()) else 0):
        if it > 0 or (emits and run_direct):
            ftop, fbot = stop, sbot
        stop, sbot = torch.zeros_like(rin), torch.zeros_like(rin)
        diffuse(2 + it, ftop, fbot, torch.zeros_like(sky))
    return (rin + stop + sbot).cpu()


def _exact_energy(s):
    """The secant iteration of the balance in 64 bits, from (T, 400 K) to a relative step of 1e-4."""
    q = {k: np.asarray(v, np.float64) for k, v in s["surface"].items()}
    R, Tp = s["R"].astype(np.float64), s["T"].astype(np.float64)
    gH, gS, sd = q["bl_conductance"], q["moisture_conductance"], q["stomatal_sidedness"]
    with np.errstate(divide="ignore", invalid="ignore"):
        gM = np.where((gH == 0) | (gS == 0), 0.0,
                      1.08 * gH * gS * (sd / (1.08 * gH + gS * sd) + (1 - sd) / (1.08 * gH + gS * (1 - sd))))

    def es(T, zero):
        return 611.0 * np.exp(17.502 * (T - zero) / (T - zero + 240.97))

    def residual(T):
        return (R - q["nsides"] * q["emissivity"] * 5.67e-8 * T ** 4 - 29.25 * gH * (T - q["air_temperature"])
                - gM * 44000.0 * (es(T, 273.0) - q["air_vapor_pressure"] * q["surface_humidity"]) / q["air_pressure"]
                - q["other_flux"])

    T0, T1 = Tp.copy(), np.where(Tp == 400.0, Tp + 100.0, 400.0)
    r0, r1, T = residual(T0), residual(T1), T0.copy()
    going = np.ones(T.size, bool)
    for _ in range(100):
        going &= r0 != r1
        if not going.any():
            break
        with np.errstate(divide="ignore", invalid="ignore"):
            Tn = np.abs((T1 * r0 - T0 * r1) / (r0 - r1))
        rn, err = residual(Tn), np.abs(Tn - T0) / np.abs(T0)
        T = np.where(going, Tn, T)
        T1, r1 = np.where(going, T0, T1), np.where(going, r0, r1)
        T0, r0 = np.where(going, Tn, T0), np.where(going, rn, r0)
        going &= err > 1e-4
    T = np.where(np.isfinite(T), T, 300.0)
    vpd = (es(T, 273.15) - q["air_vapor_pressure"]) / q["air_pressure"]
    out = np.stack([29.25 * gH * (T - q["air_temperature"]), 44000.0 * gM * vpd, np.zeros_like(T),
                    R - q["nsides"] * q["emissivity"] * 5.67e-8 * T ** 4, vpd], 1)
    return {"temperature": T, "fluxes": out}
