"""Performance cases of the prognostic flow solver: what a program that uses it has it do.

A program keeps a solver context, its grid's static arrays and its host buffers, and for every
weather situation builds the initial field, solves, and takes the fields back; around that it
rasterises the set-up, writes and reads the flow-field cache, interpolates the wind at particles,
and, when it fits observations, runs the adjoint.  Grids, buildings and situations follow the
repository's own workloads (16x14 test grid, 100x100 cube, 160x160 and 400x400 city, 200x200
vegetated grid, hilly domains); the seed draws buildings, inflow, stability and particles.
"""
import math

import numpy as np
import torch

from gral_b200 import prep
from gral_b200.abi import PARTICLE_DTYPE, FieldArrays, MetProfile
from gral_b200.prognostic import PrognosticSolver

F32 = np.float32


def listed():
    return [
        # the smallest call: a test-size grid, a handful of iterations, host fields in and out
        {"name": "tiny", "kind": "solve", "domain": "small", "nii": 16, "njj": 14, "vert": 12, "model": 1, "simd": 8,
         "iterations": 5, "n": 1, "host": True, "diagnostic": False},
        # one cube in the open, one convergence interval of 100 iterations: the classic validation case
        {"name": "cube", "kind": "solve", "domain": "cube", "nii": 100, "njj": 100, "vert": 20, "model": 1, "simd": 8,
         "iterations": 100, "n": 1, "host": False, "diagnostic": False},
        # odd-sized hilly site, 16-lane parity, with the diagnostic step that follows the solve
        {"name": "hills", "kind": "solve", "domain": "hills", "nii": 203, "njj": 157, "vert": 20, "model": 1,
         "simd": 16, "iterations": 40, "n": 1, "host": True, "diagnostic": True},
        # a production city quarter, one weather situation
        {"name": "city", "kind": "solve", "domain": "city", "nii": 400, "njj": 400, "vert": 30, "model": 1, "simd": 8,
         "iterations": 60, "n": 1, "host": False, "diagnostic": False},
        # the k-epsilon turbulence model
        {"name": "keps", "kind": "solve", "domain": "city", "nii": 100, "njj": 90, "vert": 20, "model": 2, "simd": 8,
         "iterations": 20, "n": 1, "host": False, "diagnostic": False},
        # the model without diffusion on an odd grid, a few situations together
        {"name": "upwind", "kind": "solve", "domain": "city", "nii": 97, "njj": 131, "vert": 18, "model": 0, "simd": 8,
         "iterations": 20, "n": 3, "host": False, "diagnostic": False},
        # a batch of weather situations on a small quarter; 48 leaves a half-filled group of 32
        {"name": "batch_small", "kind": "solve", "domain": "city", "nii": 96, "njj": 96, "vert": 20, "model": 1,
         "simd": 8, "iterations": 20, "n": 48, "host": False, "diagnostic": False},
        # a larger batch on a larger quarter, the throughput form of the weather loop
        {"name": "batch_large", "kind": "solve", "domain": "city", "nii": 160, "njj": 160, "vert": 30, "model": 1,
         "simd": 8, "iterations": 12, "n": 64, "host": False, "diagnostic": False},
        # the differentiation workload: forward with checkpoints, then the vector-Jacobian product
        {"name": "gradient", "kind": "vjp", "nii": 200, "njj": 200, "vert": 25, "iterations": 12, "every": 4},
        # writing a solved production field to the flow-field cache and reading one back
        {"name": "cache", "kind": "cache", "nii": 400, "njj": 400, "vert": 30, "mode": 1},
        # wind at the particles of one time step
        {"name": "particles", "kind": "particles", "nii": 256, "njj": 256, "vert": 30, "particles": 1 << 19,
         "terrain": 0},
        # the set-up of a quarter: sub-domains, initial field, vegetation
        {"name": "setup", "kind": "setup", "nii": 200, "njj": 180, "vert": 25, "lines": 500, "heights": 1},
    ]


def _between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    # single solves are most of the use; batches, gradients, cache, particles and set-up the rest
    kind = rng.choice(["solve"] * 6 + ["batch"] * 2 + ["vjp", "cache", "particles", "setup"])
    if kind == "solve":
        model = rng.choice([1, 1, 1, 1, 2, 0])
        domain = rng.choice(["small", "cube", "hills", "city", "city"])
        hi = 60 if domain == "small" else 330
        lo = 14 if domain == "small" else 64
        nii, njj, n = _between(rng, lo, hi), _between(rng, lo, hi), rng.choice([1, 1, 1, 2, 5])
        # no more work than the largest listed single solve
        most = min(50, 9600000 // (n * nii * njj), (20000 if model == 1 else 8000) // (nii + njj))
        return {"kind": "solve", "domain": domain, "nii": nii, "njj": njj,
                "vert": rng.randint(12, 30) if domain != "hills" else rng.randint(12, 20), "model": model,
                "simd": rng.choice([8, 8, 16]), "iterations": _between(rng, 5, most), "n": n,
                "host": rng.random() < 0.5, "diagnostic": rng.random() < 0.25}
    if kind == "batch":
        return {"kind": "solve", "domain": "city", "nii": _between(rng, 48, 140), "njj": _between(rng, 48, 140),
                "vert": rng.randint(15, 30), "model": rng.choice([1, 1, 1, 2]), "simd": rng.choice([8, 16]),
                "iterations": rng.randint(4, 10), "n": rng.randint(33, 64), "host": False, "diagnostic": False}
    if kind == "vjp":
        return {"kind": "vjp", "nii": (n := _between(rng, 48, 200)), "njj": n, "vert": rng.randint(15, 25),
                "iterations": rng.randint(3, 12), "every": rng.choice([0, 2, 4])}
    if kind == "cache":
        return {"kind": "cache", "nii": _between(rng, 40, 400), "njj": _between(rng, 40, 400),
                "vert": rng.randint(15, 30), "mode": rng.choice([0, 1, 2])}
    if kind == "particles":
        return {"kind": "particles", "nii": _between(rng, 40, 256), "njj": _between(rng, 40, 256),
                "vert": rng.randint(15, 30), "particles": _between(rng, 1000, 1 << 19), "terrain": rng.choice([0, 1])}
    return {"kind": "setup", "nii": _between(rng, 40, 200), "njj": _between(rng, 40, 200), "vert": rng.randint(15, 30),
            "lines": _between(rng, 10, 500), "heights": rng.choice([1, 3])}


def _domain(case, seed):
    nii, njj, vert = case["nii"], case["njj"], case["vert"]
    domain = case.get("domain", "city")
    if domain == "small":
        return prep.small_domain(nii, njj, seed=seed, vert_cells_ff=vert)
    if domain == "hills":
        return prep.hilly_domain(nii, njj, 2.0, vert, seed, n_hills=2, n_buildings=12)
    if domain == "cube":
        c0, d0 = nii // 2 - 4, njj // 2 - 4
        return prep.make_domain(nii, njj, 2.0, 2.0, 1.01, vert, [prep.Building(c0, c0 + 9, d0, d0 + 9, 20.0)])
    count = max(3, nii * njj * 64 // 160000)
    blocks = prep.random_buildings(nii, njj, 2.0, count, seed)
    return prep.make_domain(nii, njj, 2.0, 2.0, 1.05, vert, blocks)


def _situations(n, rng):
    out = []
    for _ in range(n):
        speed = float(rng.uniform(0.5, 4.0))
        k = int(rng.integers(0, 3))
        out.append(prep.Situation(direction_deg=float(rng.uniform(0, 360)), speed_10m=speed, z0=0.5,
                                  ustar=0.1 * speed + 0.1, obukhov=(50.0, 1000.0, -50.0)[k],
                                  potdtdz=(0.01, 0.0, -0.01)[k]))
    return out


def _met(sit):
    th = math.radians(sit.direction_deg)
    u, v = -sit.speed_10m * math.sin(th), -sit.speed_10m * math.cos(th)
    return MetProfile(np.array([0, 10.0], F32), np.array([0, u], F32), np.array([0, v], F32), sit.obukhov)


def _grid(dom):
    return dict(nii=dom.nii, njj=dom.njj, nkk=dom.nkk, vert_cells_ff=dom.vert_cells_ff, dxk=dom.dxk, dyk=dom.dyk,
                near_wall=0, igeb=10)


def _pinned(*shape, dtype=torch.float32):
    return torch.zeros(shape, dtype=dtype, pin_memory=True).numpy()


def _solver(dom, n=1):
    return PrognosticSolver(dom.nii, dom.njj, dom.nkk, dom.kadvmax, max_batch=n)


def _particles(dom, n, rng):
    p = np.zeros(n, dtype=PARTICLE_DTYPE)
    p["i"] = rng.integers(2, dom.nii, n)
    p["j"] = rng.integers(2, dom.njj, n)
    p["x"] = (p["i"] - 1 + rng.random(n)) * dom.dxk
    p["y"] = (p["j"] - 1 + rng.random(n)) * dom.dyk
    p["z"] = (120.0 * rng.random(n) ** 2 + 0.1).astype(F32)
    return p


def _lines(dom, n, rng):
    out = []
    for _ in range(n):
        crown = float(rng.uniform(2.0, 25.0))
        out.append(dict(crown_height=crown, trunk_height=crown * float(rng.uniform(0, 0.6)),
                        trunk_lad=float(rng.uniform(0.05, 0.5)), crown_lad=float(rng.uniform(0.1, 1.5)),
                        cov=float(rng.uniform(0.1, 1.0)), i=int(rng.integers(1, dom.nii + 1)),
                        j=int(rng.integers(1, dom.njj + 1)), drag=int(rng.random() < 0.85)))
    return out


def _profile(case, rng):
    """A met profile for the set-up cases: one height, or three with one wind direction each."""
    if case["heights"] == 1:
        return _met(_situations(1, rng)[0])
    u, v = np.sort(rng.uniform(0.5, 4.0, 3)), rng.uniform(-1.5, 1.5, 3)
    return MetProfile(np.array([0, 3.0, 12.0, 40.0], F32), np.array([0, *u], F32), np.array([0, *v], F32),
                      float(rng.choice([-60.0, 80.0, 1000.0])))


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    st = {"case": dict(case)}
    if kind == "vjp":
        dom = st["dom"] = prep.adjoint_domain(case["nii"], vert_cells_ff=case["vert"], seed=seed % 100000,
                                              n_buildings=max(3, case["nii"] * case["njj"] * 30 // 40000))
        sit = _situations(1, rng)[0]
        st["params"] = dom.params(sit, model=1, iterations=case["iterations"], quantise=0)
        st["start"] = prep.initial_fields(dom, sit)
        shape = st["start"].uk.shape
        st["work"] = FieldArrays(*(_pinned(*shape) for _ in range(3)))
        st["cot"] = []
        idx, _ = prep.probe_misfit(dom, st["start"], n_probes=1000, seed=seed % 100000)
        for _ in range(3):
            g = np.zeros(st["start"].uk.size, F32)
            g[idx] = rng.normal(0.0, 1.0, idx.size).astype(F32)
            st["cot"].append(g.reshape(shape))
        st["solver"] = _solver(dom)
        return st
    dom = st["dom"] = _domain(case, seed % 100000)
    shape = (dom.nii + 2, dom.njj + 2, dom.nkk + 2)
    if kind == "setup":
        st["solver"] = _solver(dom)
        st["met"] = _profile(case, rng)
        st["lines"] = _lines(dom, case["lines"], rng)
        st["cov"] = np.full((dom.nii + 2, dom.njj + 2), 0.1, F32)
        return st
    n = case.get("n", 1)
    sits = _situations(n, rng)
    st["solver"] = _solver(dom, n)
    st["static"], st["grid"], st["mets"] = dom.static, _grid(dom), [_met(s) for s in sits]
    model = case.get("model", 1)
    names = ("uk", "vk", "wk") if model == 1 else ("uk", "vk", "wk", "turb", "tdiss")
    # one page-locked buffer per field for all situations, one view per situation
    st["out"] = {name: _pinned(n, *shape) for name in names}
    st["fields"] = [FieldArrays(*(st["out"][name][b] for name in names)) for b in range(n)]
    iterations = case.get("iterations", 2)
    st["params"] = [dom.params(s, model=model, iterations=iterations, simd_width=case.get("simd", 8),
                               post_diagnostic=int(case.get("diagnostic", False))) for s in sits]
    if kind == "solve":
        if case["host"]:
            st["start"] = [prep.initial_fields(dom, s, model) for s in sits]
        return st
    # the cache and the particles work on a solved field that is resident on the device
    s = st["solver"]
    s.load_flat(st["params"], st["static"], st["mets"], st["grid"], st["fields"])
    s.iterate()
    s.store(st["fields"])
    if kind == "cache":
        st["payload"] = _pinned(s.gff_size(case["mode"]), dtype=torch.uint8)
        st["read"] = FieldArrays(*(_pinned(*shape) for _ in range(3)))
    else:
        st["where"] = dict(terrain=case["terrain"], buildings=1, ikooa=0, jkooa=0, dxk=dom.dxk, dyk=dom.dyk, ahmin=0.0)
        st["particles"] = _particles(dom, case["particles"], rng)
    return st


def run(st):
    case, s, dom = st["case"], st["solver"], st["dom"]
    kind = case["kind"]
    if kind == "solve":
        if case["host"]:
            for f, f0 in zip(st["fields"], st["start"]):
                for a, b in ((f.uk, f0.uk), (f.vk, f0.vk), (f.wk, f0.wk), (f.turb, f0.turb), (f.tdiss, f0.tdiss)):
                    if a is not None:
                        np.copyto(a, b)
            stats = s.calculate_batch(st["params"], st["static"], st["fields"])
        else:
            s.load_flat(st["params"], st["static"], st["mets"], st["grid"], st["fields"])
            s.iterate()
            stats = s.store(st["fields"])
        return {**st["out"], "iterations": [x["iterations"] for x in stats[:8]],
                "residual": [x["last_delta_umax"] for x in stats[:8]]}
    if kind == "vjp":
        w, f0 = st["work"], st["start"]
        for a, b in ((w.uk, f0.uk), (w.vk, f0.vk), (w.wk, f0.wk)):
            np.copyto(a, b)
        s.vjp_forward(st["params"], dom.static, w, case["iterations"], case["every"])
        veg, u0, v0, w0, _ = s.vjp(*st["cot"])
        return {"uk": w.uk, "vk": w.vk, "wk": w.wk, "d_veg": veg, "d_u0": u0, "d_v0": v0, "d_w0": w0}
    if kind == "cache":
        payload = s.gff_pack(0, case["mode"], 240.0, 2.5, 4, out=st["payload"])
        uk, vk, wk, head = s.gff_unpack(payload, dom.nii, dom.njj, dom.nkk, dom.dxk,
                                        kkart=dom.static.kkart if case["mode"] == 2 else None, out=st["read"])
        return {"payload": payload, "uk": uk, "vk": vk, "wk": wk, "flag": head[3]}
    if kind == "particles":
        ux, uy, uz, kk = s.wind_at(0, st["where"], dom.static.dzk, dom.static.hokart, st["particles"])
        return {"ux": ux, "uy": uy, "uz": uz, "level": kk}
    c = dom.static
    adv = s.subdomains(c.cutk, dom.nii, dom.njj, dom.dxk, dom.dyk)
    kk, ahk, kadv, f = s.flat_init(_grid(dom), c.cutk, c.dzk, c.hokart, st["met"], adv)
    veg, mask, cov = s.vegetation(dom.nii, dom.njj, dom.nkk, kk, c.dzk, c.hokart, st["lines"], st["cov"])
    return {"advdom": adv, "kkart": kk, "ahk": ahk, "kadvmax": kadv, "uk": f.uk, "vk": f.vk, "wk": f.wk, "veg": veg,
            "mask": mask, "cov": cov}


def _levels(case):
    """Full-height levels of the case's vertical grid (2 m first layer up to 800 m)."""
    stretch = 1.01 if case.get("domain") == "cube" else 1.05
    return int(math.log(1 + 800 * (stretch - 1) / 2) / math.log(stretch)) + 2


def work(case):
    cols = (case["nii"] + 2) * (case["njj"] + 2)
    field = 4.0 * cols * _levels(case)
    cells = float(case["nii"] * case["njj"] * case["vert"])
    kind = case["kind"]
    if kind == "solve":
        n, model = case["n"], case["model"]
        # a phase reads and writes each of its persistent fields once: 112 bytes and about 350
        # operations a cell and iteration (152 and 600 with the k-epsilon equations), and the
        # fields leave once (and enter once from the host)
        per, ops = (152.0, 600.0) if model == 2 else (112.0, 350.0)
        ends = (3 if model == 1 else 5) * field * (2 if case["host"] else 1)
        return {"bytes": n * (cells * per * case["iterations"] + ends), "flops": n * cells * ops * case["iterations"]}
    if kind == "vjp":
        # forward and its transpose, each phase's fields and their cotangents once
        return {"bytes": cells * 112.0 * 3 * case["iterations"] + 13 * field,
                "flops": cells * 350.0 * 4 * case["iterations"]}
    if kind == "cache":
        return {"bytes": 2 * (3 * field + 1.5 * field), "flops": 6.0 * cols * _levels(case)}
    if kind == "particles":
        # a particle's record, six field values in their 32-byte sectors, four results
        return {"bytes": case["particles"] * (32.0 + 6 * 32 + 16), "flops": case["particles"] * 30.0}
    return {"bytes": 4 * field, "flops": 10.0 * cols * _levels(case)}


def exact(case, seed):
    """The set-up's initial wind in 64 bits.

    The solves have no 64-bit counterpart to compare with: their sequential Gauss-Seidel sweeps
    round the velocities to a grid in every iteration, and the cache and particle cases work on
    solved fields."""
    if case["kind"] != "setup":
        return None
    rng = np.random.default_rng(seed)
    dom = _domain(case, seed % 100000)
    met = _profile(case, rng)
    _lines(dom, case["lines"], rng)
    nii, njj, nkk = dom.nii, dom.njj, dom.nkk
    cut = dom.static.cutk
    z32 = np.zeros(nkk + 2, F32)
    z32[1:nkk + 1] = dom.static.hokart[:nkk] + dom.static.dzk[1:nkk + 1] * F32(0.5)
    z = z32.astype(np.float64)
    h, ob = met.heights.astype(np.float64), float(F32(met.ob_length))
    power = 0.56 * ob ** -0.15 if ob > 0 else max(0.35 - 0.4 * abs(ob) ** -0.15, 0.05)
    inside = z32[None, None, :] <= cut[:, :, None]
    out = {"advdom": None, "kkart": None, "ahk": None, "kadvmax": None}
    for name, obs, axis in (("uk", met.obs_u, 0), ("vk", met.obs_v, 1)):
        o = obs.astype(np.float64)
        prof = np.interp(z, h[1:], o[1:])
        low = z <= h[1]
        prof[low] = o[1] * (z[low] / h[1]) ** power
        if h.size == 2:
            prof = o[1] * (z / h[1]) ** power
        prof[0] = prof[nkk + 1] = 0.0
        f = np.zeros((nii + 2, njj + 2, nkk + 2))
        f[1:nii + 1, 1:njj + 1, :] = prof
        f[inside] = 0.0
        if axis == 0:
            f[2:nii + 1][inside[1:nii]] = 0.0
            f[nii + 1, 1:njj + 1] = f[nii, 1:njj + 1]
        else:
            f[:, 2:njj + 1][inside[:, 1:njj]] = 0.0
            f[1:nii + 1, njj + 1] = f[1:nii + 1, njj]
        f[:, :, 0] = 0.0
        out[name] = f
    out["wk"] = np.zeros((nii + 2, njj + 2, nkk + 2))
    out.update(veg=None, mask=None, cov=None)
    return out
