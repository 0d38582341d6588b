"""The calls of this framework that its speed is judged by.

Every case goes through a public entry point (``opticks_b200.engine``, ``opticks_b200.adjoint`` or the
C ABI of ``include/phox.h``) with the geometries of ``opticks_b200.scenes``.  A program keeps one
engine per geometry for its life, as the reference keeps one simulator per GPU, so the engines here
are made once and the states of all cases share them; gensteps, rays, hit records, the event index
and the output buffers belong to a state and come from its seed.
"""
from __future__ import annotations

import math
from statistics import NormalDist

import numpy as np
import torch

from opticks_b200 import _lib, adjoint, engine, scenes

WL = (300.0, 620.0)              # wavelength range of the adjoint's eight property bins (nm)
T_MIN, T_MAX = 0.05, 1.0e6       # the ray interval of a closest-hit query (mm)
SD = 0x40                        # surface-detect flag, what a hit selection asks for


# ---------------------------------------------------------------- the cases
def listed() -> list[dict]:
    return [
        # one low-energy event of an event loop on the host: gensteps go up, hits come back into the caller's array
        dict(name="host_1k", kind="event", scene="detector", source="scint", gensteps=1, photons=1_000, host=True),
        # the median event of a Monte Carlo production, one call per event, every output on the GPU
        dict(name="event_50k", kind="event", scene="detector", source="scint", gensteps=1, photons=50_000, host=False),
        # a muon-like event: the headline 10M scintillation photons from 1,000 gensteps
        dict(name="event_10m", kind="event", scene="detector", source="scint", gensteps=1_000, photons=10_000, host=False),
        # Cerenkov light of 200 tracks (rejection sampling against the property table)
        dict(name="cerenkov_1m", kind="event", scene="detector", source="cerenkov", gensteps=200, photons=5_000, host=False),
        # calibration source in a small geometry: three surfaces, no hierarchy to walk
        dict(name="torch_1m", kind="event", scene="box", source="torch", gensteps=1, photons=1_000_000, host=False),
        # bodies made of the rarer leaves (cones, polyhedra, phi cuts): the full CSG evaluator
        dict(name="leaf_zoo_200k", kind="event", scene="zoo", source="torch", gensteps=1, photons=200_000, host=False),
        # uneven events submitted together (lognormal photon counts), as a production server queues them
        dict(name="batched_256", kind="batched", events=256, median=50_000),
        # one optimisation step of material properties: expected hits per sensor and their gradient
        dict(name="adjoint_1m", kind="adjoint", gensteps=100, photons=10_000),
        # geometry validation: rays against one 15-node boolean tree holding a torus
        dict(name="scan_16m", kind="scan", rays=1 << 24, polish=False),
        # the same with the FP64 root polish, at a ragged size
        dict(name="scan_polish_1m", kind="scan", rays=1_000_003, polish=True),
        # closest hits of arbitrary rays over the whole detector (simtrace, visibility maps)
        dict(name="trace_1m", kind="trace", rays=1 << 20),
        # hits of an event merged per (sensor, 1 ns): selection from a million photons
        dict(name="merge_1m", kind="merge", records=1_000_000, lite=False, select=True),
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return min(hi, max(lo, int(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng) -> dict:
    kind = rng.choice(["event", "event", "event", "event", "batched", "adjoint", "scan", "trace", "merge"])
    if kind == "event":
        scene, source = rng.choice([("detector", "scint"), ("detector", "scint"), ("detector", "cerenkov"), ("detector", "input"),
                                    ("box", "torch"), ("zoo", "torch"), ("lists", "torch")])
        n = _log_int(rng, 1_000, 10_000_000 if source == "scint" else 1_000_000)
        g = 1 if source in ("torch", "input") else _log_int(rng, 1, min(1_000, n // 100))
        return dict(kind=kind, scene=scene, source=source, gensteps=g, photons=n // g, host=n < 100_000 and rng.random() < 0.5)
    if kind == "batched":
        return dict(kind=kind, events=_log_int(rng, 8, 256), median=_log_int(rng, 2_000, 50_000))
    if kind == "adjoint":
        g = _log_int(rng, 1, 100)
        return dict(kind=kind, gensteps=g, photons=_log_int(rng, 50_000, 1_000_000) // g)
    if kind == "scan":
        return dict(kind=kind, rays=_log_int(rng, 10_000, 1 << 24), polish=rng.random() < 0.5)
    if kind == "trace":
        return dict(kind=kind, rays=_log_int(rng, 10_000, 1 << 20))
    return dict(kind=kind, records=_log_int(rng, 1_000, 2_000_000), lite=rng.random() < 0.5, select=rng.random() < 0.5)


# ---------------------------------------------------------------- what a program keeps
_KEPT: dict = {}


def _scene(name: str) -> dict:
    """the engine of a geometry (one per process) with its boundary library and property tables"""
    if name not in _KEPT:
        icdf, sensors, most = None, 0, 1_000_000
        if name == "detector":
            fd, lib, icdf = scenes.detector()
            sensors, most = scenes.NUM_PMT, 10_000_000
        elif name == "box":
            fd, lib, _, _ = scenes.sphere_in_box(1)
        elif name == "zoo":
            fd, lib, _, _ = scenes.leaf_zoo_detector(1)
        elif name == "lists":
            fd, lib, _, _ = scenes.list_zoo_detector(1)
        else:
            fd, _ = scenes.csg_scan_tree(with_torus=True)
            _, lib, _, _ = scenes.sphere_in_box(1)
            most = 64
        phys = lib.arrays()
        if icdf is not None:
            phys["icdf"] = icdf
        eng = engine.Engine(fd.arrays(), phys, engine.default_config(max_photon=most, num_sensor=sensors))
        _KEPT[name] = dict(fd=fd, lib=lib, phys=phys, engine=eng, stream=torch.cuda.Stream())
    return _KEPT[name]


def _event_index(seed: int) -> int:
    return 1 + seed % 4095


def _gensteps(case: dict, seed: int, lib) -> np.ndarray:
    g, n = case["gensteps"], case["photons"]
    if case.get("source", "scint") == "scint":
        return scenes.detector_gensteps(g, n, seed=seed, lib=lib)
    if case["source"] == "input":
        return scenes.input_photon_genstep(n)[None]
    if case["source"] == "torch":
        return scenes.torch_genstep(n, wavelength=440.0, radius=0.0)[None]
    rng = np.random.Generator(np.random.PCG64(seed))      # Cerenkov tracks in the scintillator
    line = lib.material_line("LS")
    pos = scenes.uniform_ball(g, 16000.0, rng)
    out = []
    for k in range(g):
        d = rng.normal(size=3)
        d *= rng.uniform(1.0, 40.0) / np.linalg.norm(d)
        out.append(scenes.cerenkov_genstep(n, tuple(pos[k]), line, delta=tuple(d), beta_inverse=1.0 / rng.uniform(0.75, 0.9999),
                                           time=float(rng.uniform(0.0, 5.0))))
    return np.stack(out)


def _outputs(n: int) -> dict:
    """an event's output buffers; hits fill the first rows of theirs, so it starts out zero"""
    return dict(photon=torch.empty((n, 4, 4), dtype=torch.float32, device="cuda"),
                seq=torch.empty((n, 2, 2), dtype=torch.int64, device="cuda"),
                hit=torch.zeros((n, 4, 4), dtype=torch.float32, device="cuda"))


def _unit(n: int, gen) -> torch.Tensor:
    v = torch.randn((n, 3), generator=gen, device="cuda", dtype=torch.float64)
    return v / v.norm(dim=1, keepdim=True)


def _rays(case: dict, seed: int) -> torch.Tensor:
    """(6,n) SoA rays: origins uniform in a 2 m cube (scan) or in the water sphere (trace), isotropic"""
    gen = torch.Generator("cuda").manual_seed(seed)
    n = case["rays"]
    if case["kind"] == "scan":
        o = torch.rand((n, 3), generator=gen, device="cuda", dtype=torch.float64) * 2000.0 - 1000.0
    else:
        r = 19000.0 * torch.rand((n, 1), generator=gen, device="cuda", dtype=torch.float64) ** (1.0 / 3.0)
        o = r * _unit(n, gen)
    return torch.cat([o, _unit(n, gen)], dim=1).t().to(torch.float32).contiguous()


def _records(case: dict, seed: int) -> torch.Tensor:
    """photon (sphoton) or sphotonlite records of an event: about a fifth carry the detect flag"""
    gen = torch.Generator("cuda").manual_seed(seed)
    n = case["records"]

    def integers(hi):
        return torch.randint(0, hi, (n,), generator=gen, device="cuda", dtype=torch.int64)
    t = 60.0 + 40.0 * torch.rand((n,), generator=gen, device="cuda") - 5.0 * torch.rand((n,), generator=gen, device="cuda").log()
    sensor = integers(scenes.NUM_PMT) + 1
    flags = torch.where(torch.rand((n,), generator=gen, device="cuda") < 0.2, 0x2 | 0x800 | SD, 0x2 | 0x800 | 0x8)
    if case["lite"]:
        rec = torch.empty((n, 4), dtype=torch.int32, device="cuda")
        rec[:, 0] = (1 << 16) | sensor.to(torch.int32)
        rec[:, 1] = t.view(torch.int32)
        rec[:, 2] = integers(1 << 31).to(torch.int32)
        rec[:, 3] = flags.to(torch.int32)
        return rec
    rec = torch.randn((n, 4, 4), generator=gen, device="cuda", dtype=torch.float32)
    rec[:, 0, 3] = t
    words = rec.view(torch.int32)
    words[:, 1, 3] = (1 << 16) | (sensor.to(torch.int32) & 0xffff)
    words[:, 3, 0] = 0x40
    words[:, 3, 1] = sensor.to(torch.int32)
    words[:, 3, 2] = torch.arange(n, device="cuda", dtype=torch.int32)
    words[:, 3, 3] = flags.to(torch.int32)
    return words


# ---------------------------------------------------------------- one pass
def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    s = dict(case=case, event=_event_index(seed))
    if kind == "event":
        s.update(_scene(case["scene"]))
        gs = _gensteps(case, seed, s["lib"])
        n = case["gensteps"] * case["photons"]
        if case["source"] == "input":
            s["input"] = torch.from_numpy(scenes.input_photons(n, seed=seed, radius=17000.0)).cuda()
        if case["host"]:
            s.update(gs=gs, hit=torch.zeros((n, 4, 4), dtype=torch.float32).pin_memory().numpy())
        else:
            s.update(n=n, gs=torch.from_numpy(gs).cuda(), out=_outputs(n))
    elif kind == "batched":
        s.update(_scene("detector"))
        # the quantiles of the lognormal counts, in an order of the seed's (so that a case has one size)
        z = [NormalDist().inv_cdf((k + 0.5) / case["events"]) for k in range(case["events"])]
        counts = np.clip(np.round(case["median"] * np.exp(z)), 1_000, 5_000_000).astype(int)
        np.random.Generator(np.random.PCG64(seed)).shuffle(counts)
        gs = scenes.detector_gensteps(case["events"], 1, seed=seed, lib=s["lib"])
        gs.view(np.int32)[:, 0, 3] = counts
        n = int(counts.sum())
        s.update(n=n, gs=torch.from_numpy(gs).cuda(), out=_outputs(n),
                 ev=torch.arange(s["event"], s["event"] + len(gs), dtype=torch.int32, device="cuda"))
    elif kind == "adjoint":
        s.update(_scene("detector"))
        s["line"] = s["lib"].material_line("LS")
        rng = np.random.Generator(np.random.PCG64(seed))
        theta = adjoint.nominal_theta(s["phys"], s["line"], *WL) * (1.0 + 0.01 * rng.uniform(-1.0, 1.0, 32)).astype(np.float32)
        s.update(n=case["gensteps"] * case["photons"], gs=torch.from_numpy(_gensteps(case, seed, s["lib"])).cuda(),
                 theta=torch.from_numpy(theta), weight=torch.from_numpy(rng.uniform(0.5, 1.5, scenes.NUM_PMT)).cuda())
    elif kind == "scan":
        s.update(_scene("scan"), rays=_rays(case, seed), out=torch.empty((case["rays"], 4), dtype=torch.float32, device="cuda"))
    elif kind == "trace":
        s.update(_scene("detector"), rays=_rays(case, seed), out=torch.empty((case["rays"], 2, 4), dtype=torch.float32, device="cuda"))
    else:
        rec = _records(case, seed)
        s.update(_scene("detector"), rec=rec, out=torch.zeros_like(rec))
    return s


def _photon_rows(p):
    """sphoton rows: position, time, direction, polarisation, wavelength as numbers, flags and indices as words"""
    words = p.view(np.int32) if isinstance(p, np.ndarray) else p.view(torch.int32)
    return {"value": p[:, :3], "flags": words[:, 3]}


def run(s: dict):
    case, eng, stream = s["case"], s["engine"], s["stream"].cuda_stream
    kind = case["kind"]
    if kind == "event":
        if "input" in s:
            eng.set_input_photon(s["input"])
        if case["host"]:
            r = eng.simulate_into(s["gs"], s["event"], None, None, s["hit"])
            return {"hit": _photon_rows(s["hit"]), "num_hit": r["num_hit"], "status": r["status"]}
        o = s["out"]
        nh, status = eng.simulate_device(s["gs"], s["n"], s["event"], photon=o["photon"], seq=o["seq"], hit=o["hit"],
                                         hit_capacity=s["n"], stream=stream)
        return {"photon": _photon_rows(o["photon"]), "seq": o["seq"], "hit": _photon_rows(o["hit"]), "num_hit": nh, "status": status}
    if kind == "batched":
        o = s["out"]
        nh, status = eng.simulate_batched_device(s["gs"], s["ev"], s["n"], photon=o["photon"], seq=o["seq"], hit=o["hit"],
                                                 hit_capacity=s["n"], stream=stream)
        return {"photon": _photon_rows(o["photon"]), "seq": o["seq"], "hit": _photon_rows(o["hit"]), "num_hit": nh, "status": status}
    if kind == "adjoint":
        with torch.cuda.stream(s["stream"]):
            theta = s["theta"].clone().requires_grad_()
            hits = adjoint.expected_hits(theta, eng, s["gs"], s["n"], s["event"], s["line"], *WL)
            grad, = torch.autograd.grad((hits * s["weight"]).sum(), theta)
        return {"hits": hits.detach(), "grad": grad}
    if kind == "scan":
        eng.scan_device(0, s["rays"], case["rays"], s["out"], 0.0, int(case["polish"]), stream)
        return s["out"]
    if kind == "trace":
        L = _lib.lib()
        _lib.check(L.phx_trace_device(eng._h, s["rays"].data_ptr(), case["rays"], T_MIN, T_MAX, s["out"].data_ptr(), None, stream),
                   "phx_trace_device")
        return {"normal_t": s["out"][:, 0], "lposcost": s["out"][:, 1, 0], "ids": s["out"].view(torch.int32)[:, 1, 2:]}
    n = eng.merge_hits_device(s["rec"], s["out"], SD if case["select"] else 0xFFFFFFFF, 1.0, stream)
    return {"records": s["out"], "n": n}


def work(case: dict) -> dict:
    """bytes a pass cannot do without; the operations of a random walk have no closed count"""
    kind = case["kind"]
    if kind in ("event", "batched"):
        n = case["events"] * case["median"] * math.exp(0.5) if kind == "batched" else case["gensteps"] * case["photons"]
        hits = 1.0 if case.get("scene", "detector") != "detector" else 0.19
        rows = 64 * hits if case.get("host") else 64 + 32 + 64 * hits
        return {"bytes": n * (24 + rows) + 96 * case.get("gensteps", case.get("events", 1)), "flops": 0}
    if kind == "adjoint":
        return {"bytes": 24 * case["gensteps"] * case["photons"] + 33 * 8 * scenes.NUM_PMT, "flops": 0}
    if kind == "scan":
        return {"bytes": 40 * case["rays"], "flops": 0}
    if kind == "trace":
        return {"bytes": 56 * case["rays"], "flops": 0}
    row = 16 if case["lite"] else 64
    n, kept = case["records"], case["records"] * (0.2 if case["select"] else 1.0)
    # every record's flags are read; the kept ones are read whole and leave at most as many groups
    return {"bytes": 4 * n + row * kept + row * min(kept, scenes.NUM_PMT * 60), "flops": 0}


# ---------------------------------------------------------------- the same in 64 bits
# A solid's boundary along a ray: every leaf surface gives candidate distances, and the first
# candidate at which membership of the boolean combination changes is the intersection.
def _first_change(cands, inside, t_min):
    """cands (n,k) distances (junk allowed), inside(t) (n,k) membership along the ray; returns
    (t, index of the surface hit, found)"""
    big = torch.full_like(cands[:, :1], 1e30)
    c = torch.where(torch.isfinite(cands) & (cands > t_min), cands, big)
    t, order = c.sort(dim=1)
    edges = torch.cat([torch.full_like(big, t_min), t], dim=1)
    nxt = torch.cat([t, t[:, -1:] + 1.0], dim=1)
    mid = 0.5 * (edges + torch.where(nxt >= 1e29, edges + 1.0, nxt))
    state = inside(mid)
    change = (state[:, 1:] != state[:, :-1]) & (t < 1e29)
    found = change.any(dim=1)
    first = change.to(torch.int8).argmax(dim=1, keepdim=True)
    return t.gather(1, first)[:, 0], order.gather(1, first)[:, 0], found


def _quadratic(a, b, c):
    """both roots of a t^2 + 2 b t + c (not finite where there is none)"""
    disc = b * b - a * c
    root = torch.where(disc > 0, disc.clamp_min(0).sqrt(), torch.full_like(disc, float("nan")))
    q = torch.where(b > 0, -(b + root), -(b - root))
    return [q / a, c / q]


def _torus_roots(o, d, R, r):
    """roots of the torus quartic along unit rays between the ends of its bounding sphere"""
    b0 = (o * d).sum(1)
    disc = b0 * b0 - ((o * o).sum(1) - (R + r + 1.0) ** 2)
    out = torch.full((len(o), 4), float("nan"), dtype=o.dtype, device=o.device)
    at = (disc > 0).nonzero()[:, 0]
    if not len(at):
        return out
    s0, half = -b0[at], disc[at].sqrt()
    p, v = o[at] + s0[:, None] * d[at], d[at]
    B, C = 2 * (p * v).sum(1), (p * p).sum(1) + R * R - r * r
    c3, c2 = 2 * B, B * B + 2 * C - 4 * R * R * (v[:, 0] ** 2 + v[:, 1] ** 2)
    c1 = 2 * B * C - 8 * R * R * (p[:, 0] * v[:, 0] + p[:, 1] * v[:, 1])
    c0 = C * C - 4 * R * R * (p[:, 0] ** 2 + p[:, 1] ** 2)

    def f(u):
        return (((u + c3[:, None]) * u + c2[:, None]) * u + c1[:, None]) * u + c0[:, None]

    # stationary points: the real roots of the derivative's monic cubic (Cardano, trigonometric form)
    a, bq, cq = 0.75 * c3, 0.5 * c2, 0.25 * c1
    P, Q = bq - a * a / 3, 2 * a ** 3 / 27 - a * bq / 3 + cq
    D = 0.25 * Q * Q + P ** 3 / 27
    sq = D.clamp_min(0).sqrt()

    def cbrt(x):
        return x.sign() * x.abs() ** (1.0 / 3.0)
    one = cbrt(-0.5 * Q + sq) + cbrt(-0.5 * Q - sq)
    m = 2 * (-P / 3).clamp_min(0).sqrt()
    th = (3 * Q / (P * m)).nan_to_num(0.0).clamp(-1, 1).acos() / 3
    three = torch.stack([m * (th - 2 * math.pi * k / 3).cos() for k in range(3)], 1)
    crit = torch.where((D > 0)[:, None], one[:, None].expand(-1, 3), three) - a[:, None] / 3
    edges = torch.cat([-half[:, None], crit.clamp(-half[:, None], half[:, None]), half[:, None]], 1).sort(dim=1)[0]
    lo, hi = edges[:, :-1].clone(), edges[:, 1:].clone()
    flo = f(lo)
    crosses = (flo < 0) != (f(hi) < 0)
    for _ in range(70):
        x = 0.5 * (lo + hi)
        same = (f(x) < 0) == (flo < 0)
        lo, hi = torch.where(same, x, lo), torch.where(same, hi, x)
    out[at] = torch.where(crosses, 0.5 * (lo + hi) + s0[:, None], torch.full_like(lo, float("nan")))
    return out


def _exact_scan(rays: torch.Tensor) -> torch.Tensor:
    o, v = rays[:3].t().double(), rays[3:].t().double()
    length = v.norm(dim=1)
    d = v / length[:, None]
    ones = torch.ones_like(length)
    oo, od = (o * o).sum(1), (o * d).sum(1)
    rr, rd, dd = (o[:, :2] ** 2).sum(1), (o[:, :2] * d[:, :2]).sum(1), (d[:, :2] ** 2).sum(1)
    shift = torch.tensor([0.0, 0.0, 200.0], dtype=o.dtype, device=o.device)

    def plane(axis, at):
        return (at - o[:, axis]) / d[:, axis]
    cands = (_quadratic(dd, rd, rr - 250.0 ** 2) + [plane(2, -200.0), plane(2, 200.0)]                       # 0-3 cylinder
             + _quadratic(ones, od, oo - 254.0 ** 2) + [plane(2, 0.0), plane(2, 190.0)]                      # 4-7 zsphere
             + _quadratic(ones, od, oo - 240.0 ** 2)                                                         # 8-9 sphere
             + [plane(k, h * e) for k, e in ((0, 250.0), (1, 250.0), (2, 150.0)) for h in (-1.0, 1.0)])      # 10-15 box
    cands = torch.cat([torch.stack(cands, 1), _torus_roots(o + shift, d, 200.0, 20.0)], 1)                   # 16-19 torus

    def inside(t):
        x, y, z = (o[:, k, None] + t * d[:, k, None] for k in range(3))
        r2 = x * x + y * y
        q2 = r2 + z * z
        left = ((r2 < 250.0 ** 2) & (z.abs() < 200.0)) | ((q2 < 254.0 ** 2) & (z > 0.0) & (z < 190.0))
        cut = (q2 < 240.0 ** 2) & (x.abs() < 250.0) & (y.abs() < 250.0) & (z.abs() < 150.0)
        return (left & ~cut) | ((r2.sqrt() - 200.0) ** 2 + (z + 200.0) ** 2 < 400.0)
    t, k, found = _first_change(cands, inside, 0.0)
    p = o + t[:, None] * d
    n = torch.zeros_like(p)
    rad = p[:, :2].norm(dim=1)
    e = torch.eye(3, dtype=p.dtype, device=p.device)
    tor = p + shift
    ring = torch.cat([tor[:, :2] * (1.0 - 200.0 / rad)[:, None], tor[:, 2:]], 1)
    zero = torch.zeros_like(rad)
    n = torch.where((k < 2)[:, None], torch.stack([p[:, 0] / 250.0, p[:, 1] / 250.0, zero], 1), n)
    n = torch.where((k == 2)[:, None] | (k == 6)[:, None], -e[2], n)
    n = torch.where((k == 3)[:, None] | (k == 7)[:, None], e[2], n)
    n = torch.where(((k == 4) | (k == 5))[:, None], p / 254.0, n)
    n = torch.where(((k == 8) | (k == 9))[:, None], -p / 240.0, n)
    for j in range(6):                                     # the box bounds what is taken away
        n = torch.where((k == 10 + j)[:, None], e[j // 2] * (1.0 if j % 2 == 0 else -1.0), n)
    n = torch.where((k >= 16)[:, None], ring / 20.0, n)
    out = torch.cat([n, (t / length)[:, None]], 1)
    return torch.where(found[:, None], out, torch.zeros_like(out))


def _exact_trace(rays: torch.Tensor) -> dict:
    kept = _scene("detector")
    inst = np.asarray(kept["fd"].arrays()["inst"], np.float64).reshape(-1, 4, 4)[1:]      # the PMTs follow the global solid
    rot, pos = torch.from_numpy(inst[:, :3, :3].copy()).cuda(), torch.from_numpy(inst[:, 3, :3].copy()).cuda()
    o, v = rays[:3].t().double(), rays[3:].t().double()
    length = v.norm(dim=1)
    d = v / length[:, None]
    n = len(o)
    best = torch.full((n,), 1e30, dtype=o.dtype, device=o.device)
    normal, cost = torch.zeros_like(o), torch.zeros_like(best)
    ones = torch.ones_like(best)
    for radius in (scenes.R_WATER, scenes.R_LS + scenes.T_ACRYLIC, scenes.R_LS):
        for t in _quadratic(ones, (o * d).sum(1), (o * o).sum(1) - radius ** 2):
            take = torch.isfinite(t) & (t > T_MIN) & (t < best)
            p = o + t[:, None] * d
            best = torch.where(take, t, best)
            normal = torch.where(take[:, None], p / radius, normal)
            cost = torch.where(take, p[:, 2] / p.norm(dim=1), cost)
    near = []
    for a in range(0, n, 16384):                           # pairs whose ray passes a PMT's bounding ball
        oa, da = o[a:a + 16384], d[a:a + 16384]
        along = da @ pos.t() - (oa * da).sum(1)[:, None]
        gap = (oa * oa).sum(1)[:, None] + (pos * pos).sum(1)[None] - 2 * (oa @ pos.t()) - along * along
        ij = ((gap < 255.0 ** 2) & (along > -256.0) & (along - 256.0 < best[a:a + 16384, None])).nonzero()
        near.append(torch.stack([ij[:, 0] + a, ij[:, 1]], 1))
    near = torch.cat(near)
    i, j = near[:, 0], near[:, 1]
    R = rot[j].transpose(1, 2).inverse()                   # world to local, as row vectors: (p - pos) @ inverse
    lo = torch.linalg.solve(rot[j].transpose(1, 2), (o[i] - pos[j])[:, :, None])[:, :, 0]
    ld = torch.linalg.solve(rot[j].transpose(1, 2), d[i][:, :, None])[:, :, 0]
    a2, ab, aa = (ld * ld).sum(1), (lo * ld).sum(1), (lo * lo).sum(1)
    r2, rb, ra = (ld[:, :2] ** 2).sum(1), (lo[:, :2] * ld[:, :2]).sum(1), (lo[:, :2] ** 2).sum(1)
    cands = (_quadratic(a2, ab, aa - 254.0 ** 2) + [(z - lo[:, 2]) / ld[:, 2] for z in (0.0, 190.0)]
             + _quadratic(r2, rb, ra - 50.0 ** 2) + [(-200.0 - lo[:, 2]) / ld[:, 2]])

    def inside(t):
        x, y, z = (lo[:, k, None] + t * ld[:, k, None] for k in range(3))
        q = x * x + y * y
        return ((q + z * z < 254.0 ** 2) & (z > 0.0) & (z < 190.0)) | ((q < 50.0 ** 2) & (z > -200.0) & (z <= 0.0))
    t, k, found = _first_change(torch.stack(cands, 1), inside, T_MIN)
    p = lo + t[:, None] * ld
    e = torch.eye(3, dtype=p.dtype, device=p.device)[2]
    nl = torch.where((k < 2)[:, None], p / 254.0, torch.where(((k == 2) | (k == 6))[:, None], -e, e.expand_as(p)))
    side = torch.stack([p[:, 0] / 50.0, p[:, 1] / 50.0, torch.zeros_like(t)], 1)
    nl = torch.where(((k == 4) | (k == 5))[:, None], side, nl)
    t = torch.where(found, t, torch.full_like(t, 1e30))
    first = best.scatter_reduce(0, i, t, "amin")
    win = (t == first[i]) & (t < best[i])
    normal[i[win]] = (R[win].transpose(1, 2) @ nl[win][:, :, None])[:, :, 0]
    cost[i[win]] = p[win, 2] / p[win].norm(dim=1)
    hit = first < 1e29
    nt = torch.cat([normal, (first / length)[:, None]], 1)
    return {"normal_t": torch.where(hit[:, None], nt, torch.zeros_like(nt)), "lposcost": torch.where(hit, cost, torch.zeros_like(cost)),
            "ids": None}


def exact(case: dict, seed: int):
    """64-bit values of the ray queries.  A photon's fate hangs on its own stream of random numbers and
    the rounding of every step before it, so the simulations have no such values; merged hits are
    copied words."""
    if case["kind"] == "scan":
        rays = _rays(case, seed)
        return torch.cat([_exact_scan(rays[:, a:a + (1 << 20)]) for a in range(0, rays.shape[1], 1 << 20)])
    if case["kind"] == "trace":
        return _exact_trace(_rays(case, seed))
    return None
