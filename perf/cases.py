"""Workloads that a user of this framework has it do, through its public entry
points: single-scene traces in every precision, with and without bounding
surfaces; a batch of scenes in one launch; the add-rays-until-converged loop;
and the checks and smoothing of a traced view-factor matrix.

A case is a dict of plain values.  ``listed()`` names the representative ones,
``draw(rng)`` gives more of the same ranges, ``prepare`` makes what the caller
has in hand (scene tables, budgets, a context holding its scene), ``run`` is one
pass, ``work`` what a pass cannot do without, and ``exact`` the same result in
64 bits by plain torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from rayfactorcl_gb300 import generators
from rayfactorcl_gb300.tracer import (COMPAT_ALL, COMPAT_BV_STALE, COMPAT_SPHERE, COMPAT_STREAMS, PREC_EXACT,
                                      PREC_FAST, PREC_FP64, PREC_MIXED, Tracer)

PRECISION = {"exact": PREC_EXACT, "fast": PREC_FAST, "mixed": PREC_MIXED, "fp64": PREC_FP64}
EPS = 1e-3  # the reference's self-hit threshold, the default of every trace


def listed():
    return [
        # a quick look at a small model in the default precision: latency and launches
        {"name": "exact-enclosure", "kind": "trace", "scene": "enclosure", "n": 3, "rays": 12288,
         "precision": "exact", "bv": False, "compat": False},
        # the default precision on an ordinary model of a few tens of surfaces
        {"name": "exact-mixed64", "kind": "trace", "scene": "mixed", "n": 64, "rays": 10_000_000,
         "precision": "exact", "bv": False, "compat": False},
        # the drop-in run of the reference host: a furnace with bounding surfaces, reference quirks kept
        {"name": "exact-furnace-bv", "kind": "trace", "scene": "furnace", "n": 252, "rays": 10_000_000,
         "precision": "exact", "bv": True, "compat": True},
        # hardware approximations (the counterpart of native_*) on a larger, ragged model
        {"name": "fast-mixed201", "kind": "trace", "scene": "mixed", "n": 201, "rays": 5_000_001,
         "precision": "fast", "bv": False, "compat": False},
        # the FP64 tracer, the accuracy reference of the other precisions
        {"name": "fp64-mixed48", "kind": "trace", "scene": "mixed", "n": 48, "rays": 1_000_000,
         "precision": "fp64", "bv": False, "compat": False},
        # mixed precision: the closed three-surface enclosure at production accuracy
        {"name": "mixed-enclosure", "kind": "trace", "scene": "enclosure", "n": 3, "rays": 30_000_000,
         "precision": "mixed", "bv": False, "compat": False},
        # mixed precision where it is needed: thin annuli, flat cones, 1e4 from the origin
        {"name": "mixed-stress", "kind": "trace", "scene": "stress", "n": 16, "rays": 20_000_000,
         "precision": "mixed", "bv": False, "compat": False},
        # the benchmark's workload
        {"name": "mixed-mixed64", "kind": "trace", "scene": "mixed", "n": 64, "rays": 100_000_000,
         "precision": "mixed", "bv": False, "compat": False},
        # the fibre-drawing furnace with its bounding surfaces
        {"name": "mixed-furnace-bv", "kind": "trace", "scene": "furnace", "n": 252, "rays": 50_000_000,
         "precision": "mixed", "bv": True, "compat": False},
        # a design sweep: new scenes every call, uneven sizes and budgets, one launch
        {"name": "batch-sweep", "kind": "batch", "scenes": 24, "min_n": 10, "max_n": 400, "rays": 300_000},
        # rays added until every row's standard error is below a tolerance
        {"name": "converge-sweep", "kind": "converge", "scenes": 8, "min_n": 10, "max_n": 100, "tol": 1e-3,
         "rays": 10_000, "round_rays": 100_000},
        # checks, reciprocity and summation of a ring-resolved furnace's traced matrix
        {"name": "smooth-tube412", "kind": "smooth", "n": 412, "rays": 1_000_000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["trace"] * 7 + ["batch", "converge", "smooth"])
    if kind == "batch":
        lo = _log(rng, 8, 24)
        return {"kind": kind, "scenes": rng.randint(1, 24), "min_n": lo, "max_n": max(lo, _log(rng, 24, 400)),
                "rays": _log(rng, 10_000, 300_000)}
    if kind == "converge":
        lo = _log(rng, 8, 16)
        return {"kind": kind, "scenes": rng.randint(1, 8), "min_n": lo, "max_n": max(lo, _log(rng, 16, 100)),
                "tol": math.exp(rng.uniform(math.log(1e-3), math.log(5e-3))), "rays": _log(rng, 1000, 10_000),
                "round_rays": _log(rng, 10_000, 100_000)}
    if kind == "smooth":
        return {"kind": kind, "n": _log(rng, 16, 1200), "rays": _log(rng, 100_000, 4_000_000)}
    precision = rng.choice(["exact", "exact", "fast", "mixed", "mixed", "mixed", "fp64"])
    scene = rng.choice(["enclosure", "mixed", "mixed", "mixed", "furnace", "stress"])
    if scene == "stress" and precision in ("exact", "fast"):
        scene = "mixed"  # plain FP32 is no use 1e4 from the origin
    n = {"enclosure": 3, "furnace": 252, "stress": 16}.get(scene) or _log(rng, 13, 400)
    # brute-force tests of a pass, at most those of the largest listed case of the precision
    tests = {"exact": 2.5e9, "fast": 1e9, "fp64": 4.8e7, "mixed": 2.5e10}[precision]
    most = min({"enclosure": 3e7, "stress": 2e7, "furnace": 5e7}.get(scene, 1e8), tests / n)
    return {"kind": "trace", "scene": scene, "n": n, "rays": _log(rng, min(1e4, most / 2), most) + rng.randint(0, 3),
            "precision": precision, "bv": scene == "furnace" and rng.random() < 0.75,
            "compat": precision != "mixed" and rng.random() < 0.3}


# -- inputs -------------------------------------------------------------------

def _mixed(n, seed):
    """n surfaces in the type mix of the 64-surface benchmark scene."""
    counts = np.floor(np.array([16, 16, 12, 10, 10], float) / 64.0 * n).astype(int)
    counts[0] += n - counts.sum()
    return generators.mixed_scene(seed=seed, total_rays=4, counts=tuple(int(c) for c in counts))


def _workload(case, seed):
    """The scene and its areas; the seed moves the surfaces where the model is a random one."""
    if case["scene"] == "enclosure":
        return generators.enclosure3(4)
    if case["scene"] == "furnace":
        return generators.furnace_scene(4)
    if case["scene"] == "stress":
        return generators.precision_stress(4, seed=seed)
    return _mixed(case["n"], seed)


def _budgets(case, areas):
    """The rays spread over the emitters by area (an odd remainder goes to the first)."""
    total = int(case["rays"])
    rays = np.maximum(np.floor(areas / areas.sum() * total).astype(np.int64), 1)
    rays[0] += max(0, total - int(rays.sum()))
    return rays


def _sweep(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    scenes, rays = [], []
    for s in range(case["scenes"]):  # sizes spread evenly over their logarithm
        n = int(round(case["min_n"] * (case["max_n"] / case["min_n"]) ** ((s + 0.5) / case["scenes"])))
        w = _mixed(n, seed * 1009 + s)
        scenes.append(w.scene)
        b = np.exp(rng.uniform(math.log(case["rays"] / 10), math.log(case["rays"]), size=n))
        rays.append(np.floor(b).astype(np.int64) if case["kind"] == "batch" else np.full(n, case["rays"], np.int64))
    return scenes, rays


def _tube(case, seed):
    """A closed tube (radius 0.1, length 1.8) of n - 2 rings and two end discs: the
    closed-form view factors of its surfaces, traced with `rays` rays each, of which
    about one in a thousand is lost to the self-hit threshold near an edge."""
    n, radius = case["n"], 0.1
    rings = n - 2
    step = 1.8 / rings

    def coaxial(d):  # equal coaxial discs a distance d apart
        x = 2.0 + (np.maximum(d, 0.0) / radius) ** 2
        return 0.5 * (x - np.sqrt(x * x - 4.0))

    disc = math.pi * radius * radius
    z = np.arange(rings) * step
    gap = np.abs(z[:, None] - z[None, :]) - step  # between the near edges of two rings
    ring = disc * (coaxial(gap) - 2.0 * coaxial(gap + step) + coaxial(gap + 2.0 * step))
    ring_area = 2.0 * math.pi * radius * step
    np.fill_diagonal(ring, ring_area - 2.0 * disc * (1.0 - coaxial(np.array(step))))
    ends = disc * np.stack([coaxial(z) - coaxial(z + step), coaxial(1.8 - z - step) - coaxial(1.8 - z)])
    exchange = np.zeros((n, n))
    exchange[:rings, :rings] = ring
    exchange[rings:, :rings] = ends
    exchange[:rings, rings:] = ends.T
    exchange[rings, rings + 1] = exchange[rings + 1, rings] = disc * coaxial(np.array(1.8))
    areas = np.concatenate([np.full(rings, ring_area), [disc, disc]])
    F = np.maximum(exchange, 0.0) / areas[:, None]
    F /= F.sum(axis=1, keepdims=True)
    rng = np.random.Generator(np.random.PCG64(seed))
    lost = rng.uniform(0.5e-3, 1.5e-3, size=(n, 1))
    hits = rng.multinomial(case["rays"], np.concatenate([F * (1.0 - lost), lost], axis=1))
    return hits[:, :n] / float(case["rays"]), areas


def prepare(case, seed):
    key1 = (seed * 2654435761 + 12345) & 0xFFFFFFFF
    if case["kind"] == "smooth":
        F, areas = _tube(case, seed)
        return {"case": case, "tracer": Tracer(), "F": F, "areas": areas}
    if case["kind"] in ("batch", "converge"):
        scenes, rays = _sweep(case, seed)
        return {"case": case, "tracer": Tracer(precision=PREC_MIXED, key1=key1), "scenes": scenes, "rays": rays}
    w = _workload(case, seed)
    tracer = Tracer(precision=PRECISION[case["precision"]], key1=key1, compat=COMPAT_ALL if case["compat"] else 0)
    tracer.set_scene(w.scene)
    return {"case": case, "tracer": tracer, "rays": _budgets(case, w.areas)}


def run(state):
    case, tracer = state["case"], state["tracer"]
    if case["kind"] == "trace":
        hits, F = tracer.trace(state["rays"], use_bv=case["bv"])
        return {"hits": hits, "F": F}
    if case["kind"] == "batch":
        # all scenes' matrices end to end, as one array each
        hits, F = tracer.trace_batch(state["scenes"], state["rays"])
        return {"hits": np.concatenate([h.ravel() for h in hits]), "F": np.concatenate([f.ravel() for f in F])}
    if case["kind"] == "converge":
        hits, F, rays, rounds = tracer.converge_batch(state["scenes"], state["rays"], case["tol"],
                                                      case["round_rays"], 64)
        return {"hits": np.concatenate([h.ravel() for h in hits]), "F": np.concatenate([f.ravel() for f in F]),
                "rays": np.concatenate(rays), "rounds": rounds}
    sums, reciprocity = tracer.check_F(state["F"], state["areas"])
    # (the residual that smooth_F also gives is the rounding left in a converged iteration)
    F, iterations, _ = tracer.smooth_F(state["F"], state["areas"], closed=True)
    return {"sums": sums, "reciprocity": reciprocity, "F": F, "iterations": iterations}


def work(case):
    """Per ray: the emission (about 50 operations) and the test of the surface it hits
    (about 33); tables in, tallies and F out.  Smoothing: F read and written once, the
    symmetric matrix formed and scaled."""
    if case["kind"] == "smooth":
        return {"bytes": 16.0 * case["n"] ** 2, "flops": 6.0 * case["n"] ** 2}
    if case["kind"] == "trace":
        rays, nn, n = case["rays"], case["n"] ** 2, case["n"]
    else:
        lo, hi, k = case["min_n"], case["max_n"], case["scenes"]
        span = math.log(hi / lo)
        mean = (hi - lo) / span if span else lo  # of a log-uniform count, and of its square
        square = (hi * hi - lo * lo) / (2.0 * span) if span else lo * lo
        n, nn = k * mean, k * square
        # budgets: log-uniform over a factor of ten; converged: about 0.1 / tol^2 rays a row
        rays = n * (case["rays"] * 0.9 / math.log(10) if case["kind"] == "batch" else 0.1 / case["tol"] ** 2)
    return {"bytes": 112.0 * n + 16.0 * nn, "flops": 83.0 * rays}


# -- the same results in 64 bits ----------------------------------------------

def _mul32(a, b):
    """High and low words of the 64-bit product of a 32-bit constant and int64 tensors of 32-bit words."""
    p0, p1 = (a & 0xFFFF) * b, (a >> 16) * b
    return (p1 + (p0 >> 16)) >> 16, (p0 + ((p1 & 0xFFFF) << 16)) & 0xFFFFFFFF


def _uniforms(emitter, key1, compat, scene, gid):
    """The four 24-bit uniforms of Philox4x32-10 draws gid, in 64 bits."""
    one = torch.ones_like(gid)
    if compat & COMPAT_STREAMS:
        c = [one, one * 0xF00DCAFE, one * 0xDEADBEEF, one * 0xBEEFF00D]
    else:
        c = [one, one * emitter, gid >> 32, one * (0xBEEFF00D ^ scene)]
    k0, k1 = gid & 0xFFFFFFFF, key1
    for _ in range(10):
        h0, l0 = _mul32(0xD2511F53, c[0])
        h1, l1 = _mul32(0xCD9E8D57, c[2])
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return [(w >> 8).double() * 2.0 ** -24 for w in c]


def _emit(p, r, plain):
    """Origins and directions (3-vectors of tensors) of the rays of surface record p with uniforms r.
    plain: the FP32 paths that keep the reference's frame formula, which switches where 1 + nz is 0."""
    m = [float(v) for v in p["m"]]
    im = [float(v) for v in p["invm"]]
    u1, u2, kind = float(p["util1"]), float(p["util2"]), int(p["type"])
    zero = torch.zeros_like(r[0])
    turn = 2.0 * math.pi
    if kind in (5, 3):  # disc, annulus
        rho = torch.sqrt(r[1] if kind == 5 else (u2 - u1) * r[1] + u1)
        pt, nrm = (rho * torch.sin(turn * r[0]), rho * torch.cos(turn * r[0]), zero), (zero, zero, zero + 1.0)
    elif kind == 4:  # rectangle
        pt, nrm = (2.0 * r[0] - 1.0, 2.0 * r[1] - 1.0, zero), (zero, zero, zero + 1.0)
    elif kind == 0:  # cylinder
        x, y = torch.cos(turn * r[0]), torch.sin(turn * r[0])
        pt, nrm = (x, y, r[1]), (x * u2, y * u2, zero)
    elif kind == 1:  # frustum
        z = (torch.sqrt(1.0 - r[0] + r[0] * u1 * u1) - 1.0) / (u1 - 1.0)
        rho = 1.0 + z * (u1 - 1.0)
        x, y = rho * torch.cos(turn * r[1]), rho * torch.sin(turn * r[1])
        pt, nrm = (x, y, z), (x * u2, y * u2, (1.0 - u1) * rho * u2)
    else:  # sphere
        z = 2.0 * r[0] - 1.0
        rho = torch.sqrt(1.0 - z * z)
        x, y = rho * torch.cos(turn * r[1]), rho * torch.sin(turn * r[1])
        pt, nrm = (x, y, z), (x * u2, y * u2, z * u2)
    s = [m[4 * k] * pt[0] + m[4 * k + 1] * pt[1] + m[4 * k + 2] * pt[2] + m[4 * k + 3] for k in range(3)]
    n = [im[k] * nrm[0] + im[4 + k] * nrm[1] + im[8 + k] * nrm[2] for k in range(3)]
    length = torch.sqrt(n[0] ** 2 + n[1] ** 2 + n[2] ** 2)
    nx, ny, nz = (v / length for v in n)
    # cosine-weighted direction about +z, turned onto the normal
    ox, oy = torch.sqrt(r[3]) * torch.cos(turn * r[2]), torch.sqrt(r[3]) * torch.sin(turn * r[2])
    oz = torch.sqrt(1.0 - r[3])
    d = torch.where(nz < 0, (1.0 - nz) / (nx * nx + ny * ny), 1.0 / (1.0 + nz))  # 1/(1 + nz)
    d = torch.where(torch.isinf(d), torch.full_like(d, 0.5), d)
    if plain and kind in (3, 4, 5):
        row = np.asarray(p["invm"][8:11], np.float32)
        if np.float32(row[2] * (np.float32(1.0) / np.sqrt(np.sum(row * row, dtype=np.float32)))) == -1.0:
            d = torch.full_like(d, 0.5)
    c = [nz * ox + ny * d * (ny * ox - nx * oy) + nx * oz,
         nx * d * (nx * oy - ny * ox) + nz * oy + ny * oz,
         -nx * ox - ny * oy + nz * oz]
    return s, c


class _Group:
    """The surfaces of one type, as columns: hit distances of rays (rows) against all of them."""

    def __init__(self, kind, recs, index, dev):
        self.kind = kind
        self.index = torch.tensor(index, device=dev)
        im = torch.tensor(np.stack([r["invm"] for r in recs]).astype(np.float64), device=dev).T
        self.im = [im[k][None, :] for k in range(12)]
        self.u1 = torch.tensor([float(r["util1"]) for r in recs], dtype=torch.float64, device=dev)[None, :]
        self.u2 = torch.tensor([float(r["util2"]) for r in recs], dtype=torch.float64, device=dev)[None, :]

    def hit(self, s, c, compat):
        im, inf = self.im, math.inf
        sx, sy, sz = (im[4 * k] * s[0] + im[4 * k + 1] * s[1] + im[4 * k + 2] * s[2] + im[4 * k + 3] for k in range(3))
        cx, cy, cz = (im[4 * k] * c[0] + im[4 * k + 1] * c[1] + im[4 * k + 2] * c[2] for k in range(3))
        if self.kind in (3, 4, 5):
            t = -sz / cz
            x, y = sx + cx * t, sy + cy * t
            e = x * x + y * y
            ok = {5: e <= 1.0, 3: (e >= self.u1) & (e <= self.u2), 4: (x.abs() <= 1.0) & (y.abs() <= 1.0)}[self.kind]
            return torch.where(ok & (t > EPS), t, inf)
        if self.kind == 2:
            A, B = cx * cx + cy * cy + cz * cz, cx * sx + cy * sy + cz * sz
            D = B * B - A * (sx * sx + sy * sy + sz * sz - 1.0)
            if compat & COMPAT_SPHERE:  # discriminant used as it is, the far root never
                t = (-B - D) / A
                return torch.where((D > 0) & (t > EPS), t, inf)
            root = torch.sqrt(D)
            t1, t2 = (-B - root) / A, (-B + root) / A
            return torch.where(t1 > EPS, t1, torch.where(t2 > EPS, t2, inf))
        f = self.u1 - 1.0 if self.kind == 1 else 0.0  # radius 1 + f z
        fd, fs = f * cz, f * sz + 1.0
        A = cx * cx + cy * cy - fd * fd
        B = -(sx * cx + sy * cy - fs * fd)
        D = B * B - A * (sx * sx + sy * sy - fs * fs)
        root = torch.sqrt(D)
        t1, t2 = (B - root) / A, (B + root) / A
        z1, z2 = sz + cz * t1, sz + cz * t2
        t1 = torch.where((D >= 0) & (t1 >= EPS) & (z1 >= 0) & (z1 <= 1), t1, inf)
        return torch.where((D >= 0) & (t2 < t1) & (z2 > 0) & (z2 < 1) & (t2 > EPS), t2, t1)


class _Surfaces:
    def __init__(self, recs, first, dev):
        kinds = sorted({int(r["type"]) for r in recs})
        self.groups = [_Group(k, [r for r in recs if int(r["type"]) == k],
                              [first + i for i, r in enumerate(recs) if int(r["type"]) == k], dev) for k in kinds]

    def nearest(self, s, c, compat):
        """Distance and index (-1: none) of every ray's nearest hit."""
        best = torch.full_like(s[0][:, 0], math.inf)
        who = torch.full_like(best, -1, dtype=torch.int64)
        for g in self.groups:
            t, k = g.hit(s, c, compat).min(dim=1)
            nearer = t < best
            best = torch.where(nearer, t, best)
            who = torch.where(nearer, g.index[k], who)
        return best, who


def _traced(scene, rays, key1, compat=0, bv=False, scene_id=0, plain=False):
    """F of a scene by brute force in 64 bits; bv: the reference's walk of bounding surfaces."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    n = scene.n
    everything = _Surfaces(list(scene.primitives), 0, dev)
    walk = []
    if bv:
        for b in scene.bounding_volumes:
            lo, hi = int(b["objStartIndex"]), int(b["objEndIndex"])
            walk.append((_Surfaces([b], 0, dev), int(b["settings"]), _Surfaces(list(scene.primitives[lo:hi]), lo, dev)))
    F = np.zeros((n, n))
    chunk = max(4, (1 << 24) // max(n, 1) // 4 * 4)
    for e in range(n):
        counts = torch.zeros(n + 1, dtype=torch.int64, device=dev)
        for r0 in range(0, int(rays[e]), chunk):
            ray = torch.arange(r0, min(int(rays[e]), r0 + chunk), device=dev)
            u = torch.stack(_uniforms(e, key1, compat, scene_id, torch.arange(r0 // 4, r0 // 4 + (len(ray) + 3) // 4, device=dev)), 1)
            turn = (torch.arange(4, device=dev)[None, :] + (ray % 4)[:, None] + 1) % 4  # ray 4 g + v: the draw turned v + 1 times
            r = torch.gather(u[(ray - r0) // 4], 1, turn)
            s, c = _emit(scene.primitives[e], [r[:, k] for k in range(4)], plain)
            s, c = [v[:, None] for v in s], [v[:, None] for v in c]
            if not bv:
                who = everything.nearest(s, c, compat)[1]
            else:
                best = torch.full_like(s[0][:, 0], math.inf)
                who = torch.full_like(best, -1, dtype=torch.int64)
                child = who.clone()  # nearest child of the winning surface
                for shell, now, children in walk:
                    t = shell.nearest(s, c, compat)[0]
                    nearer = t < best
                    nw = children.nearest(s, c, compat)[1]
                    if now == 1:  # counts only where a child is hit
                        who = torch.where(nearer, nw, who)
                        nearer = nearer & (nw != -1)
                    elif not compat & COMPAT_BV_STALE:
                        who = torch.where(nearer, torch.full_like(who, -1), who)
                    best = torch.where(nearer, t, best)
                    child = torch.where(nearer, nw, child)
                who = torch.where(who == -1, child, who)
            counts += torch.bincount(who + 1, minlength=n + 1)
        F[e] = counts[1:].cpu().numpy() / float(rays[e])
    return F


def exact(case, seed):
    if case["kind"] == "converge":
        return None  # hundreds of rows in tens of rounds, one after another: minutes
    if case["kind"] == "smooth":
        F, A = _tube(case, seed)
        G = A[:, None] * F
        G = 0.5 * (G + G.T)
        both = (F > 0) & (F.T > 0)
        AF = A[:, None] * F
        with np.errstate(divide="ignore", invalid="ignore"):
            recip = np.where(both, np.abs(AF - AF.T) / np.maximum(AF, AF.T), 0.0).max()
        x = np.ones(len(A))
        for _ in range(4000):
            s = G @ x
            if np.max(np.abs(x * s / A - 1.0)) < 2e-15:
                break
            x = np.sqrt(x * A / s)
        return {"sums": float(np.max(np.abs(F.sum(axis=1) - 1.0))), "reciprocity": float(recip),
                "F": x[:, None] * G * x[None, :] / A[:, None], "iterations": None}
    key1 = (seed * 2654435761 + 12345) & 0xFFFFFFFF
    if case["kind"] == "batch":
        scenes, rays = _sweep(case, seed)
        if sum(float(r.sum()) * sc.n for sc, r in zip(scenes, rays)) > 2e10:
            return None  # over 20 seconds
        F = [_traced(sc, r, key1, scene_id=i).ravel() for i, (sc, r) in enumerate(zip(scenes, rays))]
        return {"hits": None, "F": np.concatenate(F)}
    w = _workload(case, seed)
    F = _traced(w.scene, _budgets(case, w.areas), key1, COMPAT_ALL if case["compat"] else 0, case["bv"],
                plain=case["precision"] in ("exact", "fast"))
    return {"hits": None, "F": F}
