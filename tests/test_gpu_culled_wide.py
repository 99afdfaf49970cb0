"""The culled kernel where a packet's 32 rays point all over the sphere, so that no packet
bound applies, among frusta made for those rays: a ray almost parallel to a generator
meets the cone at a root that rounding moves by many lengths of the frustum, and the plain
kernel then reports a hit far outside the frustum's sphere.  The culled kernel must too,
whatever else is in the packet."""
import numpy as np
import pytest

from rayfactorcl_gb300.scene import BV_DTYPE, DISC, FRUSTUM, PRIM_DTYPE, SPHERE, Scene
from rayfactorcl_gb300.tracer import PREC_EXACT, PREC_FAST, Tracer

pytestmark = pytest.mark.gpu
PREC = {"exact": PREC_EXACT, "fast": PREC_FAST}
KEY = 5


def record(kind, axes, origin, scale, util1=0.0):
    p = np.zeros((), PRIM_DTYPE)
    m = np.eye(4)
    m[:3, :3] = axes * np.asarray(scale, float)
    m[:3, 3] = origin
    p["m"] = m[:3].astype(np.float32).ravel()
    p["invm"] = np.linalg.inv(m)[:3].astype(np.float32).ravel()
    p["type"], p["util1"], p["util2"] = kind, util1, 1.0
    return p


def frame(z, rng):
    z = z / np.linalg.norm(z)
    x = np.cross(z, rng.normal(size=3))
    x /= np.linalg.norm(x)
    return np.stack([x, np.cross(z, x), z], axis=1)


def aimed(s, c, rng):
    """A small frustum with a generator along c, beside the ray (s, c), and how far beside."""
    half, h, top = rng.uniform(0.3, 1.2), np.exp(rng.uniform(np.log(0.05), np.log(0.3))), rng.uniform(0.0, 0.9)
    r = h * np.tan(half) / (1.0 - top)
    size = np.hypot(r, h)
    f = frame(c, rng)
    axis = (np.cos(half) * f[:, 2] + np.sin(half) * f[:, 0]) * rng.choice([-1.0, 1.0])
    w = rng.uniform(0.0, 2.0 * np.pi)
    beside = f[:, 0] * np.cos(w) + f[:, 1] * np.sin(w)
    base = s + c * rng.uniform(2.0, 8.0) + beside * (1.0 + size * rng.uniform(2.0, 5.0))
    far = np.linalg.norm(np.cross(base + axis * h / 2 - s, c)) - size
    return record(FRUSTUM, frame(axis, rng), base, (r, r, h), top), far


def crafted(oracle, n, exact):
    """A sphere that emits, and frusta made for its first 32 rays: for each ray one that the
    exact test hits from more than its size and 0.8 beside (the spheres are larger than their
    frusta by a hundredth of the longest ray), with tiny discs to make n surfaces; for the other
    arithmetic, whose hits cannot be foreseen here, as many as make n."""
    rng = np.random.default_rng(0)
    p = oracle.params(compat=0, key1=KEY)
    out = [record(SPHERE, np.eye(3), np.zeros(3), (1.0, 1.0, 1.0))]
    rays = [[np.array(v, float) for v in oracle.emit_ray(np.array(out), 0, p, k)] for k in range(32)]
    if exact:
        for k, (s, c) in enumerate(rays):
            for _ in range(60):
                some = [aimed(s, c, rng) for _ in range(60)]
                sc = Scene()
                sc.primitives = np.array(out[:1] + [f[0] for f in some])
                hit = int(oracle.trace_rays(sc, p, 0, k, k + 1)[0])
                if hit > 0 and some[hit - 1][1] > 0.8:
                    out.append(some[hit - 1][0])
                    break
        assert len(out) > 20
        while len(out) < n:
            out.append(record(DISC, np.eye(3), rng.uniform(2.0, 4.0, 3), (1e-3, 1e-3, 1.0)))
    else:
        while len(out) < n:
            f, far = aimed(*rays[len(out) % 32], rng)
            if far > 0.8:
                out.append(f)
    sc = Scene()
    sc.primitives = np.array(out)
    return sc


@pytest.mark.parametrize("prec", sorted(PREC))
@pytest.mark.parametrize("n,shell", [(500, True), (1100, False)])  # (1100: too many for the narrow kernel)
def test_wide_packets_equal_plain(built_lib, oracle_lib, n, shell, prec):
    sc = crafted(oracle_lib, n, prec == "exact")
    if shell:
        b = np.zeros(1, BV_DTYPE)
        b["type"], b["objEndIndex"], b["util2"] = SPHERE, n, -1.0
        b["invm"][0] = (np.eye(4)[:3] / 50.0).astype(np.float32).ravel()
        sc.bounding_volumes = b
    rays = np.zeros(n, np.int64)
    rays[0] = 32
    got = []
    for kw in ({}, {"table_mode": 1}):
        with Tracer(precision=PREC[prec], key1=KEY, **kw) as t:
            t.set_scene(sc)
            got.append((t.trace_rays(0, 0, 32, use_bv=shell), t.trace(rays, use_bv=shell)[0]))
    assert (got[1][0] > 0).sum() > (15 if prec == "exact" else 0)  # the plain kernel's far hits
    assert np.array_equal(got[0][0], got[1][0])
    assert np.array_equal(got[0][1], got[1][1])
