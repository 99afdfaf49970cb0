"""A ray's result in mixed precision is a function of the ray alone: of neither its packet
nor the kernel that its trace takes.  Transforms whose invm describes a larger surface
than m (both are the caller's) put hits outside the bounding spheres, which follow m, so
that any kernel that keeps a hit its ray's own sphere check refuses shows up."""
import numpy as np
import pytest

from rayfactorcl_gb300 import generators
from rayfactorcl_gb300.scene import BV_DTYPE, SPHERE, Scene, parse_scene_xml
from rayfactorcl_gb300.tracer import PREC_EXACT, PREC_MIXED, Tracer

from test_gpu_culled import mixed

pytestmark = pytest.mark.gpu


def coaxial(x, kind, k):
    """k rings that tile a cylinder, or k annuli that tile an annulus, on a tilted axis."""
    rot = (-50.0, (0.6, 0.8, 0.0))
    t = np.array([1.0, -2.0, 0.5])
    if kind == "rings":
        axis = _axis(rot)
        for i in range(k):
            x.prim("cylinderSurface", small=1.0, scale=(0.4, 0.4, 0.2), rotate=rot, translate=t + 0.2 * i * axis)
            x.close()
    else:
        e = np.linspace(0.2, 1.0, k + 1)
        for i in range(k):
            x.prim("annulus", small=float(e[i]), large=float(e[i + 1]), rotate=rot, translate=t)
            x.close()


def _axis(rot):
    x = generators._Xml("axis")
    x.prim("cylinderSurface", small=1.0, scale=(1.0, 1.0, 1.0), rotate=rot)
    x.close()
    return parse_scene_xml(x.text()).primitives["m"][0].reshape(3, 4)[:, 2].astype(float)


def scene(n, stack=None, grown=1.0):
    """n surfaces of every type, the odd ones `grown` times as large for the tests as for
    emission, and a stack or plate of four."""
    sc = mixed(n, seed=29)
    sc.primitives["invm"][1::2] /= np.float32(grown)
    if stack:
        x = generators._Xml("stack")
        coaxial(x, stack, 4)
        out = Scene()
        out.primitives = np.concatenate([sc.primitives, parse_scene_xml(x.text()).primitives])
        sc = out
    return sc


def with_shells(sc):
    """The halves of the surfaces under two bounding spheres, one of them larger than its invm says."""
    b = np.zeros(2, BV_DTYPE)
    h = sc.n // 2
    b["type"], b["util2"], b["settings"] = SPHERE, -1.0, (1, 0)
    b["objStartIndex"], b["objEndIndex"] = (0, h), (h, sc.n)
    for k, r in enumerate((7.0, 9.0)):
        b["invm"][k] = (np.eye(4)[:3] / r).astype(np.float32).ravel()
    sc.bounding_volumes = b
    return sc


def budgets(sc, total):
    rng = np.random.Generator(np.random.PCG64(7))
    return np.floor(rng.uniform(0.2, 1.8, size=sc.n) * total / sc.n).astype(np.int64) + 1


@pytest.mark.parametrize("bv", [False, True])
def test_packets_do_not_matter(built_lib, bv):
    """Packets form in another order with another grid, and from run to run."""
    sc = scene(60, "rings", grown=1.5)
    if bv:
        sc = with_shells(sc)
    rays = budgets(sc, 3_000_000)
    got = []
    for grid in (0, 0, 37):
        with Tracer(precision=PREC_MIXED, key1=3, batched_grid=grid) as t:
            t.set_scene(sc)
            got.append(t.trace(rays, use_bv=bv)[0])
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])


@pytest.mark.parametrize("n,stack", [(14, None), (60, None), (60, "rings"), (60, "plate"), (600, None)])
def test_split_run_is_the_whole_run(built_lib, n, stack):
    """Ranges of few rays take another kernel than the whole run."""
    sc = scene(n, stack, grown=1.5)
    rays = budgets(sc, 300_000)
    with Tracer(precision=PREC_MIXED, key1=3) as t:
        t.set_scene(sc)
        whole = t.trace(rays)[0]
        first = np.zeros(sc.n, np.int64)
        while (first < rays).any():
            count = np.minimum(rays - first, 20_000 // sc.n + 3)
            t.trace_range(first, count, accumulate=bool(first.any()))
            first = first + count
        parts = t.results()[0]
    assert np.array_equal(whole, parts)


@pytest.mark.parametrize("member", [0, 2])
def test_emitters_of_a_plate(built_lib, member):
    """With next to no self-hit threshold a plate's emitter sees its plate's plane at
    rounding distance: the same in every kernel."""
    sc = scene(40, "plate")
    e = 40 + member
    with Tracer(precision=PREC_MIXED, eps=1e-12) as t:
        t.set_scene(sc)
        whole = t.trace_rays(e, 0, 300_000)
        parts = np.concatenate([t.trace_rays(e, k, 30_000) for k in range(0, 300_000, 30_000)])
    assert np.array_equal(whole, parts)


def test_spheres_follow_the_surface_that_is_hit(built_lib):
    """Round surfaces a tenth larger for the tests than for emission: the mixed kernels
    find the hits that the exact ones do."""
    sc = generators.mixed_scene(seed=23, total_rays=4, counts=(0, 0, 14, 12, 14)).scene
    sc.primitives["invm"] /= np.float32(1.1)
    a, b = Tracer(precision=PREC_EXACT), Tracer(precision=PREC_MIXED)
    with a, b:
        a.set_scene(sc)
        b.set_scene(sc)
        for e in (0, 20, 39):
            for count in (30_000, 400_000):
                d = a.trace_rays(e, 0, count) != b.trace_rays(e, 0, count)
                assert d.mean() < 1e-3, (e, count)
