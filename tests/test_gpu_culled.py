"""The culled kernel (rf_culled.cuh) against the plain kernel, whose results it must
give bit for bit: tallies and per-ray hits, in every plain precision, over the scenes
and budgets that take it.  ``table_mode=1`` pins the plain kernel."""
import numpy as np
import pytest

from helpers import golden_scene
from rayfactorcl_gb300 import generators
from rayfactorcl_gb300.scene import CYLINDER, FRUSTUM
from rayfactorcl_gb300.tracer import (COMPAT_ALL, PREC_EXACT, PREC_FAST, PREC_FP64, Tracer)

pytestmark = pytest.mark.gpu
PREC = {"exact": PREC_EXACT, "fast": PREC_FAST, "fp64": PREC_FP64}


def mixed(n, seed=11):
    c = np.floor(np.array([16, 16, 12, 10, 10], float) / 64 * n).astype(int)
    c[0] += n - c.sum()
    return generators.mixed_scene(seed=seed, total_rays=4, counts=tuple(int(x) for x in c)).scene


def odd_scene():
    """Emitters and surfaces the bounds do not speak for: a frustum of top radius 1
    (its emission divides by zero) and one a rounding away from it, a singular
    transform, a surface scaled down a millionfold, nearly parallel flat cones."""
    sc = mixed(40, seed=5)
    p = sc.primitives
    fr = np.flatnonzero(p["type"] == FRUSTUM)
    p["util1"][fr[0]] = 1.0
    p["util1"][fr[1]] = np.float32(1.0) + np.finfo(np.float32).eps
    p["util1"][fr[2]] = 0.0
    cy = np.flatnonzero(p["type"] == CYLINDER)
    p["invm"][cy[0]][:4] = 0.0
    s = np.float32(1e-6)
    m, im = p["m"][cy[1]].reshape(3, 4), p["invm"][cy[1]].reshape(3, 4)
    im[:, 3] /= s  # about the same centre line: m = T R S, invm = S^-1 R^-1 T^-1
    im[:, :3] /= s
    m[:, :3] *= s
    return sc


SCENES = {
    "mixed16": lambda: mixed(16), "mixed33": lambda: mixed(33), "mixed64": lambda: mixed(64),
    "mixed520": lambda: mixed(520),  # beyond the shared-memory tables
    "mixed1030": lambda: mixed(1030),  # two blocks of candidate words
    "furnace": lambda: generators.furnace_scene(4).scene, "furnace-bv": lambda: generators.furnace_scene(4).scene,
    "input-furnace": lambda: golden_scene("input-furnace"), "input-W100": lambda: golden_scene("input-W100"),
    "stress": lambda: generators.precision_stress(4).scene, "odd": odd_scene,
}


@pytest.mark.parametrize("compat", [0, COMPAT_ALL])
@pytest.mark.parametrize("prec", sorted(PREC))
@pytest.mark.parametrize("name", sorted(SCENES))
def test_culled_tallies_equal_plain(built_lib, name, prec, compat):
    sc = SCENES[name]()
    bv = name.endswith("-bv")
    total = {"exact": 600_000, "fast": 1_200_000, "fp64": 60_000}[prec]
    if compat and sc.n > 500:
        pytest.skip("the quirks are covered by the smaller scenes")
    rng = np.random.Generator(np.random.PCG64(3))
    rays = np.floor(rng.uniform(0.2, 1.8, size=sc.n) * total / sc.n).astype(np.int64) + 1
    rays[0] += total // 8  # one long row: several chunks
    rays[-1] = 0
    got = []
    for kw in ({}, {"table_mode": 1}):
        with Tracer(precision=PREC[prec], compat=compat, key1=77, **kw) as t:
            t.set_scene(sc)
            got.append(t.trace(rays, use_bv=bv)[0])
    assert np.array_equal(got[0], got[1])


@pytest.mark.parametrize("name,prec", [("mixed64", "exact"), ("mixed520", "exact"), ("furnace-bv", "exact"),
                                       ("input-furnace", "exact"), ("mixed64", "fp64"), ("furnace-bv", "fp64"),
                                       ("furnace", "fast")])
def test_culled_rays_equal_plain(built_lib, name, prec):
    """Per ray, over a range that starts and ends inside a draw, of curved and planar emitters."""
    sc = SCENES[name]()
    bv = name.endswith("-bv")
    first, count = 123_457, {"fp64": 30_001, "exact": 401_003, "fast": 50_001}[prec]
    with Tracer(precision=PREC[prec]) as a, Tracer(precision=PREC[prec], table_mode=1) as b:
        a.set_scene(sc)
        b.set_scene(sc)
        for e in (0, sc.n // 2, sc.n - 1):
            ra, rb = a.trace_rays(e, first, count, use_bv=bv), b.trace_rays(e, first, count, use_bv=bv)
            assert np.array_equal(ra, rb)
