"""Scenes whose surfaces cannot be culled (coaxial shells, parallel baffles, surfaces
through one another) are traced in the plain kernel's time; scenes whose surfaces lie apart
in less."""
import numpy as np
import pytest

from rayfactorcl_gb300 import generators
from rayfactorcl_gb300.scene import parse_scene_xml
from rayfactorcl_gb300.tracer import PREC_EXACT, PREC_FAST, PREC_FP64, Tracer

from test_gpu_culled import mixed

pytestmark = pytest.mark.gpu
PREC = {"exact": PREC_EXACT, "fast": PREC_FAST, "fp64": PREC_FP64}


def shells(n):
    x = generators._Xml("coaxial cylinders")
    for k in range(n):
        r = 0.5 + k / n
        x.prim("cylinderSurface", bounding=bool(k % 2), small=1.0, scale=(r, r, 2.0))
        x.close()
    return parse_scene_xml(x.text())


def baffles(n):
    x = generators._Xml("parallel discs, close together")
    for k in range(n):
        x.prim("disc", scale=(1.0, 1.0, 1.0), rotate=(180.0 * (k % 2), (1.0, 0.0, 0.0)), translate=(0.0, 0.0, 0.02 * k))
        x.close()
    return parse_scene_xml(x.text())


def crossed(n):
    rng = np.random.default_rng(4)
    x = generators._Xml("rectangles through one another")
    for _ in range(n):
        x.prim("rectangle", scale=(1.0, 1.0, 1.0), rotate=generators._axis_rotation(rng.normal(size=3)),
               translate=rng.uniform(-0.2, 0.2, 3))
        x.close()
    return parse_scene_xml(x.text())


def times(sc, prec, total):
    """Kernel times of the trace as it comes and of the plain kernel."""
    rays = np.full(sc.n, total // sc.n, np.int64)
    out = []
    for kw in ({}, {"table_mode": 1}):
        with Tracer(precision=PREC[prec], key1=6, **kw) as t:
            t.set_scene(sc)
            ms = []
            for _ in range(5):
                h = t.trace(rays)[0]
                ms.append(t.last_stats()[0])
            out.append((min(ms), h))
    assert np.array_equal(out[0][1], out[1][1])
    return out[0][0], out[1][0]


@pytest.mark.parametrize("prec,total", [("exact", 410_000), ("exact", 10_000_000), ("fast", 1_100_000),
                                        ("fast", 10_000_000), ("fp64", 100_000)])
@pytest.mark.parametrize("make", [shells, baffles, crossed])
@pytest.mark.parametrize("n", [24, 140])
def test_dense_scene_as_fast_as_plain(built_lib, make, n, prec, total):
    took, plain = times(make(n), prec, total)
    assert took < 1.2 * plain, (took, plain)


@pytest.mark.parametrize("prec,total", [("exact", 10_000_000), ("fast", 10_000_000), ("fp64", 1_000_000)])
def test_sparse_scene_is_culled(built_lib, prec, total):
    took, plain = times(mixed(64), prec, total)
    assert took < 0.8 * plain, (took, plain)
