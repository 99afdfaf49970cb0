"""Culled and plain kernel compared where the other tests' budgets end in the narrow or the
plain kernel: FAST from 24 surfaces and 1e6 rays, EXACT from 16 and 1e6, per ray and in
tallies, with rows of very uneven length."""
import numpy as np
import pytest

from rayfactorcl_gb300 import generators
from rayfactorcl_gb300.tracer import COMPAT_ALL, PREC_EXACT, PREC_FAST, PREC_FP64, Tracer

from test_gpu_culled import mixed

pytestmark = pytest.mark.gpu
PREC = {"exact": PREC_EXACT, "fast": PREC_FAST, "fp64": PREC_FP64}


def apart(n):
    """Surfaces far enough apart that the rule takes the culled kernel at any of these sizes."""
    sc = mixed(n, seed=37)
    m, im = sc.primitives["m"], sc.primitives["invm"]
    shift = m[:, 3::4].astype(np.float64) * 3.0  # centres four times as far out
    m[:, 3::4] = (m[:, 3::4].astype(np.float64) + shift).astype(np.float32)
    lin = im.reshape(-1, 3, 4)[:, :, :3].astype(np.float64)
    im[:, 3::4] = (im[:, 3::4].astype(np.float64) - np.einsum("nij,nj->ni", lin, shift)).astype(np.float32)
    return sc


SCENES = {"apart16": lambda: apart(16), "apart24": lambda: apart(24), "mixed64": lambda: mixed(64),
          "furnace": lambda: generators.furnace_scene(4).scene}


@pytest.mark.parametrize("name,prec", [("apart16", "exact"), ("apart24", "fast"), ("mixed64", "fast"),
                                       ("furnace", "fast"), ("apart24", "fp64")])
@pytest.mark.parametrize("compat", [0, COMPAT_ALL])
def test_tallies(built_lib, name, prec, compat):
    sc = SCENES[name]()
    total = 400_000 if prec == "fp64" else 3_000_000
    rays = np.full(sc.n, total // (2 * sc.n), np.int64)
    rays[sc.n // 3] += total // 2 + 1
    rays[1::5] = 7
    got = []
    for kw in ({}, {"table_mode": 1}):
        with Tracer(precision=PREC[prec], compat=compat, key1=19, **kw) as t:
            t.set_scene(sc)
            got.append(t.trace(rays)[0])
    assert np.array_equal(got[0], got[1])


@pytest.mark.parametrize("name,prec", [("apart16", "exact"), ("apart24", "fast"), ("mixed64", "fast"),
                                       ("furnace", "fast")])
def test_rays(built_lib, name, prec):
    sc = SCENES[name]()
    first, count = 123_457, 1_100_003
    with Tracer(precision=PREC[prec]) as a, Tracer(precision=PREC[prec], table_mode=1) as b:
        a.set_scene(sc)
        b.set_scene(sc)
        for e in (0, sc.n // 2, sc.n - 1):
            assert np.array_equal(a.trace_rays(e, first, count), b.trace_rays(e, first, count))
