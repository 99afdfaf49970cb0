"""The narrow kernel (rf_narrow.cuh: few rays, a ray's surfaces split over warps)
against the kernels that take the same rays when a launch shape is pinned; the
results must be equal bit for bit."""
import numpy as np
import pytest

from rayfactorcl_gb300 import generators
from rayfactorcl_gb300.tracer import COMPAT_ALL, PREC_EXACT, PREC_FAST, PREC_FP64, PREC_MIXED, Tracer

from test_gpu_culled import mixed

pytestmark = pytest.mark.gpu
PREC = {"exact": PREC_EXACT, "fast": PREC_FAST, "fp64": PREC_FP64, "mixed": PREC_MIXED}
SCENES = {
    "enclosure": lambda: generators.enclosure3(4).scene,
    "mixed13": lambda: mixed(13), "mixed40": lambda: mixed(40), "mixed64": lambda: mixed(64),
    "mixed201": lambda: mixed(201), "mixed1024": lambda: mixed(1024),  # the largest
    "mixed1025": lambda: mixed(1025),
    "furnace": lambda: generators.furnace_scene(4).scene,  # parts end inside its stacks
    "stress": lambda: generators.precision_stress(4).scene,  # FP64 re-evaluations
}


def pinned(prec):
    return {"batched_grid": 40} if prec == "mixed" else {"table_mode": 1}


# 1: most chunks hold one ray; 9000 to 70000: splits of 8 to 1
@pytest.mark.parametrize("total", [1, 9_000, 33_000, 70_000])
@pytest.mark.parametrize("prec", sorted(PREC))
@pytest.mark.parametrize("name", sorted(SCENES))
def test_narrow_tallies_equal(built_lib, name, prec, total):
    sc = SCENES[name]()
    if prec == "fp64":
        if sc.n > 64:
            pytest.skip("not taken")
        total = min(total, 40_000)
    rng = np.random.Generator(np.random.PCG64(total))
    rays = np.floor(rng.uniform(0.2, 1.8, size=sc.n) * total / sc.n).astype(np.int64) + 1
    rays[-1] = 0
    got = []
    for kw in ({}, pinned(prec)):
        with Tracer(precision=PREC[prec], compat=COMPAT_ALL if total == 33_000 else 0, key1=5, **kw) as t:
            t.set_scene(sc)
            got.append(t.trace(rays)[0])
    assert np.array_equal(got[0], got[1])


@pytest.mark.parametrize("prec", sorted(PREC))
@pytest.mark.parametrize("name", ["mixed40", "furnace", "stress"])
def test_narrow_rays_equal(built_lib, name, prec):
    """Per ray, ranges that start and end inside a draw."""
    sc = SCENES[name]()
    with Tracer(precision=PREC[prec]) as a, Tracer(precision=PREC[prec], **pinned(prec)) as b:
        a.set_scene(sc)
        b.set_scene(sc)
        for e, first, count in ((0, 3, 1), (sc.n // 2, 123_457, 2_001), (sc.n - 1, 1_000_002, 20_003)):
            assert np.array_equal(a.trace_rays(e, first, count), b.trace_rays(e, first, count))
