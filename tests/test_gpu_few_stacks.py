"""A scene with one pair of rings that touch, among many other surfaces, is traced like the
same scene without stacks: same tallies, and in the same time."""
import numpy as np
import pytest

from rayfactorcl_gb300 import generators
from rayfactorcl_gb300.scene import parse_scene_xml
from rayfactorcl_gb300.tracer import PREC_MIXED, Tracer, segment_stacks

pytestmark = pytest.mark.gpu


def rectangles(n):
    """n large rectangles through one another, and two rings that tile a cylinder."""
    rng = np.random.default_rng(2)
    x = generators._Xml("rectangles")
    for _ in range(n):
        v = rng.normal(size=3)
        x.prim("rectangle", scale=(1.0, 1.0, 1.0), rotate=generators._axis_rotation(v), translate=rng.uniform(-1, 1, 3))
        x.close()
    for i in range(2):
        x.prim("cylinderSurface", small=1.0, scale=(0.3, 0.3, 0.2), translate=(0.0, 0.0, 0.2 * i))
        x.close()
    return parse_scene_xml(x.text())


def test_one_ring_pair(built_lib):
    sc = rectangles(198)
    assert [c for _, c in segment_stacks(sc)] == [2]
    rays = np.full(sc.n, 20_001, np.int64)
    hits, ms = [], []
    for split in (0, 1):
        with Tracer(precision=PREC_MIXED, key1=8, split_stacks=split) as t:
            t.set_scene(sc)
            times = []
            for _ in range(5):
                h = t.trace(rays)[0]
                times.append(t.last_stats()[0])
            hits.append(h)
            ms.append(min(times))
    # (a hit within rounding of the rim between the rings may go to either)
    assert np.abs(hits[0] - hits[1])[:, :198].sum() == 0
    assert ms[0] < 1.15 * ms[1], ms
