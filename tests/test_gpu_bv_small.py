"""Scenes of 13 to 16 surfaces with bounding surfaces in mixed precision: the walk's own
tests are counted, and the surfaces that a ray cannot hit are left out."""
import numpy as np
import pytest

from rayfactorcl_gb300.scene import BV_DTYPE, SPHERE
from rayfactorcl_gb300.tracer import PREC_MIXED, Tracer

from test_gpu_culled import mixed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [13, 16, 24])
def test_children_of_the_nearer_shell_only(built_lib, n):
    """Two bounding spheres around everything: every ray's nearest is the smaller one,
    whose children are tested once, and the other's never."""
    sc = mixed(n, seed=3)
    h = n // 2
    b = np.zeros(2, BV_DTYPE)
    b["type"], b["util2"] = SPHERE, -1.0
    b["objStartIndex"], b["objEndIndex"] = (0, h), (h, n)
    for k, r in enumerate((30.0, 50.0)):
        b["invm"][k] = (np.eye(4)[:3] / r).astype(np.float32).ravel()
    sc.bounding_volumes = b
    rays = np.arange(1, n + 1, dtype=np.int64) * 1001
    got = []
    for count in (False, True):
        with Tracer(precision=PREC_MIXED, work_counts=count) as t:
            t.set_scene(sc)
            got.append((t.trace(rays, use_bv=True)[0], t.work_counts()))
    assert np.array_equal(got[0][0], got[1][0])
    assert got[0][1].sum() == 0
    w = got[1][1][:6].astype(np.int64)
    types = sc.primitives["type"]
    planar = np.isin(types, (3, 4, 5))
    most = np.zeros(6, np.int64)
    for j in range(h):  # a planar emitter is not tested by its own rays
        most[types[j]] += rays.sum() - (rays[j] if planar[j] else 0)
    assert (w <= most).all() and w.sum() > 0  # spheres leave some out


def test_sixteen_cost_no_more_than_twentyfour(built_lib):
    """Far-apart surfaces under one shell: most of them are left out."""
    ms = {}
    for n in (16, 24):
        sc = mixed(n, seed=3)
        b = np.zeros(1, BV_DTYPE)
        b["type"], b["objEndIndex"], b["util2"] = SPHERE, n, -1.0
        b["invm"][0] = (np.eye(4)[:3] / 30.0).astype(np.float32).ravel()
        sc.bounding_volumes = b
        rays = np.full(n, 12_000_000 // n, np.int64)
        with Tracer(precision=PREC_MIXED) as t:
            t.set_scene(sc)
            times = []
            for _ in range(4):
                t.trace(rays, use_bv=True)
                times.append(t.last_stats()[0])
            ms[n] = min(times)
    assert ms[16] < 1.4 * ms[24], ms
