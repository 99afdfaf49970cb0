"""The small-scene mixed kernel's pair tests (two rays a lane in packed FP32) against
its scalar ones, which eight rays a thread takes: equal tallies and FP64 re-evaluations."""
import numpy as np
import pytest

from rayfactorcl_gb300 import generators
from rayfactorcl_gb300.scene import DISC, RECTANGLE
from rayfactorcl_gb300.tracer import COMPAT_SPHERE, PREC_MIXED, Tracer

from test_gpu_culled import mixed

pytestmark = pytest.mark.gpu


def with_rectangles():
    sc = mixed(16, seed=21)
    p = sc.primitives
    p["type"][p["type"] == DISC] = RECTANGLE
    return sc


@pytest.mark.parametrize("compat", [0, COMPAT_SPHERE])
@pytest.mark.parametrize("scene", ["5", "6", "16", "rectangles", "stress"])  # pairs from 6 surfaces on
def test_pairs_equal_single_rays(built_lib, scene, compat):
    sc = (with_rectangles() if scene == "rectangles" else
          generators.precision_stress(4).scene if scene == "stress" else mixed(int(scene), seed=9))
    rng = np.random.default_rng(4)
    rays = rng.integers(60_000, 400_000, sc.n).astype(np.int64)  # odd remainders of a draw and of a chunk
    got = []
    for rpt in (0, 8):
        with Tracer(precision=PREC_MIXED, rays_per_thread=rpt, compat=compat, key1=3) as t:
            t.set_scene(sc)
            got.append((t.trace(rays)[0], t.refined_count()))
    assert np.array_equal(got[0][0], got[1][0])
    assert got[0][1] == got[1][1]
