"""The FP64 culled kernel's FP32 look before a test: tallies equal to the plain kernel's
where its error bounds matter (grazing rays, thin and flat surfaces, far from the origin,
every type) and where it must stay out of the way."""
import numpy as np
import pytest

from rayfactorcl_gb300 import generators
from rayfactorcl_gb300.scene import DISC, RECTANGLE
from rayfactorcl_gb300.tracer import COMPAT_SPHERE, PREC_FP64, Tracer

from test_gpu_culled import mixed, odd_scene

pytestmark = pytest.mark.gpu


def rectangles():
    sc = mixed(48, seed=31)
    sc.primitives["type"][sc.primitives["type"] == DISC] = RECTANGLE
    return sc


SCENES = {"enclosure": lambda: generators.enclosure3(4).scene, "mixed9": lambda: mixed(9),
          "mixed17": lambda: mixed(17), "mixed120": lambda: mixed(120), "rectangles": rectangles,
          "odd": odd_scene, "stress": lambda: generators.precision_stress(4).scene}


@pytest.mark.parametrize("compat", [0, COMPAT_SPHERE])
@pytest.mark.parametrize("name", sorted(SCENES))
def test_fp32_look_keeps_every_hit(built_lib, name, compat):
    sc = SCENES[name]()
    rays = np.full(sc.n, 600_003 // sc.n, np.int64)
    got = []
    for kw in ({}, {"table_mode": 1}):
        with Tracer(precision=PREC_FP64, key1=41, compat=compat, **kw) as t:
            t.set_scene(sc)
            got.append(t.trace(rays)[0])
    assert np.array_equal(got[0], got[1])
