"""The cell masks (rf_masks.cu) leave out no surface a ray can hit: a traced scene with
masks gives the tallies of the allocation-free call, which culls with per-packet bounds
instead.  Sizes at the edges of the builder's words of 32 surfaces, of its two launch
shapes, of the smallest masked scene, and elongated surfaces (sphere chains)."""
import ctypes

import numpy as np
import pytest

from rayfactorcl_gb300 import _lib, generators
from rayfactorcl_gb300.scene import FRUSTUM, PRIM_DTYPE
from rayfactorcl_gb300.tracer import PREC_MIXED, REF_KEY1, Tracer

pytestmark = pytest.mark.gpu


def scene(n, long=False):
    c = np.floor(np.array([16, 16, 12, 10, 10], float) / 64 * n).astype(int)
    c[0] += n - c.sum()
    sc = generators.mixed_scene(seed=n, total_rays=4, counts=tuple(int(x) for x in c)).scene
    if long:  # axes stretched five times: z column of m, row 2 of invm
        for p in sc.primitives[: c[0] + c[1]]:
            p["m"][2::4] *= np.float32(5.0)
            p["invm"][8:12] /= np.float32(5.0)
        sc.primitives["util1"][np.flatnonzero(sc.primitives["type"] == FRUSTUM)[:1]] = 1.0  # no finite patch
    return sc


@pytest.mark.parametrize("n,long", [(17, False), (31, False), (32, True), (33, False), (64, True), (65, False),
                                    (180, True), (200, False), (512, False)])
def test_masks_against_packet_bounds(built_lib, n, long):
    torch = pytest.importorskip("torch")
    sc = scene(n, long)
    rays = np.full(n, max(400, 400_000 // n) | 1, np.int64)
    with Tracer(precision=PREC_MIXED) as t:
        t.set_scene(sc)
        ref, _ = t.trace(rays)
    prims = np.ascontiguousarray(sc.primitives, PRIM_DTYPE)
    hits = torch.zeros(n * n, dtype=torch.int64, device="cuda:0")
    status = _lib.load().rf_trace_mixed_noalloc(_lib.ptr(prims), n, _lib.ptr(rays), 0, REF_KEY1, ctypes.c_float(1e-3),
                                                ctypes.c_void_p(hits.data_ptr()), None)
    assert status == _lib.RF_OK
    torch.cuda.synchronize()
    assert np.array_equal(hits.cpu().numpy().reshape(n, n), ref)
