"""One context per host thread on a shared GPU: calls whose launches need different
amounts of shared memory, in flight at once from several threads, all succeed."""
import threading

import numpy as np
import pytest

from rayfactorcl_gb300.tracer import PREC_EXACT, PREC_MIXED, Tracer

from test_gpu_culled import mixed

pytestmark = pytest.mark.gpu


def trace(prec, n, total):
    sc = mixed(n)
    rays = np.full(sc.n, total // n, np.int64)
    t = Tracer(precision=prec, key1=9)
    t.set_scene(sc)

    def call():
        for _ in range(30):  # launches one after another, not one a read-back
            t.trace_async(rays)
        return t.results()[0]

    return call


def smooth(n):
    rng = np.random.default_rng(n)
    F = rng.uniform(0.5, 1.5, (n, n))
    F /= F.sum(axis=1, keepdims=True)
    A, t = rng.uniform(1.0, 2.0, n), Tracer()
    return lambda: t.smooth_F(F, A)[0]


CALLS = {
    # chunks of 1024 and of 1280 draws
    "culled": [(trace, PREC_EXACT, 24, 410_000), (trace, PREC_EXACT, 24, 3_000_000)],
    # tables of 45 and of 64 KB
    "narrow": [(trace, PREC_EXACT, 700, 20_000), (trace, PREC_EXACT, 1000, 20_000)],
    "narrow-mixed": [(trace, PREC_MIXED, 700, 20_000), (trace, PREC_MIXED, 1000, 20_000)],
    # rows of 50 and of 104 KB a block
    "smooth": [(smooth, 900), (smooth, 1300)],
}


@pytest.mark.parametrize("name", sorted(CALLS))
def test_threads_share_the_gpu(built_lib, name):
    calls = [f(*a) for f, *a in CALLS[name] * 2]  # four contexts, four threads
    want = [c() for c in calls]
    errors = []

    def work(i):
        try:
            for _ in range({"smooth": 500, "culled": 120}.get(name, 40)):
                got = calls[i]()
                assert np.array_equal(got, want[i])
        except Exception as ex:  # reported by the main thread
            errors.append(repr(ex))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
