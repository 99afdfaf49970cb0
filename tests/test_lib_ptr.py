"""The address of an array, as the library's calls take it, keeps the array alive."""
import gc
import weakref

import numpy as np

from rayfactorcl_gb300._lib import ptr


def test_pointer_keeps_its_array():
    a = np.arange(1000)
    dead = weakref.ref(a)
    p = ptr(a)
    assert p.value == a.ctypes.data
    del a
    gc.collect()
    assert dead() is not None
    del p
    gc.collect()
    assert dead() is None
    assert ptr(None) is None
