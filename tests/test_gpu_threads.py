"""Calls of several host threads at the same time."""
import ctypes as C
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_mie_calls_of_different_sizes():
    """Mie series of one, some and many thousand orders from three threads:
    each needs its own amount of shared memory, and none may lower what
    another has asked for."""
    from jscat import lib as L
    lib = L.load()
    lib.jsc_mie_eval.restype = C.c_int
    dp = C.POINTER(C.c_double)

    def run(size):
        x, nr, ni = np.full(4, size), np.full(4, 1.31), np.full(4, 0.01)
        out = np.empty((4, 183))
        st = lib.jsc_mie_eval(0, 4, *[a.ctypes.data_as(dp) for a in (x, nr, ni)], out.ctypes.data_as(dp))
        return st, out

    sizes = (1250.0, 2400.0, 4500.0)
    want = [run(v) for v in sizes]
    assert all(st == 0 for st, _ in want)
    bad = []

    def loop(i):
        for _ in range(150):
            st, out = run(sizes[i])
            if st or not np.array_equal(out, want[i][1]):
                bad.append((sizes[i], st))

    threads = [threading.Thread(target=loop, args=(i,)) for i in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
