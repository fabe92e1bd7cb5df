"""Single-kernel entry points from several host threads at once, with sizes that
change from call to call: their device arrays come from one pool, and every
result equals the one of the same call alone."""
import ctypes as C
import threading

import numpy as np
import pytest

import qssgpu as Q

pytestmark = pytest.mark.gpu


def _rhs(lib, g, phi, vel, b):
    rhs, h = np.zeros(phi.shape), C.c_double(0)
    lib.getrhs3d5th_(Q.dptr(phi), Q.dptr(vel), Q.dptr(b), Q.dptr(vel), Q.dptr(b), Q.dptr(vel), C.byref(h),
                     Q.dptr(rhs), *Q.gb_args(g), *Q.fb_args(g), *(Q.dref(g.dx[d]) for d in range(3)))
    return rhs


def test_concurrent_calls(gpu, oracle):
    work = []
    for k, n in enumerate([(40, 33, 27), (17, 9, 12), (64, 31, 18), (25, 25, 25)]):
        g = Q.make_grid(oracle, n)
        shape = tuple(s + 6 for s in n)[::-1]
        rng = np.random.default_rng(k)
        a = [0.04 * rng.standard_normal(shape).cumsum(axis=2), rng.uniform(-1, 1, shape), rng.uniform(0, 0.05, shape)]
        work.append((g, *a, _rhs(gpu, g, *a)))
    bad = []

    def loop(start):
        for r in range(12):
            g, phi, vel, b, want = work[(start + r) % len(work)]
            if not np.array_equal(_rhs(gpu, g, phi, vel, b), want) or gpu.qssgpu_last_error():
                bad.append((start, r))

    threads = [threading.Thread(target=loop, args=(s,)) for s in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
    Q.check(gpu)
    # giving the pool's memory back leaves the next call right
    v = Q.Volume(work[1][0])
    gpu.qssgpu_release(C.byref(v.p))
    assert np.array_equal(_rhs(gpu, *work[0][:4]), work[0][4])
