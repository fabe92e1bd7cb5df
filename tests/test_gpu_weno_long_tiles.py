"""The WENO5 tiles where they are longest: boxes large enough for tiles of 64 positions
(full ones and uneven ones of 34 to 63), with sides that are no multiple of a tile, the
three axes in one launch and in three, over smooth fields and over values that send
single tiles down the native path, against the oracle's right-hand side bit for bit."""
import ctypes as C

import numpy as np
import pytest

import qssgpu as Q
from test_gpu_weno_tiles import _phi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,kind", [((129, 67, 131), k) for k in ("smooth", "flat", "huge", "tiny")] +
                         [((127, 65, 191), k) for k in ("smooth", "huge")] +
                         [((97, 161, 83), k) for k in ("smooth", "tiny")] + [((131, 197, 179), "huge")])
def test_long_tiles(gpu, oracle, n, kind):
    g = Q.make_grid(oracle, n)
    shape = tuple(s + 6 for s in n)[::-1]
    phi = _phi(kind, shape, seed=sum(n))
    if kind in ("huge", "tiny"):  # most tiles on the fast path, some voxels' tiles not
        phi = np.where(np.random.default_rng(2).random(shape) < 2e-5, phi, _phi("smooth", shape, seed=sum(n)))
    rng = np.random.default_rng(11)
    vel, b = rng.uniform(-1, 1, shape), rng.uniform(0, 0.05, shape)
    u = [rng.uniform(-1, 1, shape) for _ in range(3)]
    out = []
    for lib in (gpu, oracle):
        rhs, h = np.zeros(shape), C.c_double(0)
        lib.getrhs3d5th_(Q.dptr(phi), Q.dptr(vel), Q.dptr(b), *(Q.dptr(a) for a in u), C.byref(h), Q.dptr(rhs),
                         *Q.gb_args(g), *Q.fb_args(g), *(Q.dref(g.dx[d]) for d in range(3)))
        Q.check(lib)
        out.append((rhs, h.value))
    assert out[0][1] == out[1][1]
    nan = np.isnan(out[1][0])
    assert np.array_equal(np.isnan(out[0][0]), nan)
    bad = np.argwhere((out[0][0].view(np.int64) != out[1][0].view(np.int64)) & ~nan)
    assert not len(bad), bad[:4]
