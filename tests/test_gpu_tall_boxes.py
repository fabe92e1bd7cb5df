"""Labelling, trapping and percolation on boxes of more planes than a grid's z dimension
holds blocks (65535), against the oracle."""
import ctypes as C

import numpy as np
import pytest

import qssgpu as Q
from qss_cases import options

pytestmark = pytest.mark.gpu

PLANES = 66000


def _volume(oracle, density):
    g = Q.make_grid(oracle, (2, 2, PLANES))
    v = Q.Volume(g)
    rng = np.random.default_rng(3)
    for a in v.arrays.values():
        a[...] = rng.uniform(-1, 1, a.shape) if a.dtype == np.float64 else rng.random(a.shape) < density
    return g, v


@pytest.mark.parametrize("density", [0.1, 0.3, 1.0])
def test_labels(gpu, oracle, density):
    out = []
    for lib in (gpu, oracle):
        g, v = _volume(oracle, density)
        lib.findConnectivity3d(C.byref(v.p), C.byref(g))
        Q.check(lib)
        if lib is gpu:
            lib.qssgpu_release(C.byref(v.p))
        out.append(v["connectivity"])
    assert np.array_equal(*out)


def test_trapping_and_percolation(gpu, oracle):
    out = []
    for lib in (gpu, oracle):
        g, v = _volume(oracle, 0.5)
        o = options(lib)
        lib.getMainInd_new(C.byref(o), C.byref(v.p), C.byref(g))
        diff, connected, percolates = np.zeros(v.shape), np.zeros(v.shape), C.c_int(-1)
        steps = lib.qssgpu_diff_steps if lib is gpu else lib.oracle_diff_steps
        assert steps(Q.dptr(v["phi"]), Q.dptr(v["mask"]), C.byref(g), Q.dptr(diff), Q.dptr(connected),
                     C.byref(percolates)) == 0
        lib.trapComponents_mask(C.byref(v.p), C.byref(g), C.byref(o))
        Q.check(lib)
        if lib is gpu:
            lib.qssgpu_release(C.byref(v.p))
        out.append([v[k] for k in ("phi", "mask_w", "mask_nw", "connectivity", "phi_bin")] +
                   [diff, connected, np.array(percolates.value)])
    for k, (a, b) in enumerate(zip(*out)):
        assert np.array_equal(a, b), k
