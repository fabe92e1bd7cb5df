"""Reinitialisation sweeps whose threads walk several planes (5, 8 and 16), on sides that
are no multiple of the 32 x 4 patch and with a shorter last walk, and two masks swept in
one launch (trapping), against the oracle bit for bit."""
import ctypes as C

import numpy as np
import pytest

import qssgpu as Q
from qss_cases import clone, options, pack_case, prepare_model
from test_gpu_reinit_edges import _field

pytestmark = pytest.mark.gpu


def _same(a, b):
    return np.array_equal(np.isnan(a), np.isnan(b)) and np.array_equal(a.view(np.int64)[~np.isnan(a)],
                                                                       b.view(np.int64)[~np.isnan(b)])


@pytest.mark.parametrize("kind", ["distance", "plane", "wild"])
@pytest.mark.parametrize("n,iters", [((130, 67, 152), 1), ((130, 67, 152), 4), ((257, 259, 37), 3), ((193, 131, 170), 2)])
def test_walks(gpu, oracle, n, iters, kind):
    g = Q.make_grid(oracle, n)
    f = _field(kind, tuple(s + 6 for s in n)[::-1], g, seed=sum(n))
    out = []
    for lib in (gpu, oracle):
        a = np.ascontiguousarray(f.copy())
        o = options(lib)
        o.tmax_r = (iters - 0.5) * 0.5 * g.dx[0]
        with np.errstate(all="ignore"):
            lib.reinitializeSubcellFix3d(Q.dptr(a), C.byref(g), C.byref(o))
        Q.check(lib)
        out.append(a)
    assert _same(*out), np.argwhere(out[0] != out[1])[:4]


def test_two_masks_at_once(gpu, oracle):
    """One curvature step with trapping: walks of 10 planes for the two masks, of 5 for phi."""
    g, v = pack_case(oracle, (130, 67, 152), seed=5, radius=5.0)
    out = []
    for lib in (gpu, oracle):
        w = clone(v)
        o = options(lib, tmax=0.004, tplot=0.004)
        prepare_model(lib, o, w, o.a)
        lib.constCurvModel3dNoVar(C.byref(o), C.byref(w.p), C.byref(g), None, o.a)
        Q.check(lib)
        if lib is gpu:
            lib.qssgpu_release(C.byref(w.p))
        out.append(w)
    for k in ("phi", "phi_prev", "phi_next", "mask_w", "mask_nw"):
        assert _same(out[0][k], out[1][k]), k
    assert np.array_equal(out[0]["connectivity"], out[1]["connectivity"])
