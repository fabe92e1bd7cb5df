"""The straight-line stage arithmetic (Godunov term, curvature, advection of
every scheme) where its operand tests decide: flat and exactly linear parts,
zero velocities and coefficients, voxels at rest, differences out of its range,
on ragged boxes, against the oracle's right-hand sides bit for bit."""
import ctypes as C

import numpy as np
import pytest

import qssgpu as Q
from test_gpu_weno_tiles import _phi

pytestmark = pytest.mark.gpu

ENTRIES = {"getrhs3d2ndconst_": False, "getrhs3d3rdconst_": False, "getrhs3d2nd_": True, "getrhs3d3rd_": True,
           "getrhs3d5th_": True}


@pytest.mark.parametrize("entry", list(ENTRIES))
@pytest.mark.parametrize("kind", ["smooth", "flat", "huge", "tiny"])
@pytest.mark.parametrize("n", [(2, 2, 2), (9, 5, 11), (33, 6, 8)])
@pytest.mark.parametrize("still", [0.0, 0.5])
def test_rhs_operand_ranges(gpu, oracle, entry, kind, n, still):
    g = Q.make_grid(oracle, n)
    shape = tuple(s + 6 for s in n)[::-1]
    phi = _phi(kind, shape, seed=3 + sum(n))
    rng = np.random.default_rng(12)
    drop = rng.uniform(0, 1, shape) < still

    def field(lo, hi):
        return np.where(drop, 0.0, rng.uniform(lo, hi, shape))

    vel, b, u = field(-1, 1), field(0, 0.05), [field(-1, 1) for _ in range(3)]
    vel[rng.uniform(0, 1, shape) < 0.1] = 5e-6
    if not ENTRIES[entry]:
        vel, b = np.full(1, 0.7), np.full(1, 0.0 if still else 0.04)
    out = []
    for lib in (gpu, oracle):
        rhs, h = np.zeros(shape), C.c_double(0)
        coef = [Q.dptr(vel), Q.dptr(b)] + ([Q.dptr(a) for a in u] if ENTRIES[entry] else [])
        getattr(lib, entry)(Q.dptr(phi), *coef, C.byref(h), Q.dptr(rhs), *Q.gb_args(g), *Q.fb_args(g),
                            *(Q.dref(g.dx[d]) for d in range(3)))
        Q.check(lib)
        out.append((rhs, h.value))
    assert out[0][1] == out[1][1]
    bad = np.argwhere((out[0][0].view(np.int64) != out[1][0].view(np.int64)) & ~np.isnan(out[1][0]))
    assert np.array_equal(np.isnan(out[0][0]), np.isnan(out[1][0])) and not len(bad), bad[:4]
