"""The ENO2 right-hand side on fill boxes at the edges of a warp's 8 x 4 patch
and of the walk along z (one row or column, one past a patch, walks of one to
sixteen planes), against the oracle bit for bit."""
import ctypes as C

import numpy as np
import pytest

import qssgpu as Q

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(1, 1, 1), (1, 9, 2), (9, 1, 3), (8, 4, 5), (16, 5, 17), (31, 7, 4), (41, 33, 40),
                               (256, 256, 35), (130, 260, 150)])
@pytest.mark.parametrize("var", [False, True])
def test_eno2_boxes(gpu, oracle, n, var):
    g = Q.make_grid(oracle, n)
    shape = tuple(s + 6 for s in n)[::-1]
    rng = np.random.default_rng(sum(n))
    # smooth along every axis with kinks, so that both candidates of a difference are taken
    phi = sum(0.01 * rng.normal(size=s).cumsum().reshape([-1 if d == a else 1 for a in range(3)])
              for d, s in enumerate(shape)) + 0.002 * rng.normal(size=shape)
    phi[rng.random(shape) < 0.02] = 0.25
    vel, b, u = rng.uniform(-1, 1, shape), rng.uniform(0, 0.05, shape), [rng.uniform(-1, 1, shape) for _ in range(3)]
    if not var:
        vel, b = np.full(1, 0.7), np.full(1, 0.04)
    out = []
    for lib in (gpu, oracle):
        rhs, h = np.zeros(shape), C.c_double(0)
        coef = [Q.dptr(vel), Q.dptr(b)] + ([Q.dptr(a) for a in u] if var else [])
        getattr(lib, "getrhs3d2nd_" if var else "getrhs3d2ndconst_")(
            Q.dptr(phi), *coef, C.byref(h), Q.dptr(rhs), *Q.gb_args(g), *Q.fb_args(g),
            *(Q.dref(g.dx[d]) for d in range(3)))
        Q.check(lib)
        out.append((rhs, h.value))
    assert out[0][1] == out[1][1]
    assert np.array_equal(out[0][0].view(np.int64), out[1][0].view(np.int64))
