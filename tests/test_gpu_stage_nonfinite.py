"""The ENO2 / ENO3 right-hand sides on level sets with infinities, NaNs and values whose
squares or doubles overflow, with half of the voxels' curvature coefficients zero (0 x inf
is NaN there) and with constant coefficients, against the oracle: NaNs at the same voxels,
the same bits elsewhere."""
import ctypes as C

import numpy as np
import pytest

import qssgpu as Q

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("entry", ["getrhs3d2nd_", "getrhs3d3rd_"])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf, 1.7e308, -1e200, 1e150, 2.0 ** 200, 2.0 ** 199, 1e60])
@pytest.mark.parametrize("n", [(9, 5, 11), (33, 6, 18)])
def test_zero_coefficient(gpu, oracle, entry, value, n):
    g = Q.make_grid(oracle, n)
    shape = tuple(s + 6 for s in n)[::-1]
    rng = np.random.default_rng(sum(n))
    phi = 0.04 * rng.normal(size=shape).cumsum(axis=2)
    phi[rng.random(shape) < 0.02] = value
    vel, b = rng.uniform(-1, 1, shape), np.where(rng.random(shape) < 0.5, 0.0, 0.04)
    u = [rng.uniform(-1, 1, shape) for _ in range(3)]
    out = []
    for lib in (gpu, oracle):
        rhs, h = np.zeros(shape), C.c_double(0)
        with np.errstate(all="ignore"):
            getattr(lib, entry)(Q.dptr(phi), Q.dptr(vel), Q.dptr(b), *(Q.dptr(a) for a in u), C.byref(h), Q.dptr(rhs),
                                *Q.gb_args(g), *Q.fb_args(g), *(Q.dref(g.dx[d]) for d in range(3)))
        Q.check(lib)
        out.append(rhs)
    _agree(*out)


def _agree(got, want):
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan), np.argwhere(np.isnan(got) != nan)[:4]
    assert np.array_equal(got.view(np.int64)[~nan], want.view(np.int64)[~nan])


@pytest.mark.parametrize("entry", ["getrhs3d2ndconst_", "getrhs3d3rdconst_"])
@pytest.mark.parametrize("n", [(2, 2, 2), (9, 5, 11), (33, 6, 18)])
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("base,b", [(0.03, 3.0), (1e-94, 0.0)])
def test_doubles_that_overflow(gpu, oracle, entry, n, axis, base, b):
    """M, M, small, M, small along an axis with 2 M infinite: M + small - 2 M is infinite in the
    reference's order of operations although its exact value is not, and decides the choice of
    the difference at the small value between."""
    g = Q.make_grid(oracle, n)
    shape = tuple(s + 6 for s in n)[::-1]
    rng = np.random.default_rng(7 + sum(n) + axis)
    phi = base * rng.uniform(-1, 1, shape)
    view = np.moveaxis(phi, 2 - axis, 0)
    for _ in range(max(2, phi.size // 500)):
        at = tuple(int(rng.integers(3, s - 3)) for s in view.shape)
        for d, m in ((-2, 1.7e308), (-1, 1.7e308), (1, 1.7e308)):
            view[(at[0] + d, *at[1:])] = m
    out = []
    for lib in (gpu, oracle):
        rhs, h = np.zeros(shape), C.c_double(0)
        with np.errstate(all="ignore"):
            getattr(lib, entry)(Q.dptr(phi), Q.dref(0.7), Q.dref(b), C.byref(h), Q.dptr(rhs), *Q.gb_args(g),
                                *Q.fb_args(g), *(Q.dref(g.dx[d]) for d in range(3)))
        Q.check(lib)
        out.append(rhs)
    _agree(*out)
