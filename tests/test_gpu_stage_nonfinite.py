"""The ENO2 / ENO3 right-hand sides on level sets with infinities, NaNs and values whose
squares overflow, half of the voxels with a zero curvature coefficient (0 x inf is NaN
there), against the oracle: NaNs at the same voxels, the same bits elsewhere."""
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
    nan = np.isnan(out[1])
    assert np.array_equal(np.isnan(out[0]), nan), np.argwhere(np.isnan(out[0]) != nan)[:4]
    assert np.array_equal(out[0].view(np.int64)[~nan], out[1].view(np.int64)[~nan])
