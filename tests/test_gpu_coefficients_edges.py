"""Coefficients from the mask (normal velocity, curvature coefficient, advection
velocity and their CFL maxima) over the voxels their kernel treats apart: pore,
solid and smoothing band, the band's two ends, a flat mask, gradients and
masks out of the integer range, infinities and NaN, and fill boxes around a
block's 1024 voxels, against the oracle bit for bit."""
import ctypes as C

import numpy as np
import pytest

import qssgpu as Q

pytestmark = pytest.mark.gpu


def _fields(kind, g, shape, seed):
    rng = np.random.default_rng(seed)
    dx = g.dx[0]
    m = rng.uniform(-6, 6, shape) * dx
    grad = [rng.normal(0, 0.6, shape) for _ in range(3)]
    theta = rng.uniform(-1.0, 2.0, shape)
    if kind == "pore":
        m = -np.abs(m) - 2 * dx
    elif kind == "solid":
        m = np.abs(m) + 2 * dx
        for q in grad:
            q[rng.random(shape) < 0.3] = 0.0
    elif kind == "band":
        m = np.clip(m, -1.5 * dx, 1.5 * dx)
    elif kind == "wild":
        eps = 1.5 * dx
        for a, vals in ((m, (0.0, -0.0, eps, -eps, np.nextafter(eps, 1), np.nextafter(-eps, -1), 1e200, -1e200, 5e-324,
                            -np.inf, np.inf, np.nan)),
                        *((q, (0.0, -0.0, 1e-200, -5e-324, 1e160, np.inf, np.nan)) for q in grad),
                        (theta, (0.0, -0.0, 1e9, -3e30, np.pi / 2, np.inf))):
            pick = rng.integers(0, 60, shape)
            for n, val in enumerate(vals):
                a[pick == n] = val
    return m, grad, theta


@pytest.mark.parametrize("kind", ["mixed", "pore", "solid", "band", "wild"])
@pytest.mark.parametrize("n", [(1, 1, 1), (16, 8, 8), (31, 3, 11), (5, 41, 5), (37, 29, 3)])
@pytest.mark.parametrize("a0,b", [(1.1, 0.04), (0.0, -0.0), (-0.7, -0.04)])
def test_coefficient_edges(gpu, oracle, kind, n, a0, b):
    g = Q.make_grid(oracle, n)
    shape = tuple(s + 6 for s in n)[::-1]
    m, (gx, gy, gz), theta = _fields(kind, g, shape, seed=sum(n))
    res = []
    for lib in (gpu, oracle):
        vb, vx, vy, vz, vn, v0, vt = (np.full(shape, 7.0) for _ in range(7))
        bm, um = C.c_double(0), C.c_double(0)
        box = (*Q.gb_args(g), *Q.fb_args(g), Q.dref(g.dx[0]))
        grad = (Q.dptr(m), Q.dptr(gx), Q.dptr(gy), Q.dptr(gz))
        lib.setvarcurvadv3d_(*grad, Q.dptr(vb), Q.dptr(vx), Q.dptr(vy), Q.dptr(vz), C.byref(bm), C.byref(um),
                             Q.dref(b), *box)
        lib.setvarnorm3d_(*grad, Q.dptr(vn), Q.dref(a0), Q.dref(0.6981), *box)
        lib.setvarnorm3d_(*grad, Q.dptr(v0), Q.dref(a0), Q.dref(0.0), *box)
        lib.setvarnorm3dtheta_(*grad, Q.dptr(vt), Q.dref(a0), Q.dptr(theta), *box)
        Q.check(lib)
        res.append([vb, vx, vy, vz, vn, v0, vt, np.array([bm.value, um.value])])
    for q, (x, y) in enumerate(zip(*res)):
        assert np.array_equal(x, y, equal_nan=True), q
        if q == 7:  # which of +0 and -0 is the larger is open
            continue
        zero = x == 0
        assert np.array_equal(np.signbit(x[zero]), np.signbit(y[zero])), q
