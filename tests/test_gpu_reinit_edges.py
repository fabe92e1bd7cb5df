"""The reinitialisation sweeps on fill boxes at the edges of a warp's 8 x 4
patch and of the walk along z, over fields that take every path of the kernel
(signed distances, a constant field, exact zeros, values whose differences are
out of the straight-line range), against the oracle bit for bit."""
import ctypes as C

import numpy as np
import pytest

import qssgpu as Q
import synthetic as S
from qss_cases import options

pytestmark = pytest.mark.gpu


def _field(kind, shape, g, seed):
    rng = np.random.default_rng(seed)
    nz, ny, nx = shape
    z, y, x = np.meshgrid(*(np.arange(s) for s in shape), indexing="ij")
    d = 0.04 * (np.sqrt((x - 0.4 * nx) ** 2 + (y - 0.5 * ny) ** 2 + (z - 0.6 * nz) ** 2) - 0.3 * max(shape))
    if kind == "distance":
        return d + 0.01 * rng.uniform(-1, 1, shape)
    if kind == "flat":
        return np.full(shape, -0.8)
    if kind == "plane":  # exactly equal differences along x
        return 0.03125 * (x - nx // 2).astype(float)
    wild = rng.uniform(-1, 1, shape)
    pick = rng.integers(0, 40, shape)
    for n, val in enumerate((0.0, -0.0, 5e-324, -1e-310, 1e-5, -1e-5, 1e140, -1e35, 2.0 ** -300)):
        wild[pick == n] = val
    return wild


@pytest.mark.parametrize("kind", ["distance", "flat", "plane", "wild"])
@pytest.mark.parametrize("n", [(2, 2, 2), (8, 4, 16), (9, 5, 17), (7, 3, 15), (33, 13, 6)])
@pytest.mark.parametrize("iters", [1, 2, 5])
def test_reinit_edges(gpu, oracle, n, kind, iters):
    g = Q.make_grid(oracle, n)
    shape = tuple(s + 6 for s in n)[::-1]
    f = _field(kind, shape, g, seed=sum(n))
    out = []
    for lib in (gpu, oracle):
        a = np.ascontiguousarray(f.copy())
        o = options(lib)
        o.tmax_r = (iters - 0.5) * 0.5 * g.dx[0]
        with np.errstate(all="ignore"):
            lib.reinitializeSubcellFix3d(Q.dptr(a), C.byref(g), C.byref(o))
        Q.check(lib)
        out.append(a)
    assert np.array_equal(out[0], out[1], equal_nan=True), np.argwhere(out[0] != out[1])[:4]


@pytest.mark.parametrize("iters", [0, 1, 2, 3])
def test_reinitialize_mask_buffers(gpu, oracle, iters):
    """qss_reinitialize_mask leaves the distances, the initial mask, the last
    right-hand side and the last iterate where the reference does, for odd and
    even numbers of sweeps."""
    n = (19, 6, 10)
    g = Q.make_grid(oracle, n)
    m = S.overlapping(n, radius_vox=3.0, porosity=0.45, seed=3).mask()
    res = []
    for lib in (gpu, oracle):
        v = Q.Volume(g)
        rng = np.random.default_rng(5)
        for k in ("scratch1", "scratch2", "lse_rhs", "phi_next"):
            v[k][...] = rng.uniform(-2, 2, v.shape)
        v["mask"][...] = m
        o = options(lib)
        o.tmax_r = (iters - 0.5) * 0.5 * g.dx[0]
        if lib is gpu:
            lib.qss_reinitialize_mask(C.byref(v.p), C.byref(g), C.byref(o))
            Q.check(lib)
        else:
            _reference_mask_reinit(lib, v, g, iters)
        res.append(v)
    for k in ("mask", "scratch1", "scratch2", "lse_rhs", "phi_next"):
        assert np.array_equal(res[0][k], res[1][k]), k


def _reference_mask_reinit(lib, v, g, iters):
    """qss_general_util.c:261-306 through the oracle's kernels."""
    dxs = [Q.dref(g.dx[d]) for d in range(3)]
    v["scratch2"][...] = v["mask"]
    lib.qss3dcomputedistanceforsubcellfix_(Q.dptr(v["scratch1"]), Q.dptr(v["scratch2"]), *Q.gb_args(g),
                                           *Q.fb_args(g), *dxs)
    for _ in range(iters):
        lib.qss3dcomputereinitializationeqnrhssubcellfixorder1_(
            Q.dptr(v["lse_rhs"]), Q.dptr(v["mask"]), *Q.gb_args(g), Q.dptr(v["scratch2"]), Q.dptr(v["scratch1"]),
            *Q.fb_args(g), *dxs)
        lib.qss3drk1step_(Q.dptr(v["phi_next"]), *Q.gb_args(g), Q.dptr(v["mask"]), *Q.gb_args(g),
                          Q.dptr(v["lse_rhs"]), *Q.gb_args(g), *Q.fb_args(g), Q.dref(0.5 * g.dx[0]))
        lib.signedLinearExtrapolationBCqss(Q.dptr(v["phi_next"]), C.byref(g), 9)
        v["mask"][...] = v["phi_next"]
