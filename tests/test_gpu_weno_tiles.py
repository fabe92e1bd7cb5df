"""The WENO5 tiles at the edges of their geometry (4 lines x 64 positions, and
the shorter tiles of small grids) and of their arithmetic's range (flat parts,
exact zeros, and differences so large or small that a tile takes the native
path), against the oracle's right-hand side bit for bit."""
import ctypes as C

import numpy as np
import pytest

import qssgpu as Q

pytestmark = pytest.mark.gpu


def _phi(kind, shape, seed):
    rng = np.random.default_rng(seed)
    z, y, x = np.meshgrid(*(np.arange(s) for s in shape), indexing="ij")
    smooth = 0.04 * np.sqrt((x - 3.3) ** 2 + (y - 1.7) ** 2 + (z + 2.1) ** 2)
    if kind == "smooth":
        return smooth + 1e-3 * rng.uniform(-1, 1, shape)
    if kind == "flat":  # constant but for a bump, exactly linear parts
        p = np.full(shape, -0.8)
        p[x > shape[2] // 2] += 0.03125 * (x - shape[2] // 2)[x > shape[2] // 2]
        return p
    scale = {"huge": 1e25, "tiny": 1e-75}[kind]
    p = smooth.copy()
    hit = rng.uniform(0, 1, shape) < 0.02
    p[hit] = scale * rng.uniform(-1, 1, hit.sum())
    if kind == "tiny":
        p[:, :, : shape[2] // 2] = scale * rng.uniform(-1, 1, (shape[0], shape[1], shape[2] // 2))
    return p


@pytest.mark.parametrize("kind", ["smooth", "flat", "huge", "tiny"])
@pytest.mark.parametrize("n", [(2, 2, 2), (64, 5, 3), (65, 4, 7), (129, 3, 6), (5, 67, 9), (6, 7, 131)])
@pytest.mark.parametrize("variant", [-1, 3, 4])
def test_weno_tiles(gpu, oracle, n, kind, variant):
    g = Q.make_grid(oracle, n)
    shape = tuple(s + 6 for s in n)[::-1]
    phi = _phi(kind, shape, seed=sum(n))
    rng = np.random.default_rng(11)
    vel, b = rng.uniform(-1, 1, shape), rng.uniform(0, 0.05, shape)
    u = [rng.uniform(-1, 1, shape) for _ in range(3)]
    prev = gpu.qssgpu_set_axis_variant(variant)
    try:
        out = []
        for lib in (gpu, oracle):
            rhs, h = np.zeros(shape), C.c_double(0)
            lib.getrhs3d5th_(Q.dptr(phi), Q.dptr(vel), Q.dptr(b), *(Q.dptr(a) for a in u), C.byref(h), Q.dptr(rhs),
                             *Q.gb_args(g), *Q.fb_args(g), *(Q.dref(g.dx[d]) for d in range(3)))
            Q.check(lib)
            out.append((rhs, h.value))
    finally:
        gpu.qssgpu_set_axis_variant(prev)
    assert out[0][1] == out[1][1]
    assert np.array_equal(out[0][0], out[1][0], equal_nan=True), np.argwhere(out[0][0] != out[1][0])[:4]
