"""26-connected labels on boxes at the edges of the 32 x 8 x 8 tiles, for random
images of every density and for images whose components wind through many tiles
or touch only diagonally, against the oracle."""
import ctypes as C

import numpy as np
import pytest

import qssgpu as Q

pytestmark = pytest.mark.gpu


def _image(kind, shape, rng):
    z, y, x = np.meshgrid(*(np.arange(s) for s in shape), indexing="ij")
    if kind == "diagonal":  # chains that touch only at corners
        return ((x + y + z) % 4 == 0) & ((x - y) % 2 == 0)
    if kind == "comb":  # one component folded through all tiles
        return (x % 4 == 0) | ((y == np.where((x // 4) % 2 == 0, 0, shape[1] - 1)) & (z == 0))
    if kind == "sheets":  # two interleaved combs
        return ((x + 2 * (y // 3)) % 6 < 2) & (z % 5 < 4)
    return rng.uniform(0, 1, shape) < kind


@pytest.mark.parametrize("n", [(2, 2, 2), (26, 2, 10), (27, 3, 11), (58, 10, 3), (59, 13, 18), (91, 27, 5)])
@pytest.mark.parametrize("kind", [0.03, 0.1, 0.2, 0.35, 0.6, 0.95, 1.0, "diagonal", "comb", "sheets"])
def test_labels(gpu, oracle, n, kind):
    g = Q.make_grid(oracle, n)
    shape = tuple(s + 6 for s in n)[::-1]
    img = _image(kind, shape, np.random.default_rng(sum(n))).astype(np.uint8)
    out = []
    for lib in (gpu, oracle):
        v = Q.Volume(g)
        v["phi_bin"][...] = img
        lib.findConnectivity3d(C.byref(v.p), C.byref(g))
        Q.check(lib)
        out.append(v["connectivity"].copy())
        if lib is gpu:
            lib.qssgpu_release(C.byref(v.p))
    assert np.array_equal(out[0], out[1])
