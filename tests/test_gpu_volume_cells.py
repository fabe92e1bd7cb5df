"""Volumes over cells of any size, those outside the range of 32-bit floats among them:
the oracle's bits, and as fast as with ordinary cells."""
import ctypes as C

import numpy as np
import pytest

import qssgpu as Q
from test_zz_no_alloc import _bind

pytestmark = pytest.mark.gpu


def _level_set(n, dx):
    z, y, x = np.meshgrid(*[np.arange(s + 6.0) for s in reversed(n)], indexing="ij")
    return dx * 4 * (np.sin(0.3 * x) + np.sin(0.31 * y) + np.sin(0.29 * z))


@pytest.mark.parametrize("n", [(9, 7, 5), (40, 33, 51)])
@pytest.mark.parametrize("dx", [1e-104, 2.0 ** -341, 2.0 ** -340, 1e-60, 1e-14, 2.0 ** -43, 2.0 ** -42, 1e-6, 1.0, 1e12,
                                2.0 ** 43, 1e30, 1e100])
def test_cell_sizes(gpu, oracle, n, dx):
    g = Q.make_grid(oracle, n)
    phi, vol = _level_set(n, dx), []
    for lib in (gpu, oracle):
        v = C.c_double(-1.0)
        lib.qss3dvolumeregionphilessthanzero_(C.byref(v), Q.dptr(phi), *Q.gb_args(g), *Q.fb_args(g),
                                              *(Q.dref(dx) for _ in range(3)), Q.dref(1.5 * dx))
        Q.check(lib)
        vol.append(v.value)
    assert vol[0].hex() == vol[1].hex()


@pytest.mark.parametrize("dx", [1e-14, 1e14])
def test_small_and_large_cells_are_no_slower(gpu, oracle, dx):
    """128^3 on the device: 0.2 ms, against 7 where every chunk goes by windows."""
    torch = pytest.importorskip("torch")
    volume = _bind(gpu)
    n = (128, 128, 128)
    box = [(C.c_int * 6)(lo, hi, lo, hi, lo, hi) for lo, hi in ((0, 133), (3, 130))]
    out, s = torch.zeros(1, dtype=torch.float64, device="cuda"), torch.cuda.Stream()
    ms = []
    for d in (0.04, dx):
        phi = torch.as_tensor(_level_set(n, d), device="cuda")
        torch.cuda.synchronize()
        best = 1e9
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(s)
            assert volume(phi.data_ptr(), *box, d, d, d, 1.5 * d, out.data_ptr(), C.c_void_p(s.cuda_stream)) == 0
            b.record(s)
            s.synchronize()
            best = min(best, a.elapsed_time(b))
        ms.append(best)
    Q.check(gpu)
    assert ms[1] < 4 * ms[0]
