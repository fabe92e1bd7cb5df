"""The volume of a box of more than 2^32 voxels (34 GB of level set): every voxel on the
interface of a lattice with spacing 1/16, so the sum of the halves of 2^-12 is exact."""
import ctypes as C

import numpy as np
import pytest

import qssgpu as Q

pytestmark = pytest.mark.gpu


def _host_available():
    with open("/proc/meminfo") as f:
        return next(int(line.split()[1]) for line in f if line.startswith("MemAvailable")) * 1024


def test_volume_beyond_2_to_32_voxels(gpu):
    torch = pytest.importorskip("torch")
    if torch.cuda.mem_get_info()[0] < 90e9 or _host_available() < 64e9:
        pytest.skip("needs 70 GB of device memory and 34 GB of host memory")
    n = (1626, 1626, 1626)
    phi = np.zeros(n)  # untouched pages
    box = [C.byref(C.c_int(v)) for s in n for v in (0, s - 1)]
    vol, dx = C.c_double(-1.0), 0.0625
    gpu.qss3dvolumeregionphilessthanzero_(C.byref(vol), Q.dptr(phi), *box, *box, Q.dref(dx), Q.dref(dx), Q.dref(dx),
                                          Q.dref(1.5 * dx))
    Q.check(gpu)
    assert vol.value == phi.size * 2.0 ** -13
