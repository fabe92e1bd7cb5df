"""The loop-order sum at the edges of its rules, against a sequential loop bit for
bit: running sums in the lowest binades of the normal range, where the chunks'
precomputed sums do not apply and the sum goes by windows of elements."""
import ctypes as C

import numpy as np
import pytest

import qssgpu as Q

pytestmark = pytest.mark.gpu


def _sum(gpu, x):
    out = C.c_double(-1.0)
    assert gpu.qssgpu_loop_sum(Q.dptr(x), x.size, C.byref(out)) == 0
    Q.check(gpu)
    return out.value


def _loop(x):
    s = 0.0
    for v in x.tolist():
        if v != 0.0:
            s += v
    return s


# 2^-1030 starts below the normal range, 2^-1022 at its lower end, 2^-1001 leaves the range
# of the precomputed sums from below
@pytest.mark.parametrize("exponent", [-1074, -1050, -1030, -1023, -1022, -1021, -1012, -1001, -1000, -999])
@pytest.mark.parametrize("n", [5, 700, 3000, 9001])
def test_lowest_binades(gpu, n, exponent):
    x = np.random.default_rng(n).random(n) * 2.0 ** exponent if exponent > -1074 else np.full(n, 5e-324)
    x[::13] = 0.0
    assert _sum(gpu, x).hex() == _loop(x).hex()
