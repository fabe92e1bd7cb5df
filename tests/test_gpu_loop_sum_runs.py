"""The loop-order sum where its runs of contributions decide: ties met with an
even and an odd running sum, zero chunks before, between and after others, and
lengths around a chunk and around the form without chunks, against a sequential
loop bit for bit."""
import ctypes as C

import numpy as np
import pytest

import qssgpu as Q

pytestmark = pytest.mark.gpu

CHUNK = 4096


@pytest.mark.parametrize("n", [1, CHUNK - 1, CHUNK, 4 * CHUNK, 4 * CHUNK + 1, 2048, 2049, 5120, 21 * CHUNK + 17, 300 * CHUNK + 5, 2100 * CHUNK + 1])
@pytest.mark.parametrize("kind", ["half units", "odd multiples", "gaps", "all zero but one", "growing"])
def test_runs(gpu, n, kind):
    rng = np.random.default_rng(n + len(kind))
    if kind == "half units":  # 2^52 first: every later element is a multiple of half a unit
        x = rng.choice([0.5, 1.5, 1.0, 0.0], n)
        x[0] = 2.0 ** 52 + 1
    elif kind == "odd multiples":  # ties at every scale on the way up
        x = 2.0 ** -30 * rng.choice([1.0, 3.0, 5.0, 0.5, 1.5, 2.0 ** -20, 3 * 2.0 ** -21], n)
    elif kind == "gaps":  # whole chunks of zeros, signed
        x = rng.random(n) * (rng.random((n + CHUNK - 1) // CHUNK) < 0.4).repeat(CHUNK)[:n]
        x[x == 0] = rng.choice([0.0, -0.0], int((x == 0).sum()))
    elif kind == "all zero but one":
        x = np.zeros(n)
        x[n - 1] = 0.1
    else:  # each element about half a unit of the sum so far
        x = np.full(n, 2.0 ** -53)
        x[::97] = 1.0
    out = C.c_double(-1.0)
    assert gpu.qssgpu_loop_sum(Q.dptr(np.ascontiguousarray(x)), n, C.byref(out)) == 0
    Q.check(gpu)
    want = 0.0
    for v in x.tolist():
        if v != 0.0:
            want += v
    assert out.value.hex() == want.hex()
