"""The loop-order sum around its chunks of 1024 elements: lengths next to one, two and the
2048 chunks from which their estimates are scanned, to where the walk takes more chunks
to a thread, and single zero chunks between others, against a sequential loop bit for bit."""
import ctypes as C

import numpy as np
import pytest

import qssgpu as Q

pytestmark = pytest.mark.gpu

CHUNK = 1024


def _values(kind, n):
    rng = np.random.default_rng(n + len(kind))
    if kind == "ties":  # 2^52 first: every later element is a multiple of half a unit
        x = rng.choice([0.5, 1.5, 1.0, 0.0], n)
        x[0] = 2.0 ** 52 + 1
    elif kind == "zero chunks":  # every second, third and fifth chunk, signed zeros
        j = np.arange(n) // CHUNK
        x = np.where((j % 2 == 1) | (j % 3 == 2) | (j % 5 == 4), rng.choice([0.0, -0.0], n), rng.random(n))
    elif kind == "climbing":  # binades crossed all along
        x = rng.random(n) * 2.0 ** (np.arange(n) / n * 60)
    else:
        x = rng.choice([0.04 ** 3, 0.0, 0.02 ** 3], n)
        x[CHUNK::3 * CHUNK] = -1e-7  # a chunk in three does not apply as a whole
    return np.ascontiguousarray(x)


@pytest.mark.parametrize("n", [CHUNK - 1, CHUNK, CHUNK + 1, 2 * CHUNK - 1, 2 * CHUNK, 2 * CHUNK + 1, 3 * CHUNK, 256 * CHUNK,
                               512 * CHUNK + 1, 2048 * CHUNK, 2048 * CHUNK + 1, 4100 * CHUNK + 3])
@pytest.mark.parametrize("kind", ["ties", "zero chunks", "climbing", "pack with negatives"])
def test_chunks(gpu, n, kind):
    x = _values(kind, n)
    out = C.c_double(-1.0)
    assert gpu.qssgpu_loop_sum(Q.dptr(x), n, C.byref(out)) == 0
    Q.check(gpu)
    want = 0.0
    for v in x.tolist():
        want += v
    assert out.value.hex() == want.hex()
