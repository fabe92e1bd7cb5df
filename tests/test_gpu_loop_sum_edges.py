"""The loop-order sum at the edges of its rules, against a sequential loop bit for
bit: running sums in the lowest binades of the normal range, where the chunks'
precomputed sums do not apply and the sum goes by windows of elements; and elements and
sums that no window takes, which go one by one."""
import ctypes as C
import time

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


def _stops(kind, n):
    rng = np.random.default_rng(n)
    x = rng.random(n)
    if kind == "negative":
        return -x
    if kind == "signs":
        return x - 0.5
    if kind.startswith("every "):  # a negative element every k-th
        x[:: int(kind[6:])] *= -1
        return x
    if kind == "bursts":  # negative runs of many lengths between positive ones
        return x * np.repeat(rng.choice([-1.0, 1.0, 1.0], n // 50 + 1), 50)[:n]
    if kind == "infinite":
        x[n // 3] = np.inf
    elif kind == "down through zero":  # the sum falls, is zero, and starts again
        x = np.concatenate([np.full(n // 2, 0.25), np.full(n // 2, -0.25), rng.random(n % 2 + 700)])
    return x


@pytest.mark.parametrize("kind", ["negative", "signs", "every 2", "every 9", "every 31", "every 33", "every 130", "bursts",
                                  "infinite", "down through zero"])
@pytest.mark.parametrize("n", [3, 1000, 1025, 7000, 40001])
def test_elements_one_by_one(gpu, n, kind):
    x = np.ascontiguousarray(_stops(kind, n))
    assert _sum(gpu, x).hex() == _loop(x).hex()


@pytest.mark.parametrize("kind", ["negative", "every 2", "infinite"])
def test_one_by_one_is_not_by_windows(gpu, kind):
    """0.4 M elements that no window takes: 17 ms one by one, 112 to 170 with a window for every
    few of them."""
    x = np.ascontiguousarray(_stops(kind, 400_000))
    _sum(gpu, x)
    best = min(_timed(gpu, x) for _ in range(3))
    assert best < 0.075


def _timed(gpu, x):
    t = time.perf_counter()
    _sum(gpu, x)
    return time.perf_counter() - t
