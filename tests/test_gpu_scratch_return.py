"""The memory that calls leave in the library's pool: qssgpu_release gives all of it back,
and on a GPU with nothing else free the library's other allocations get it."""
import ctypes as C

import numpy as np
import pytest

import qssgpu as Q

pytestmark = pytest.mark.gpu

MB = 1 << 20


@pytest.fixture
def pooled(gpu, oracle):
    """Returns a function that leaves 2 GB idle in the pool, and one that releases it."""
    torch = pytest.importorskip("torch")
    g = Q.make_grid(oracle, (260, 260, 260))
    a = np.zeros((266,) * 3)
    h = C.c_double(0)

    def call():
        gpu.getrhs3d5th_(Q.dptr(a), *(Q.dptr(a) for _ in range(5)), C.byref(h), Q.dptr(a), *Q.gb_args(g), *Q.fb_args(g),
                         *(Q.dref(g.dx[d]) for d in range(3)))
        Q.check(gpu)

    v = Q.Volume(Q.make_grid(oracle, (4, 4, 4)))

    def release():
        gpu.qssgpu_release(C.byref(v.p))

    call()
    release()
    yield torch, call, release
    release()


def _free(torch):
    return torch.cuda.mem_get_info()[0]


def test_release_gives_the_memory_back(pooled):
    torch, call, release = pooled
    before = _free(torch)
    for _ in range(3):
        call()
        assert _free(torch) < before - 1000 * MB
        release()
        assert _free(torch) >= before - 8 * MB


@pytest.mark.parametrize("what", ["sum", "sum above the pool's block size", "sphere", "box", "rates"])
def test_allocations_on_a_full_gpu(gpu, oracle, pooled, what):
    torch, call, _ = pooled
    call()
    fill = torch.empty(_free(torch) - 300 * MB, dtype=torch.uint8, device="cuda")
    try:
        if what.startswith("sum"):
            x = np.full((64 if what == "sum" else 160) * MB, 0.5)  # 512 MB, 1.25 GB
            out = C.c_double(0)
            assert gpu.qssgpu_loop_sum(Q.dptr(x), x.size, C.byref(out)) == 0
            assert out.value == 0.5 * x.size
        elif what == "rates":
            small = torch.empty(max(0, _free(torch) - 2 * MB), dtype=torch.uint8, device="cuda")
            assert gpu.qssgpu_op_rates((C.c_double * 8)()) == 0
            del small
        else:
            g = Q.make_grid(oracle, (394, 394, 394))
            phi = np.empty((400,) * 3)
            if what == "sphere":
                gpu.createSphere(Q.dptr(phi), C.c_double(1.0), C.c_double(1.0), C.c_double(1.0), C.c_double(0.5), -1,
                                 C.byref(g))
            else:
                gpu.createBox(Q.dptr(phi), *(C.c_double(0.2) for _ in range(6)), -1, C.byref(g))
        Q.check(gpu)
    finally:
        del fill
        torch.cuda.empty_cache()
        gpu.qssgpu_clear_error()
