"""The solve's diagnostic traces: records within the buffer, in order of time, with
the schedule's marks; none when switched off; and the same psi with and without."""
import ctypes as C

import numpy as np
import pytest

import ggb_api as G
import ggb_cases as K

pytestmark = pytest.mark.gpu


@pytest.fixture
def lib(gpu):
    L = gpu.lib
    L.ggb_solve_trace_enable.restype = None
    L.ggb_solve_trace_enable.argtypes = [C.c_int]
    L.ggb_solve_trace.restype = C.c_int
    L.ggb_solve_trace.argtypes = [C.POINTER(C.c_ulonglong), C.c_int]
    L.ggb_stage_trace.restype = C.c_int
    L.ggb_stage_trace.argtypes = [C.c_int, C.POINTER(C.c_ulonglong), C.c_int]
    yield L
    L.ggb_solve_trace_enable(0)
    L.ggb_stage_trace(0, None, 0)


def records(buf, n):
    a = np.frombuffer(buf, np.uint64)[: 2 * n].reshape(-1, 2)
    return a[:, 0], a[:, 1]


@pytest.mark.parametrize("cap", [1, 50, 4000])
def test_solve_trace(gpu, lib, cap):
    plain = K.poisson(gpu, 32)
    buf = (C.c_ulonglong * 8000)()
    lib.ggb_solve_trace_enable(cap)
    traced = K.poisson(gpu, 32)
    n = lib.ggb_solve_trace(buf, 4000)
    assert np.array_equal(plain["psi"], traced["psi"]) and plain["iters"] == traced["iters"]
    marks, times = records(buf, n)
    assert n == cap if cap < 100 else int(traced["iters"]) < n < cap
    assert np.all(np.diff(times.astype(np.int64)) >= 0)
    assert set(marks.tolist()) <= {10, 11, 100, 101, 300, 301, 500, 900, 901}
    assert lib.ggb_solve_trace(buf, 0) == 0
    lib.ggb_solve_trace_enable(0)
    K.poisson(gpu, 32)
    assert lib.ggb_solve_trace(buf, 4000) == 0


@pytest.mark.parametrize("every_block", [0, 1])
def test_stage_trace(gpu, lib, every_block):
    buf = (C.c_ulonglong * 8192)()
    assert lib.ggb_stage_trace(1 + every_block, None, 0) == 0
    K.poisson(gpu, 32)
    n = lib.ggb_stage_trace(0, buf, 4096)
    marks, times = records(buf, n)
    assert 0 < n <= 4096 and set((marks & np.uint64(0xFFFF)).tolist()) == {1, 2}
    blocks = set((marks >> np.uint64(16)).tolist())
    assert len(blocks) > 100 if every_block else blocks == {0}
    if not every_block:  # start and end in turn
        assert np.array_equal(marks, np.tile([1, 2], n // 2)) and np.all(np.diff(times.astype(np.int64)) >= 0)
