"""A filter's program reaches the device whole, however late the batch takes its bytes (CPU: the backend in host memory
copies a batch's writes when the batch ends)."""
import ctypes as C

import numpy as np
import pytest

from computeql_gb300 import ops
from tests import fake_backend

ROWS = 5000


@pytest.fixture()
def lib(tmp_path_factory):
    from computeql_gb300 import build
    build.build()
    return fake_backend.load(str(tmp_path_factory.mktemp("fake")))


def setup(lib, where):
    prog = ops.Program(where, {"s": ops.Column(ops.TYPE_STRING8, ROWS), "u": ops.Column(ops.TYPE_U32, ROWS, zone=(0.0, 9.0))})
    cols = prog._cols
    cols[0].buffer = lib.cqlcuda_buffer_alloc(ROWS * 8, 0, None)
    cols[0].offsets = lib.cqlcuda_buffer_alloc((ROWS + 1) * 8, 0, None)
    cols[1].buffer = lib.cqlcuda_buffer_alloc(ROWS * 4, 0, None)
    return prog, cols


def pool(prog):
    return bytes(prog.prog.str_pool[:prog.prog.str_pool_size])


def uploaded(lib, name, n):
    return C.string_at(lib.fake_pooled_data(name), n)


WHERE = ["(and (= s 'warehouse') (> u 2))", "(or (= s 'a') (= s 'bcdefghijklmnop'))", f"(or (= s '{'x' * 61}') (< u 7))"]


@pytest.mark.parametrize("where", WHERE)
@pytest.mark.parametrize("strategy", [ops.SCAN_GENERATED, ops.SCAN_INTERPRETER])
@pytest.mark.parametrize("rows", [False, True])
def test_scan(lib, where, strategy, rows):
    prog, cols = setup(lib, where)
    count, ran, out = C.c_uint64(), C.c_uint32(), np.zeros(ROWS, np.uint32)
    assert lib.cqlops_scan_filter(C.byref(prog.prog), cols, strategy, C.byref(count), out.ctypes.data if rows else None, ROWS if rows else 0,
                                  C.byref(ran)), lib.cqlops_last_error()
    assert ran.value == strategy and len(pool(prog)) > 0
    assert uploaded(lib, b"cqlops_scan_str_consts", len(pool(prog))) == pool(prog)


@pytest.mark.parametrize("where", WHERE)
def test_fused(lib, where):
    prog, cols = setup(lib, where)
    agg, one = np.array([1], np.uint32), np.zeros(4)
    assert lib.cqlops_fused_filter_aggregate(C.byref(prog.prog), cols, agg.ctypes.data, 1, one.ctypes.data, one[1:].ctypes.data, one[2:].ctypes.data,
                                             one[3:].ctypes.data), lib.cqlops_last_error()
    assert uploaded(lib, b"cqlops_scan_str_consts", len(pool(prog))) == pool(prog)
