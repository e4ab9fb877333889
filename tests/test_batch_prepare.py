"""A prepared catalog compiles every kernel its batches may take, however few queries it was prepared with (CPU: the
backend in host memory logs what is compiled)."""
import ctypes as C

import numpy as np
import pytest

from computeql_gb300 import ops
from tests import fake_backend

ROWS = 5000
RANKED = [("(< u 5)", "v"), ("(and (> d 0.25) (< u 9))", "d"), ("(or (= u 3) (<= v 0.5))", "v")]


@pytest.fixture()
def lib(tmp_path_factory):
    from computeql_gb300 import build
    build.build()
    return fake_backend.load(str(tmp_path_factory.mktemp("fake")))


def programs(lib, queries):
    cols = {"u": ops.Column(ops.TYPE_U32, ROWS, zone=(0.0, 65535.0)), "d": ops.Column(ops.TYPE_F64, ROWS, zone=(0.0, 1.0)),
            "v": ops.Column(ops.TYPE_F64, ROWS, zone=(0.0, 1.0))}
    progs = [ops.Program(w, cols) for w, _ in queries]
    base = progs[0]
    for i, size in enumerate((4, 8, 8)):
        base._cols[i].buffer = lib.cqlcuda_buffer_alloc(ROWS * size, 0, None)
    return progs, base._cols, np.array([base.index(s) for _, s in queries], dtype=np.int32)


def call(lib, f, catalog, progs, cols, sums, *out):
    ptrs = (C.c_void_p * len(progs))(*[C.addressof(p.prog) for p in progs])
    sums = np.ascontiguousarray(sums)
    assert f(catalog, ptrs, len(progs), cols, 3, sums.ctypes.data, 8, *out), lib.cqlops_last_error()


@pytest.mark.parametrize("queries", [RANKED[:1], RANKED], ids=["one template", "three templates"])
@pytest.mark.parametrize("together", [1, 2, 3])
def test_batches_of_prepared_shapes_compile_nothing(lib, queries, together):
    catalog = lib.cqlops_batch_catalog_create()
    progs, cols, sums = programs(lib, queries)
    for first in range(0, len(progs), together):
        call(lib, lib.cqlops_batch_prepare, catalog, progs[first:first + together], cols, sums[first:first + together])
    assert lib.cqlops_batch_catalog_shapes(catalog) == len(queries)
    lib.fake_clear_log()
    counts, totals, shapes = np.zeros(64, np.uint64), np.zeros(64), C.c_uint32()
    for n in (1, 2, 5, 40):
        pick = np.arange(n) % len(progs)
        call(lib, lib.cqlops_batch_filter_aggregate_cat, catalog, [progs[k] for k in pick], cols, sums[pick], counts.ctypes.data, totals.ctypes.data,
             C.byref(shapes))
        ran = [k for k in fake_backend.log(lib, "run") if k.startswith("qk_")]
        assert ran[-1].startswith("qk_batch_rank") == (n > 1)
    assert fake_backend.log(lib, "compile") == []
    lib.cqlops_batch_catalog_destroy(catalog)
