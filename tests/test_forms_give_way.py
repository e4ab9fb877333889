"""An operator form that finds no room for its scratch gives way to the form behind it, which may need less; and the
scratch of a form that is done may be evicted to make room for the next (CPU: the backend in host memory, whose
kernels do nothing)."""
import ctypes as C

import numpy as np
import pytest

from computeql_gb300 import native as N, ops
from tests import fake_backend

ROWS = 100_003


@pytest.fixture()
def lib(tmp_path_factory):
    return fake_backend.load(str(tmp_path_factory.mktemp("fake")))


def join(lib):
    a = np.arange(ROWS, dtype=np.uint32)
    b, p = fake_backend.column(lib, ops.TYPE_U32, a), fake_backend.column(lib, ops.TYPE_U32, a)
    n, out = C.c_uint64(), np.zeros(8 * ROWS, np.uint32)
    return lib.cqlops_hash_join(C.byref(b), C.byref(p), 0, 0, C.byref(n), out.ctypes.data, 4 * ROWS)


@pytest.mark.parametrize("name", ["join_unique_table", "join_unique_match", "join_unique_pairs", "join_unique_counts", "join_unique_head"])
def test_join_of_unique_keys(lib, name):
    assert join(lib), lib.cqlops_last_error()
    assert "hash_join_build_count" not in fake_backend.log(lib, "run")
    assert {"join_unique_table", "join_unique_match", "join_unique_pairs"} <= set(fake_backend.log(lib, "idle"))
    lib.fake_reset()
    lib.fake_fail_name(name.encode())
    assert join(lib), lib.cqlops_last_error()
    assert fake_backend.log(lib, "refused") == [name]
    assert "hash_join_build_count" in fake_backend.log(lib, "run")


def join_aggregate(lib, dims, listed, fraction=0.0):
    rng = np.random.default_rng(1)
    keys = rng.choice(2 ** 32, dims, replace=False).astype(np.uint32)
    fact = fake_backend.column(lib, ops.TYPE_U32, keys[rng.integers(0, dims, ROWS)], (0.0, 2.0 ** 32 - 1))
    value = fake_backend.column(lib, ops.TYPE_U32, np.ones(ROWS, np.uint32), (0.0, 1.0))
    funcs, fargs = np.array([0, 1], np.uint32), (C.c_void_p * 2)(None, C.addressof(value))
    seg = (np.arange(dims) % 20).astype(np.float64) + fraction
    gv = (C.c_void_p * 1)(seg.ctypes.data)
    visit = np.arange(0, dims, 2, dtype=np.uint64) if listed else None
    q = N.CqlJoinAgg(C.addressof(fact), 2, funcs.ctypes.data, C.addressof(fargs), None, keys.ctypes.data, dims, visit.ctypes.data if listed else None,
                     len(visit) if listed else 0, 1, C.addressof(gv), 0, None, None)
    groups, used = C.c_uint64(), C.c_uint32()
    row, res = np.zeros(dims, np.uint64), np.zeros(2 * dims)
    return lib.cqlops_join_aggregate(C.byref(q), dims, C.byref(groups), row.ctypes.data, res.ctypes.data, C.byref(used))


# (past 16384 visits the group values' range comes from a kernel, which does nothing here: the form ends there)
@pytest.mark.parametrize("dims,listed,name", [(2003, False, n) for n in ("join_hash_table", "join_hash_visit_groups", "join_hash_visits", "join_hash_dim_keys",
                                                                         "join_hash_group_values", "join_hash_slots")]
                         + [(40_003, True, n) for n in ("join_hash_visits", "join_hash_dim_keys", "join_hash_group_values", "join_hash_range")])
def test_join_aggregate_by_hash(lib, dims, listed, name):
    assert join_aggregate(lib, dims, listed), lib.cqlops_last_error()
    assert ("cql_join_group_range" if dims > 16384 else "cql_join_hash_probe") in fake_backend.log(lib, "run")
    lib.fake_reset()
    lib.fake_fail_name(name.encode())
    assert join_aggregate(lib, dims, listed), lib.cqlops_last_error()
    assert fake_backend.log(lib, "refused") == [name]
    assert not {"cql_join_group_range", "cql_join_hash_probe"} & set(fake_backend.log(lib, "run"))


@pytest.mark.parametrize("dims,listed", [(2003, True), (40_003, False), (40_003, True)])
def test_group_values_that_are_fractions_are_not_sent(lib, dims, listed):
    """such a column is met by the host pass: the values that show it are looked at before any is uploaded"""
    assert join_aggregate(lib, dims, listed, 0.5), lib.cqlops_last_error()
    assert not {"cql_join_group_range", "cql_join_hash_probe"} & set(fake_backend.log(lib, "run"))


def test_scratch_of_many_dim_rows_can_go(lib):
    assert join_aggregate(lib, 70_001, False), lib.cqlops_last_error()
    assert {"join_hash_table", "join_hash_dim_keys", "join_hash_slots"} <= set(fake_backend.log(lib, "idle"))


def group(lib, keys, hint):
    cols = [fake_backend.column(lib, ops.TYPE_U32, k, None) for k in keys]
    kc = (N.CqlColumn * len(cols))(*cols)
    value = fake_backend.column(lib, ops.TYPE_F64, np.ones(ROWS), None)
    funcs, args, params = np.array([0, 1], np.uint32), (C.c_void_p * 2)(None, C.addressof(value)), np.zeros(2)
    g, path = C.c_uint64(), C.c_uint32()
    rr, cnt, res = np.zeros(ROWS, np.uint64), np.zeros(ROWS, np.uint64), np.zeros(2 * ROWS)
    return lib.cqlops_group_hash(kc, len(cols), 2, funcs.ctypes.data, args, params.ctypes.data, hint, 0, ROWS, C.byref(g), rr.ctypes.data,
                                 cnt.ctypes.data, res.ctypes.data, C.byref(path))


@pytest.mark.parametrize("name", ["group_exact_plan", "group_exact_table", "group_exact_out", "group_exact_bits", "group_exact_list"])
def test_group_by_exact_tables(lib, name):
    keys = [np.arange(ROWS, dtype=np.uint32)]
    assert group(lib, keys, ROWS), lib.cqlops_last_error()
    assert "cql_group_exact" in fake_backend.log(lib, "run")
    assert {"group_exact_table", "group_exact_out", "group_exact_bits", "group_exact_list"} <= set(fake_backend.log(lib, "idle"))
    lib.fake_reset()
    lib.fake_fail_name(name.encode())
    assert group(lib, keys, ROWS), lib.cqlops_last_error()
    assert name in fake_backend.log(lib, "refused")
    assert "cql_group_exact" not in fake_backend.log(lib, "run") and "aggregate_assign" in fake_backend.log(lib, "run")
