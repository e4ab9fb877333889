"""The plan of an exact GROUP BY as the operator layer makes it (CPU: the backend in host memory)."""
import ctypes as C

import numpy as np
import pytest

from computeql_gb300 import ops
from tests import fake_backend

ROWS = 400_003


@pytest.fixture()
def lib(tmp_path_factory):
    return fake_backend.load(str(tmp_path_factory.mktemp("fake")))


def plan(lib, keys, hint):
    """(direct, slots, local slots, log2 of the copies, the keys' ranges) of the plan that was uploaded last"""
    kc = (type(keys[0]) * len(keys))(*keys)
    funcs = np.array([0], dtype=np.uint32)
    args = (C.c_void_p * 1)(None)
    params = np.zeros(1)
    groups, path = C.c_uint64(), C.c_uint32()
    rr, cnt, res = np.zeros(ROWS, np.uint64), np.zeros(ROWS, np.uint64), np.zeros(ROWS)
    assert lib.cqlops_group_hash(kc, len(keys), 1, funcs.ctypes.data, args, params.ctypes.data, hint, 0, ROWS, C.byref(groups), rr.ctypes.data,
                                 cnt.ctypes.data, res.ctypes.data, C.byref(path)), lib.cqlops_last_error()
    p = C.string_at(lib.fake_pooled_data(b"group_exact_plan"), 416)
    ranges = np.frombuffer(p, np.uint64, len(keys), 64)
    direct, slots, local, copies = np.frombuffer(p, np.uint32, 4, 400).tolist()
    return direct, slots, local, copies, [int(r) or 1 << 64 for r in ranges]


def keys(lib, form):
    z = np.zeros(ROWS, np.uint64)
    one = {"f64": [(ops.TYPE_F64, (-1.0, 1.0))], "i64": [(ops.TYPE_I64, None)], "u64 far": [(ops.TYPE_U64, (0.0, 2.0 ** 63))],
           "f32,f32": [(ops.TYPE_F32, (0.0, 1.0))] * 2, "u32,u32": [(ops.TYPE_U32, None)] * 2, "f32": [(ops.TYPE_F32, (0.0, 1.0))],
           "u32 sparse": [(ops.TYPE_U32, (0.0, 4.0e9))], "i64,u32": [(ops.TYPE_I64, (0.0, 2.0 ** 40)), (ops.TYPE_U32, (0.0, 2.0 ** 20))]}
    return [fake_backend.column(lib, t, z, zone) for t, zone in one[form]]


@pytest.mark.parametrize("form", ["f64", "i64", "u64 far", "f32,f32", "u32,u32", "f32", "u32 sparse", "i64,u32"])
@pytest.mark.parametrize("hint", [0, 1, 2, 50, 256, 257, 5000])
def test_the_number_and_the_copy_fit_64_bits(lib, form, hint):
    direct, slots, local, copies, ranges = plan(lib, keys(lib, form), hint)
    product = 1
    for r in ranges:
        product *= r
    assert copies == 0 or product << copies <= 1 << 64
    # fewer bits leave room for copies, so that the lanes of a warp do not meet
    if form == "u32 sparse" and hint in (1, 2, 50, 256):
        assert local and copies > 0


@pytest.mark.parametrize("form", ["f64", "u32 sparse"])
@pytest.mark.parametrize("hint", [ROWS + 1, 1 << 40, (1 << 62) + 1, (1 << 63) + 1, (1 << 64) - 1])
def test_a_hint_past_the_rows(lib, form, hint):
    """a hint of more groups than rows is met as one of as many"""
    assert plan(lib, keys(lib, form), hint) == plan(lib, keys(lib, form), ROWS)
