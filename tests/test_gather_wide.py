"""Row gathers of more columns than one launch takes (CPU: the backend in host memory logs the launches)."""
import ctypes as C

import numpy as np
import pytest

from computeql_gb300 import native as N, ops
from tests import fake_backend


@pytest.mark.parametrize("columns,launches", [(1, 1), (65535, 1), (65536, 2), (131_071, 3)])
def test_columns_past_the_grid(tmp_path_factory, columns, launches):
    lib = fake_backend.load(str(tmp_path_factory.mktemp("fake")))
    one = fake_backend.column(lib, ops.TYPE_U32, np.arange(16, dtype=np.uint32))
    cols = (N.CqlColumn * columns)(*[one] * columns)
    out = np.zeros((columns, 4), np.uint32)
    ptrs = (C.c_void_p * columns)(*(out.ctypes.data + 16 * np.arange(columns)).tolist())
    rows = np.array([3, 1, 2, 0], np.uint32)
    assert lib.cqlops_gather_rows(cols, columns, rows.ctypes.data, None, 4, ptrs), lib.cqlops_last_error()
    assert fake_backend.log(lib, "run") == ["cql_gather_columns"] * launches
