"""Row gathers of more columns than one launch takes, against the columns' values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("columns", [65535, 65537])
def test_columns_past_the_grid(gpu, columns):
    from computeql_gb300 import ops
    n = 50
    a, b = np.arange(n, dtype=np.uint32) * 3, np.arange(n) * 0.5
    ca, cb = ops.Column.from_numpy(a), ops.Column.from_numpy(b)
    rows = np.array([49, 0, 7, 7, 21], dtype=np.uint32)
    got = ops.gather_rows([cb if j % 7 == 3 else ca for j in range(columns)], rows=rows)
    assert len(got) == columns
    for j in (0, 3, 10, 65533, 65534, columns - 1):
        assert np.array_equal(got[j], (b if j % 7 == 3 else a)[rows])
    assert all(np.array_equal(g, (b if j % 7 == 3 else a)[rows]) for j, g in enumerate(got))
