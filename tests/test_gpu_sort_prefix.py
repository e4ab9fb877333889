"""ORDER BY of more than 32 key bits by a prefix and the runs that share one (cql_sort_range, cql_sort_sample,
cql_sort_prefix, cql_sort_runs), against a stable sort of the keys as doubles on the host: the permutation equals it
for every mix of key types and directions, tied and nearly tied keys, keys that do not vary, columns whose values
crowd (the sample or the runs pass sends them to the passes over every digit), selections and narrow columns."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops(gpu):
    from computeql_gb300 import ops as o
    return o


def order(arrays, desc, rows=None):
    """the rows in order: keys as doubles, -0.0 as 0.0, ties by position"""
    keys = []
    for a, d in zip(arrays, desc):
        x = a.astype(np.float64) + 0.0
        x = x if rows is None else x[rows]
        keys.append(-x if d else x)
    by = np.lexsort(keys[::-1])
    return by if rows is None else rows[by]


def column(ops, a):
    kinds = {np.dtype(np.uint32): ops.TYPE_U32, np.dtype(np.int32): ops.TYPE_I32, np.dtype(np.float32): ops.TYPE_F32,
             np.dtype(np.float64): ops.TYPE_F64, np.dtype(np.uint64): ops.TYPE_U64, np.dtype(np.int64): ops.TYPE_I64}
    return ops.Column(kinds[a.dtype], len(a), ops.DeviceBuffer(a.nbytes, a), zone_map=False)


def draw(rng, kind, n):
    if kind == "lognormal":
        return np.exp(3.0 + rng.normal(size=n))
    if kind == "signed":
        return rng.normal(size=n) * 10.0 ** rng.integers(-30, 30, n)
    if kind == "prices":
        return rng.integers(-5000, 5000, n) / 100.0
    if kind == "i64":
        return rng.integers(-2**40, 2**40, n)
    if kind == "i64 large":
        return rng.integers(-2**63, 2**63 - 1, n)          # doubles meet: ties
    if kind == "u64":
        return rng.integers(0, 2**63, n).astype(np.uint64) * np.uint64(2)
    if kind == "clock":
        return 1_700_000_000_000_000 + np.sort(rng.integers(0, 86_400_000_000, n))[rng.permutation(n)]
    if kind == "crowded":
        return 1.0 + rng.random(n) * 1e-12 + (np.arange(n) == n // 2) * -1e18
    if kind == "one crowd":
        x = np.exp(rng.normal(size=n) * 20)
        at = rng.permutation(n)[: min(n // 2, 400)]
        x[at] = 5.0 + np.arange(len(at))[::-1] * 1e-15 * 5
        return x
    if kind == "constant":
        return np.full(n, -7.25)
    if kind == "few":
        return rng.integers(0, 50, n).astype(np.uint32)
    if kind == "u32":
        return rng.integers(0, 2**32, n).astype(np.uint32)
    if kind == "i32":
        return rng.integers(-2**31, 2**31 - 1, n).astype(np.int32)
    return rng.normal(size=n).astype(np.float32)


@pytest.mark.parametrize("n", [16384, 16385, 65_537, 300_007])
@pytest.mark.parametrize("kinds,desc", [
    (["lognormal"], [0]), (["lognormal"], [1]), (["signed"], [1]), (["prices"], [0]), (["i64"], [0]), (["i64 large"], [1]), (["u64"], [0]), (["clock"], [1]),
    (["crowded"], [0]), (["one crowd"], [0]), (["constant"], [0]), (["lognormal", "u32"], [1, 0]), (["few", "i64"], [0, 1]), (["u32", "i32"], [0, 1]),
    (["constant", "few"], [0, 1]), (["few", "constant", "f32"], [1, 0, 0]), (["few", "few", "prices", "i32"], [0, 1, 0, 1]), (["f32", "lognormal"], [1, 0])])
def test_order(ops, n, kinds, desc):
    rng = np.random.default_rng(n + len(kinds[0]) + sum(desc))
    arrays = [draw(rng, k, n) for k in kinds]
    arrays[0][0] = arrays[0][n - 1]
    cols = [column(ops, a) for a in arrays]
    np.testing.assert_array_equal(ops.sort_rows(cols, desc), order(arrays, desc))
    rows = np.sort(rng.choice(n, n * 3 // 4, replace=False)).astype(np.uint32)[rng.permutation(n * 3 // 4)]
    sel = ops.DeviceBuffer(rows.nbytes, rows)
    np.testing.assert_array_equal(ops.sort_rows(cols, desc, selection=sel), order(arrays, desc, rows))


def test_narrow_and_sequence_keys(ops):
    rng = np.random.default_rng(3)
    n = 50_001
    a, b = rng.integers(1000, 1200, n).astype(np.uint32), rng.normal(size=n)
    cols = [ops.Column.from_numpy(a, narrow=True), column(ops, b), ops.Column.sequence(n)]
    assert cols[0].width == 1
    np.testing.assert_array_equal(ops.sort_rows(cols, [1, 0, 1]), order([a, b, np.arange(n)], [1, 0, 1]))
    np.testing.assert_array_equal(ops.sort_rows([cols[0], cols[2]], [0, 1]), order([a, np.arange(n)], [0, 1]))
