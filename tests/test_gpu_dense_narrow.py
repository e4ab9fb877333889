"""Dense GROUP BY over narrow columns: every stored width of the key (1- and 2-byte codes, whole words) and of the
arguments (the same, and sequences), one to eight aggregates over up to four columns, group counts of one and of several
shared-memory tiles, and rows at the remainders of a vector. Whole numbers: equal to numpy's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
COUNT, SUM, AVG, MIN, MAX = 0, 1, 2, 3, 4


@pytest.fixture(scope="module")
def ops(gpu):
    from computeql_gb300 import ops as o
    return o


def _argument(ops, kind, n, r):
    """(column, its values)"""
    if kind == "sequence":
        return ops.Column.sequence(n, first=7), np.arange(7, 7 + n, dtype=np.int64)
    lo, hi, t, narrow = {"u8": (1000, 1200, np.uint32, True), "i8": (-100, 100, np.int32, True), "u16": (5, 60_000, np.uint32, True),
                         "u32": (0, 1 << 31, np.uint32, False), "i32": (-(1 << 31), 1 << 31, np.int32, False)}[kind]
    x = r.integers(lo, hi, n).astype(t)
    return ops.Column.from_numpy(x, narrow=narrow), x.astype(np.int64)


@pytest.mark.parametrize("rows", [1, 3, 4, 5, 4097, 300_003])
@pytest.mark.parametrize("groups,narrow", [(7, True), (250, True), (3000, True), (20_000, True), (7, False)])
def test_widths(ops, rows, groups, narrow):
    r = np.random.default_rng(rows * 31 + groups)
    key = (r.integers(0, groups, rows) + 40).astype(np.uint32)
    kcol = ops.Column.from_numpy(key, narrow=narrow)
    for kinds, funcs in [(["u8"], [SUM]), (["u32"], [SUM, COUNT]), (["i8"], [MIN, MAX, SUM]), (["u16", "i32"], [SUM, AVG, MIN, MAX]),
                         (["sequence"], [SUM, MAX]), (["u8", "u16", "i8"], [SUM, MAX, MIN, COUNT, SUM]),
                         (["i32", "sequence", "u8", "u16"], [SUM, SUM, MAX, MIN, COUNT, MAX, AVG, MIN])]:
        if (not narrow and all(k in ("u32", "i32") for k in kinds)) or (groups == 20_000 and len(funcs) > 3):
            continue     # whole words throughout; more slices of the table than the operator takes
        cols = [_argument(ops, k, rows, r) for k in kinds]
        pick = [cols[e % len(cols)] for e in range(len(funcs))]
        first, counts, sums, mins, maxs = ops.group_dense(kcol, funcs, [None if f == COUNT else c for f, (c, _) in zip(funcs, pick)])
        at = key.astype(np.int64) - first
        n = np.bincount(at, minlength=len(counts))
        assert np.array_equal(counts.astype(np.int64), n)
        order = np.argsort(at, kind="stable")
        starts = np.searchsorted(at[order], np.flatnonzero(n))
        for e, (f, (_, x)) in enumerate(zip(funcs, pick)):
            if f == COUNT:
                continue
            reduce = {SUM: np.add, AVG: np.add, MIN: np.minimum, MAX: np.maximum}[f].reduceat(x[order], starts)
            got = {SUM: sums, AVG: sums, MIN: mins, MAX: maxs}[f][n > 0, e]
            assert np.array_equal(got, reduce), (kinds, funcs, e)
