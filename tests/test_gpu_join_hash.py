"""The join-aggregate through a hash table that carries each dim key's group (cql_join_hash_build, cql_join_hash_probe),
against the totals per dim row (strategy 2): every output equal, for fact keys over a wide range with and without a
range, dim tables resident and on the host, filtered dim rows, signed arguments, no GROUP BY and up to thousands of
groups; what the form does not take (repeated keys, fractional or far-apart group values) is answered or refused as
by strategy 2."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
COUNT, SUM, AVG, MIN, MAX = 0, 1, 2, 3, 4


@pytest.fixture(scope="module")
def ops(gpu):
    from computeql_gb300 import ops as o
    return o


def tables(rng, dims, rows, groups, signed):
    lo, hi = (-2**31, 2**31 - 1) if signed else (0, 2**32 - 1)
    dk = rng.choice(np.unique(rng.integers(lo, hi, 2 * dims + 8)), dims, replace=False).astype(np.int32 if signed else np.uint32)
    seg = rng.integers(0, groups, dims) if groups else np.zeros(dims, dtype=np.int64)
    # four fact rows in five join, some dim keys are never met
    fk = np.where(rng.random(rows) < 0.8, dk[rng.integers(0, max(1, dims * 3 // 4), rows)], rng.integers(lo, hi, rows).astype(dk.dtype))
    return dk, seg, fk.astype(dk.dtype)


@pytest.mark.parametrize("signed", [False, True])
@pytest.mark.parametrize("dims,rows,groups", [(1, 1, 1), (3, 33, 0), (1000, 4097, 20), (1000, 200_003, 1), (20_000, 100_003, 700), (40_000, 300_007, 5000)])
@pytest.mark.parametrize("resident", [False, True])
def test_equal_to_totals_per_dim_row(ops, signed, dims, rows, groups, resident):
    rng = np.random.default_rng(dims + rows + signed)
    dk, seg, fk = tables(rng, dims, rows, groups, signed)
    u = rng.integers(0, 2**32, rows).astype(np.uint32)
    i = rng.integers(-2**31, 2**31 - 1, rows).astype(np.int32)
    uc, ic = ops.Column.from_numpy(u), ops.Column.from_numpy(i)
    fc = ops.Column.from_numpy(fk, zone=rows > 1 and rows % 2 == 1)
    funcs, args = [COUNT, SUM, AVG, MIN, MAX, SUM], [None, uc, ic, ic, ic, ic]
    values = [(seg - 3).astype(np.float64)] if groups else []
    cols = {}
    if resident:
        cols["dim_key_col"] = ops.Column.from_numpy(dk)
        if groups:
            cols["dim_group_col"] = ops.Column.from_numpy((seg - 3).astype(np.int32))
    for dim_rows in (None, np.flatnonzero(rng.random(dims) < 0.7) if dims > 1 else np.array([0])):
        got = ops.join_aggregate(fc, funcs, args, dk.view(np.uint32), dim_rows=dim_rows, group_values=values, **cols)
        want = ops.join_aggregate(fc, funcs, args, dk.view(np.uint32), dim_rows=dim_rows, group_values=values, strategy=2)
        if dim_rows is None or len(dim_rows):
            assert got["strategy"] == want["strategy"]
        assert got["groups"] == want["groups"]
        np.testing.assert_array_equal(got["dim_row"], want["dim_row"])
        np.testing.assert_array_equal(got["results"], want["results"])


@pytest.mark.parametrize("case", ["fractional", "far apart", "minus zero", "repeated key"])
def test_what_the_form_does_not_take(ops, case):
    rng = np.random.default_rng(len(case))
    dk, seg, fk = tables(rng, 30_000, 50_001, 9, False)
    values = seg.astype(np.float64)
    if case == "fractional":
        values[::11] += 0.5
    elif case == "far apart":
        values[7] = 1.0e9
    elif case == "minus zero":
        values[values == 0] = -0.0
    else:
        dk[5] = dk[9]
    fc, uc = ops.Column.from_numpy(fk), ops.Column.from_numpy(rng.integers(0, 1000, len(fk)).astype(np.uint32))
    if case == "repeated key":
        with pytest.raises(ops.OpError):
            ops.join_aggregate(fc, [SUM], [uc], dk, group_values=[values])
        return
    got = ops.join_aggregate(fc, [SUM, COUNT], [uc, None], dk, group_values=[values])
    want = ops.join_aggregate(fc, [SUM, COUNT], [uc, None], dk, group_values=[values], strategy=2)
    np.testing.assert_array_equal(got["dim_row"], want["dim_row"])
    np.testing.assert_array_equal(got["results"], want["results"])
