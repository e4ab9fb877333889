"""GROUP BY kernels chosen per column type and kept result: every argument type with every choice of SUM, MIN and MAX,
over a small-range key (cql_group_small, one table a thread and shared ones) and over two keys of every type
(cql_group_exact), with the special values at the ends of the types and rows at the remainders of a thread's four."""
import math

import numpy as np
import pytest

from tests.test_gpu_group_exact import MAX, MIN, SUM, check, column, groups_of, members_of

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops(gpu):
    from computeql_gb300 import ops as o
    return o


def values(kind, n, r):
    if kind == "u32":
        x = r.integers(0, 1 << 32, n, dtype=np.uint32)
        x[: 2] = np.array([0, 2**32 - 1], dtype=np.uint32)[:n]
    elif kind == "i32":
        x = r.integers(-(1 << 31), 1 << 31, n).astype(np.int32)
        x[: 2] = np.array([-2**31, 2**31 - 1], dtype=np.int32)[:n]
    elif kind == "i64":
        x = r.integers(-(1 << 50), 1 << 50, n)
    else:
        x = (r.normal(size=n) * np.exp(r.normal(size=n))).astype(np.float64 if kind == "f64" else np.float32)
        x[n // 2: n // 2 + 2] = [0.0, -0.0][: len(x[n // 2: n // 2 + 2])]
    return x


KEPT = [(SUM,), (MIN,), (MAX,), (SUM, MIN, MAX)]


@pytest.mark.parametrize("kind", ["u32", "i32", "f32", "f64"])
@pytest.mark.parametrize("rows,groups", [(1, 1), (5, 3), (20_003, 3), (70_001, 64)])
def test_small_range_key(ops, kind, rows, groups):
    """sums within rows x 2^-61 of the largest value (the fixed-point step), extremes equal"""
    r = np.random.default_rng(rows + groups)
    key, x = r.integers(10, 10 + groups, rows, dtype=np.uint32), values(kind, rows, r)
    for kept in KEPT:
        res = ops.group_hash([column(ops, key)], list(kept), [column(ops, x)] * len(kept), group_hint=groups)
        got, want = groups_of(res, [key]), members_of([key])
        assert set(got) == set(want)
        big = float(np.abs(x.astype(np.float64)).max())
        for k, at in want.items():
            v = x[at].astype(np.float64)
            assert got[k][0] == len(at)
            for f, y in zip(kept, got[k][1]):
                if f == SUM:
                    exact = math.fsum(v)
                    assert abs(y - exact) <= rows * big * 2.0**-61 + abs(exact) * 2.0**-53
                else:
                    assert y == (v.min() if f == MIN else v.max())


@pytest.mark.parametrize("kind", ["u32", "i32", "f32", "f64", "i64"])
@pytest.mark.parametrize("other", ["u32", "i32", "f32", "f64", "i64"])
def test_two_keys(ops, kind, other):
    r = np.random.default_rng(17)
    rows = 30_001
    first = r.integers(5, 12, rows, dtype=np.uint32)
    second = (r.integers(0, 9, rows) * 3 - 7).astype({"u32": np.int64, "i32": np.int32, "f32": np.float32, "f64": np.float64, "i64": np.int64}[other])
    if other == "u32":
        second = (second + 1000).astype(np.uint32)
    keys = [second] if other == "f64" else [first, second]     # a key of doubles takes the whole number by itself
    x = values(kind, rows, r)
    for kept in KEPT:
        res = ops.group_hash([column(ops, k) for k in keys], list(kept), [column(ops, x)] * len(kept), group_hint=63)
        check(res, keys, list(kept), [x] * len(kept))
