"""GROUP BY in the exact tables (cql_group_exact) through the C ABI.

Every form the numbering of groups accepts (whole-number keys with and without a range, floats, 64-bit integers past
2^53, two to four keys; tables indexed and hashed, in shared and in device memory; hints right, wrong and absent) gives
the groups of the member lists (path 1): counts, MIN and MAX equal, and each f64 SUM the exactly rounded sum
(math.fsum), AVG that divided by the count. Data outside the form (NaN or -0.0 keys, keys outside their range, values
too small for the sums' window, more groups than hinted) gives the same answer by another path.
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
COUNT, SUM, AVG, MIN, MAX = 0, 1, 2, 3, 4


@pytest.fixture(scope="module")
def ops(gpu):
    from computeql_gb300 import ops as o
    return o


def column(ops, arr, zone=True):
    fin = arr[np.isfinite(arr)] if arr.dtype.kind == "f" else arr
    kinds = {np.dtype(np.uint32): ops.TYPE_U32, np.dtype(np.int32): ops.TYPE_I32, np.dtype(np.float32): ops.TYPE_F32,
             np.dtype(np.float64): ops.TYPE_F64, np.dtype(np.uint64): ops.TYPE_U64, np.dtype(np.int64): ops.TYPE_I64}
    z = zone if isinstance(zone, tuple) else (float(fin.min()), float(fin.max())) if zone and len(fin) else None
    return ops.Column(kinds[arr.dtype], len(arr), ops.DeviceBuffer(arr.nbytes, arr), zone=z)


def groups_of(res, keys):
    """{key values of the representative row: (count, results)}; -0.0 as 0.0"""
    out = {}
    for g in range(res["groups"]):
        k = tuple(float(a[int(res["repr_row"][g])]) + 0.0 for a in keys)
        assert k not in out
        out[k] = (int(res["counts"][g]), res["results"][g])
    return out


def members_of(keys):
    f = np.stack([a.astype(np.float64) + 0.0 for a in keys], 1)
    uniq, inverse = np.unique(f, axis=0, return_inverse=True)
    order = np.argsort(inverse.ravel(), kind="stable")
    bounds = np.searchsorted(inverse.ravel()[order], np.arange(len(uniq) + 1))
    return {tuple(u.tolist()): order[bounds[i]:bounds[i + 1]] for i, u in enumerate(uniq)}


def check(res, keys, funcs, args):
    got, want = groups_of(res, keys), members_of(keys)
    assert set(got) == set(want)
    for k, rows in want.items():
        n, r = got[k]
        assert n == len(rows)
        for e, (f, a) in enumerate(zip(funcs, args)):
            if f == COUNT:
                assert r[e] == len(rows)
                continue
            x = a[rows].astype(np.float64)
            if f in (SUM, AVG):
                s = math.fsum(x)
                assert r[e] == (s if f == SUM else s / len(rows)), (k, f, r[e], s)
            else:
                assert r[e] == (x.min() if f == MIN else x.max())


def keys_for(form, rng, n, groups):
    g = rng.integers(0, groups, n)
    if form == "u32":
        return [(g + 7).astype(np.uint32)]
    if form == "i32":
        return [(g - groups // 2).astype(np.int32)]
    if form == "i64 sparse":
        return [g.astype(np.int64) * 1_000_000_007 - (1 << 40)]
    if form == "u64 large":
        return [(g.astype(np.uint64) << np.uint64(40)) + np.uint64(1 << 62)]
    if form == "f64":
        return [g * 0.37 - 5.0]
    if form == "f32":
        return [(g * 0.5 - 5.0).astype(np.float32)]
    if form == "u32,i64":
        return [(g % 13).astype(np.uint32), (g // 13).astype(np.int64) * 1_000_003 - (1 << 33)]
    if form == "f32,i32":
        return [(g % 5 * 0.25).astype(np.float32), (g // 5 - 100).astype(np.int32)]
    return [(g % 3).astype(np.uint32), (g // 3 % 7).astype(np.int32), (g // 21 % 4).astype(np.uint64), (g // 84).astype(np.int64) * 77]


FORMS = ["u32", "i32", "i64 sparse", "u64 large", "f64", "f32", "u32,i64", "f32,i32", "four"]


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("groups,n,hint", [(1, 1, 1), (3, 257, 0), (90, 100_003, 90), (2000, 60_001, 2000), (2000, 60_001, 40), (30_000, 120_001, 0),
                                           (5000, 300_007, 5000)])
def test_forms_of_keys_and_tables(ops, form, groups, n, hint):
    rng = np.random.default_rng(groups + n)
    keys = keys_for(form, rng, n, groups)
    logn, mixed = np.exp(3.0 + rng.normal(size=n)), rng.normal(size=n) * 10.0 ** rng.integers(-2, 5, n)
    i32, i64 = rng.integers(-2**31, 2**31 - 1, n).astype(np.int32), rng.integers(-2**50, 2**50, n)
    funcs, args = [COUNT, SUM, AVG, MIN, MAX, SUM, AVG, MAX], [None, logn, mixed, mixed, logn, i32, i64, i32]
    cols = {id(a): column(ops, a) for a in args if a is not None}
    dev = [cols[id(a)] if a is not None else None for a in args]
    kc = [column(ops, k) for k in keys]
    res = ops.group_hash(kc, funcs, dev, group_hint=hint)
    check(res, keys, funcs, args)
    lists = ops.group_hash(kc, funcs, dev, group_hint=hint, path=1)
    a, b = groups_of(res, keys), groups_of(lists, keys)
    assert set(a) == set(b)
    for k in a:
        assert a[k][0] == b[k][0] and np.array_equal(a[k][1][[0, 3, 4, 7]], b[k][1][[0, 3, 4, 7]])


@pytest.mark.parametrize("form", ["u32", "u32,i64"])
@pytest.mark.parametrize("groups", [4, 700, 40_000])
def test_whole_numbers_and_decimals(ops, form, groups):
    rng = np.random.default_rng(groups)
    n = 200_003
    keys = keys_for(form, rng, n, groups)
    price = rng.integers(-10**7, 10**7, n) / 100.0
    u = rng.integers(0, 2**31, n).astype(np.uint32)
    funcs, args = [SUM, AVG, MIN, MAX, SUM, MIN], [price, price, price, price, u, u]
    cols = {id(a): column(ops, a) for a in (price, u)}
    res = ops.group_hash([column(ops, k) for k in keys], funcs, [cols[id(a)] for a in args], group_hint=groups)
    assert res["path"] == 2
    cents = np.round(price * 100).astype(np.int64)
    got, want = groups_of(res, keys), members_of(keys)
    assert set(got) == set(want)
    for k, rows in want.items():
        c, x = cents[rows], u[rows].astype(np.int64)
        s = float(c.sum()) / 100.0
        assert got[k][1].tolist() == [s, s / len(rows), c.min() / 100.0, c.max() / 100.0, float(x.sum()), float(x.min())]


@pytest.mark.parametrize("case", ["nan key", "minus zero key", "key outside its range", "tiny values", "infinite values", "no ranges", "huge values"])
def test_data_outside_the_form(ops, case):
    rng = np.random.default_rng(len(case))
    n = 50_001
    key = rng.integers(0, 300, n)
    x = rng.normal(size=n)
    zone = True
    k = key * 0.5 if case.endswith("zero key") or case.startswith("nan") else key.astype(np.uint32)
    if case == "minus zero key":
        k[k == 0] = -0.0
    elif case == "nan key":
        k[5] = np.nan
    elif case == "key outside its range":
        zone = (0.0, 199.0)
    elif case == "tiny values":
        x[::7] *= 1e-30
    elif case == "infinite values":
        x[11], x[12] = np.inf, -np.inf
    elif case == "no ranges":
        zone = None
    elif case == "huge values":
        x *= 1e300
    xc = column(ops, x, case != "no ranges")
    kc = column(ops, k, zone)
    res = ops.group_hash([kc], [SUM, COUNT, MIN], [xc, None, xc], max_groups=n)   # (the default result area goes by the key's range)
    if case == "nan key":
        # a NaN key equals no other: its row is a group of its own
        assert res["groups"] == len(np.unique(k[~np.isnan(k)])) + 1
        return
    got, want = groups_of(res, [k]), members_of([k])
    assert set(got) == set(want)
    for key_values, rows in want.items():
        v = x[rows]
        n_rows, r = got[key_values]
        assert n_rows == len(rows) == r[1]
        if np.isinf(v).any():
            assert r[0] == v[np.isinf(v)][0]
        else:
            s = math.fsum(v)
            assert abs(r[0] - s) <= 1e-12 * np.abs(v).sum()
        assert r[2] == max(min(v.min(), 1.0e300), -np.inf)
