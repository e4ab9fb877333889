"""The equi-join of a build side whose keys do not repeat (cql_join_unique_build, _probe, _emit) against a host join, and
what it gives way to the buckets for: repeated build keys, NaN and -0.0 keys, integers past 2^53. Pairs ascending by
probe row; LEFT JOIN gives unmatched rows; a short output array takes the first pairs."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
NONE = 0xFFFFFFFF


@pytest.fixture(scope="module")
def ops(gpu):
    from computeql_gb300 import ops as o
    return o


def column(ops, a):
    kinds = {np.dtype(np.uint32): ops.TYPE_U32, np.dtype(np.int32): ops.TYPE_I32, np.dtype(np.float32): ops.TYPE_F32,
             np.dtype(np.float64): ops.TYPE_F64, np.dtype(np.uint64): ops.TYPE_U64, np.dtype(np.int64): ops.TYPE_I64}
    return ops.Column(kinds[a.dtype], len(a), ops.DeviceBuffer(a.nbytes, a), zone_map=False)


def host_join(build, probe, left):
    """(probe, build) rows ascending, keys compared as doubles"""
    b, p = build.astype(np.float64) + 0.0, probe.astype(np.float64) + 0.0
    order = np.argsort(b, kind="stable")
    lo, hi = np.searchsorted(b[order], p, "left"), np.searchsorted(b[order], p, "right")
    lo, hi = np.where(np.isnan(p), 0, lo), np.where(np.isnan(p), 0, hi)
    n = hi - lo
    rows = np.repeat(np.arange(len(p)), n)
    at = np.arange(n.sum()) - np.repeat(np.cumsum(n) - n, n) + np.repeat(lo, n)
    pairs = np.stack([rows, order[at]], 1)
    if left:
        miss = np.flatnonzero(n == 0)
        pairs = np.concatenate([pairs, np.stack([miss, np.full(len(miss), NONE)], 1)])
    return pairs[np.lexsort((pairs[:, 1], pairs[:, 0]))].astype(np.uint32)


def keys(kind, ids):
    return {"u32": lambda: ids.astype(np.uint32) * np.uint32(2654435761), "i32": lambda: (ids - 5000).astype(np.int32),
            "i64": lambda: ids.astype(np.int64) * 1_000_003 - (1 << 40), "u64": lambda: ids.astype(np.uint64) << np.uint64(20),
            "i64 large": lambda: (ids.astype(np.int64) - 3) << 45, "f64": lambda: ids * 0.37 - 20.0, "f32": lambda: (ids * 0.5).astype(np.float32)}[kind]()


@pytest.mark.parametrize("left", [False, True])
@pytest.mark.parametrize("build_kind,probe_kind", [("u32", "u32"), ("i32", "i32"), ("i64", "i64"), ("u64", "u64"), ("i64 large", "i64 large"), ("f64", "f64"),
                                                   ("f32", "f32"), ("i32", "f64"), ("f32", "f64")])
@pytest.mark.parametrize("builds,probes", [(1, 1), (1, 5000), (7, 2047), (1000, 2049), (5000, 300_001), (40_000, 100_000)])
def test_equal_to_a_host_join(ops, builds, probes, build_kind, probe_kind, left):
    rng = np.random.default_rng(builds + probes)
    ids = rng.permutation(3 * builds)
    build, probe = keys(build_kind, ids[:builds]), keys(probe_kind, rng.integers(0, 3 * builds, probes))
    n, pairs = ops.hash_join(column(ops, build), column(ops, probe), left=left)
    want = host_join(build, probe, left)
    assert n == len(want)
    np.testing.assert_array_equal(pairs, want)


@pytest.mark.parametrize("case", ["repeated", "all equal", "nan", "minus zero build", "minus zero probe"])
@pytest.mark.parametrize("left", [False, True])
def test_gives_way(ops, case, left):
    rng = np.random.default_rng(len(case))
    build, probe = rng.permutation(3000)[:1000] * 0.5, rng.integers(0, 3000, 20_001) * 0.5
    if case == "repeated":
        build[17] = build[900]
    elif case == "all equal":
        build[:] = 2.5
        probe = probe[:50]
        probe[3] = 2.5
    elif case == "nan":
        build[5], probe[7] = np.nan, np.nan
    elif case == "minus zero build":
        build[build == 0.0] = -1.0          # 0.0 and -0.0 hash apart in the buckets: no zero key on the other side
        build[5] = -0.0
        probe[probe == 0.0] = 0.5
    else:
        build[build == 0.0] = 1e9
        probe[5] = -0.0
    n, pairs = ops.hash_join(column(ops, build), column(ops, probe), left=left)
    want = host_join(build, probe, left)
    if case == "minus zero probe":
        want = host_join(build, np.where(probe == 0.0, 1e10, probe), left)
    assert n == len(want)
    np.testing.assert_array_equal(pairs, want)


def test_short_output_and_count_only(ops):
    from computeql_gb300 import native as N
    rng = np.random.default_rng(9)
    build, probe = rng.permutation(5000).astype(np.uint32), rng.integers(0, 10_000, 50_000).astype(np.uint32)
    b, p = column(ops, build), column(ops, probe)
    want = host_join(build, probe, False)
    n, none = ops.hash_join(b, p, want_pairs=False)
    assert n == len(want) and none is None
    out, count, bc, pc = np.full((100, 2), 7, dtype=np.uint32), C.c_uint64(), b.c(), p.c()
    assert N.load_ops().cqlops_hash_join(C.byref(bc), C.byref(pc), 0, 0, C.byref(count), N.ptr(out), 90)
    assert count.value == len(want)
    np.testing.assert_array_equal(out[:90], want[:90])
    assert np.all(out[90:] == 7)
