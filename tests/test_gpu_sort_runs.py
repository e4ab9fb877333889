"""ORDER BY keys whose prefixes many rows share: runs around what the runs pass takes, runs of equal keys, and which path
each goes by - against a stable sort on the host."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def kernels(lib, native, call):
    """the call's result and how often each kernel ran"""
    lib.cqlcuda_kernel_profile_enable(1)
    lib.cqlcuda_kernel_profile_reset()
    result = call()
    name, count, i, ran = native.C.c_char_p(), native.C.c_uint64(), 0, {}
    while lib.cqlcuda_kernel_profile_entry(i, native.C.byref(name), None, native.C.byref(count)):
        if count.value:
            ran[name.value.decode()] = count.value
        i += 1
    lib.cqlcuda_kernel_profile_enable(0)
    return result, ran


def hashed(rng, n, per):
    """u32 values over the whole range, `per` rows each on average"""
    v = np.unique(rng.integers(0, 2**32, max(n // per, 1), dtype=np.uint64).astype(np.uint32))
    return v[rng.integers(0, len(v), n)]


@pytest.mark.parametrize("n", [17_000, 50_001, 300_007, 2_000_003])
@pytest.mark.parametrize("per", [3, 20, 60, 100, 127, 200, 2000])
def test_runs_of_any_length(gpu, n, per):
    from computeql_gb300 import ops
    lib = gpu.load_cuda()
    rng = np.random.default_rng(n + per)
    a, b = hashed(rng, n, per), rng.integers(0, 1 << 20, n).astype(np.uint32)
    cols = [ops.Column.from_numpy(a), ops.Column.from_numpy(b)]
    got, ran = kernels(lib, gpu, lambda: ops.sort_rows(cols))
    np.testing.assert_array_equal(got, np.lexsort([b, a]))
    # not both: the runs pass is not begun where the sample shows runs that it cannot take
    assert not ("cql_sort_runs" in ran and "cql_sort_keys" in ran), ran
    if per < 16 or per >= 60:         # (the sample draws the line at 16 rows, give or take its own spread)
        assert ("cql_sort_keys" in ran) == (per >= 60), ran


@pytest.mark.parametrize("n", [17_000, 300_007])
@pytest.mark.parametrize("lengths", [[127, 128, 129], [1, 128], [129, 1], [64, 65, 63], [1000, 1, 2]])
@pytest.mark.parametrize("state", ["sorted", "one swap", "shuffled"])
def test_runs_around_the_limit(gpu, n, lengths, state):
    """runs of given lengths at every place of the tiles, their rows in order, all but two, or in none"""
    from computeql_gb300 import ops
    rng = np.random.default_rng(n + lengths[0])
    sizes = np.resize(lengths, n)
    sizes = sizes[:np.searchsorted(np.cumsum(sizes), n) + 1]
    a = np.repeat(np.arange(len(sizes), dtype=np.uint64) * np.uint64((1 << 32) // len(sizes) | 1) % np.uint64(1 << 32), sizes)[:n].astype(np.uint32)
    a.sort()
    b = np.arange(n, dtype=np.uint32) * np.uint32(3)
    if state == "one swap":
        at = n // 2 - (a[n // 2] != a[n // 2 - 1])
        b[at], b[at - 1] = b[at - 1], b[at]
    elif state == "shuffled":
        b = rng.permutation(b)
    cols = [ops.Column.from_numpy(a), ops.Column.from_numpy(b)]
    np.testing.assert_array_equal(ops.sort_rows(cols), np.lexsort([b, a]))
    np.testing.assert_array_equal(ops.sort_rows(cols, [1, 0]), np.lexsort([b, -a.astype(np.int64)]))


@pytest.mark.parametrize("keys", [["f64"], ["i64"], ["u32", "f64"], ["f64", "u32", "i64"]])
@pytest.mark.parametrize("values", [1, 3, 300])
def test_runs_of_equal_keys(gpu, keys, values):
    from computeql_gb300 import ops
    rng = np.random.default_rng(values)
    n = 100_003
    pick = rng.integers(0, values, n)
    pool = {"f64": rng.lognormal(3.0, 2.0, values), "i64": rng.integers(-2**50, 2**50, values), "u32": rng.integers(0, 2**32, values).astype(np.uint32)}
    arrays = [pool[k][pick] for k in keys]
    kinds = {"f64": ops.TYPE_F64, "i64": ops.TYPE_I64, "u32": ops.TYPE_U32}
    cols = [ops.Column(kinds[k], n, ops.DeviceBuffer(a.nbytes, a), zone_map=False) for k, a in zip(keys, arrays)]
    np.testing.assert_array_equal(ops.sort_rows(cols), np.lexsort(arrays[::-1]))
