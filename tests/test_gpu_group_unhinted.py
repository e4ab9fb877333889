"""GROUP BY many groups without a hint, or with one far too low: the exact tables find their room in few passes, and the
groups are those of the data."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def passes(lib, native, call):
    """the call's result and how often the exact tables' kernel ran"""
    lib.cqlcuda_kernel_profile_enable(1)
    lib.cqlcuda_kernel_profile_reset()
    result = call()
    name, count, i, ran = native.C.c_char_p(), native.C.c_uint64(), 0, 0
    while lib.cqlcuda_kernel_profile_entry(i, native.C.byref(name), None, native.C.byref(count)):
        ran += count.value if name.value == b"cql_group_exact" else 0
        i += 1
    lib.cqlcuda_kernel_profile_enable(0)
    return result, ran


@pytest.mark.parametrize("rows", [700, 5000, 20_001, 50_000, 100_003, 300_000, 1_000_000])
@pytest.mark.parametrize("groups", ["all", "quarter"])
@pytest.mark.parametrize("hint", [0, 40])
def test_many_groups(gpu, rows, groups, hint):
    from computeql_gb300 import ops
    lib = gpu.load_cuda()
    rng = np.random.default_rng(rows)
    g = rng.permutation(rows) if groups == "all" else rng.integers(0, rows // 4, rows)
    key, x = g * 0.5 - 3.0, rng.lognormal(3.0, 1.0, rows)
    kc, xc = ops.Column.from_numpy(key), ops.Column.from_numpy(x)
    run = lambda: ops.group_hash([kc], [0, 3, 4], [None, xc, xc], group_hint=hint, max_groups=rows)
    run()
    r, ran = passes(lib, gpu, run)
    # one pass where the first table has room, else one that finds none and one with room for every row; tables in shared
    # memory, which few groups are thought to be worth, come first
    assert 1 <= ran <= (3 if hint or rows >= 500_000 else 2), ran
    at = g[r["repr_row"].astype(np.int64)]
    counts = np.bincount(g)
    assert r["groups"] == len(np.unique(g)) == len(np.unique(at)) and np.array_equal(r["counts"], counts[at])
    low, high = np.full(len(counts), np.inf), np.full(len(counts), -np.inf)
    np.minimum.at(low, g, x)
    np.maximum.at(high, g, x)
    assert np.array_equal(r["results"][:, 1], low[at]) and np.array_equal(r["results"][:, 2], high[at])
