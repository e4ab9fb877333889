"""Scratch of the forms that another form may follow: evictable as soon as the call is over, and a failed allocation of
it leaves the query to the form behind it with the same answer."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
N = 200_003


@pytest.fixture(scope="module")
def env(gpu):
    from computeql_gb300 import ops
    rng = np.random.default_rng(7)
    build = ops.Column.from_numpy(rng.permutation(1 << 20)[:50_001].astype(np.uint32))
    probe = ops.Column.from_numpy(rng.integers(0, 1 << 20, N).astype(np.uint32))
    key = ops.Column.from_numpy(rng.integers(0, 2 ** 32, N).astype(np.uint32) % np.uint32(100_003) * np.uint32(40_000))
    value = ops.Column.from_numpy(rng.integers(0, 1000, N).astype(np.uint32))
    dims = rng.choice(2 ** 32, 70_001, replace=False).astype(np.uint32)
    fact = ops.Column.from_numpy(dims[rng.integers(0, len(dims), N)])
    seg = rng.integers(0, 20, len(dims)).astype(np.float64)

    def joined():
        r = ops.join_aggregate(fact, [0, 1], [None, value], dims, group_values=[seg])
        return sorted(zip(seg[r["dim_row"].astype(np.int64)].tolist(), r["results"].tolist()))

    def grouped():
        r = ops.group_hash([key], [0, 1], [None, value], group_hint=100_003, max_groups=N)
        return sorted(map(tuple, r["results"].tolist()))

    return gpu.load_cuda(), {"join_pairs": lambda: ops.hash_join(build, probe)[1].tolist(), "join_sum": joined, "group_by": grouped}


@pytest.mark.parametrize("name", ["join_pairs", "join_sum", "group_by"])
def test_scratch_is_evictable_after_the_call(env, name):
    lib, queries = env
    want = queries[name]()
    before = lib.cqlcuda_memory_stats()
    freed = lib.cqlcuda_pool_evict(2 ** 64 - 1)            # the same epoch: only what is idle goes
    assert freed >= 50_001 * 2 * 8 and lib.cqlcuda_memory_stats().pool_evictions > before.pool_evictions
    assert queries[name]() == want


@pytest.mark.parametrize("name", ["join_pairs", "join_sum"])
def test_no_room_for_the_first_allocations(env, name):
    """the first allocations of these queries are the fast form's: the form behind it answers"""
    lib, queries = env
    want = queries[name]()
    for k in (1, 2, 3):
        lib.cqlcuda_pool_begin_epoch()
        lib.cqlcuda_pool_evict(2 ** 64 - 1)
        target = lib.cqlcuda_memory_stats().alloc_calls + k
        lib.cqlcuda_set_fault_alloc_at(target)
        try:
            got = queries[name]()
        finally:
            lib.cqlcuda_set_fault_alloc_at(0)
        assert lib.cqlcuda_memory_stats().alloc_calls >= target
        assert got == want
