"""Data outside a fast form, met by one CTA, ends the form's pass over the rest: its kernel takes a small part of the time
that the whole table takes, wherever the form then gives way, and the answer is the general form's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
N = 20_000_003


def nanoseconds(lib, native, prefix, call):
    """the call's result and the time of the kernels whose name starts with `prefix`"""
    lib.cqlcuda_kernel_profile_enable(1)
    lib.cqlcuda_kernel_profile_reset()
    result = call()
    total, i = 0, 0
    name, ns = native.C.c_char_p(), native.C.c_uint64()
    while lib.cqlcuda_kernel_profile_entry(i, native.C.byref(name), native.C.byref(ns), None):
        if name.value.decode().startswith(prefix):
            total += ns.value
        i += 1
    lib.cqlcuda_kernel_profile_enable(0)
    return result, total


@pytest.mark.parametrize("groups", [1000, 500_000])        # tables in shared memory, in device memory
def test_group_by_values_outside_the_window(gpu, groups):
    from computeql_gb300 import ops
    lib = gpu.load_cuda()
    rng = np.random.default_rng(groups)
    key = ops.Column.from_numpy(rng.integers(0, groups, N).astype(np.uint32))
    x = rng.lognormal(3.0, 1.0, N)
    tiny = x.copy()
    tiny[::1009] *= 1e-30
    cols = [ops.Column.from_numpy(v) for v in (x, tiny)]
    run = lambda c: ops.group_hash([key], [0, 1], [None, c], group_hint=groups, max_groups=groups)
    for c in cols:
        run(c)
    _, whole = nanoseconds(lib, gpu, "cql_group_exact", lambda: run(cols[0]))
    r, early = nanoseconds(lib, gpu, "cql_group_exact", lambda: run(cols[1]))
    assert early < whole / 2, (early, whole)
    k = key.buffer.read(np.uint32)
    counts = np.bincount(k, minlength=groups)
    sums = np.bincount(k, weights=tiny, minlength=groups)
    row = k[r["repr_row"].astype(np.int64)]
    assert np.array_equal(r["counts"], counts[row]) and len(row) == (counts > 0).sum()
    assert np.allclose(r["results"][:, 1], sums[row], rtol=1e-12, atol=0)


@pytest.mark.parametrize("where", ["all over", "first", "last"])
def test_batch_with_values_outside_their_range(gpu, where):
    from computeql_gb300 import ops
    lib = gpu.load_cuda()
    rng = np.random.default_rng(3)
    w, v = rng.random(N), rng.random(N)      # (conditions on whole numbers of small range would be answered from a table)
    bad = v.copy()
    if where == "all over":
        bad[::1009] = np.nan
    else:
        bad[0 if where == "first" else N - 1] = 1e9
    wc = ops.Column.from_numpy(w)
    cols = [{"w": wc, "v": ops.Column(ops.TYPE_F64, N, ops.DeviceBuffer(a.nbytes, a), zone=(0.0, 1.0), zone_map=False)} for a in (v, bad)]
    progs = [[ops.Program(f"(< w {(q + 1) / 70!r})", c) for q in range(64)] for c in cols]
    run = lambda p, form=8: ops.batch_aggregate(p, ["v"] * 64, form)
    for p in progs:
        run(p)
    _, whole = nanoseconds(lib, gpu, "qk_batch_rank", lambda: run(progs[0]))
    (c, s, _), early = nanoseconds(lib, gpu, "qk_batch_rank", lambda: run(progs[1]))
    c8, s8, _ = run(progs[1], 8 | (1 << 24))
    assert np.array_equal(c, c8) and np.array_equal(s.view(np.uint64), s8.view(np.uint64))
    assert np.array_equal(c, [(w < (q + 1) / 70).sum() for q in range(64)])
    assert whole > 0 and early > 0
    if where != "last":
        assert early < whole / 2, (early, whole)


def test_batch_over_a_range_that_is_not_finite(gpu):
    """a column of NaN and numbers, its range taken from it: the register form at once"""
    from computeql_gb300 import ops
    lib = gpu.load_cuda()
    rng = np.random.default_rng(4)
    n = 100_003
    w, v = rng.random(n), rng.random(n)
    v[::97] = np.nan
    cols = {"w": ops.Column.from_numpy(w), "v": ops.Column.from_numpy(v), "d": ops.Column.from_numpy(rng.random(n))}
    progs = [ops.Program(f"(< w {(q + 1) / 20!r})", cols) for q in range(16)]
    (c, s, _), ranked = nanoseconds(lib, gpu, "qk_batch_rank", lambda: ops.batch_aggregate(progs, ["v"] * 16))
    c8, s8, _ = ops.batch_aggregate(progs, ["v"] * 16, 8 | (1 << 24))
    assert ranked == 0
    assert np.array_equal(c, c8) and np.array_equal(s.view(np.uint64), s8.view(np.uint64))
    # the other columns' batches still run as ranks
    (c, s, _), ranked = nanoseconds(lib, gpu, "qk_batch_rank", lambda: ops.batch_aggregate(progs, ["d"] * 16))
    assert ranked > 0 and np.array_equal(c, c8)


@pytest.mark.parametrize("kind", ["u32", "f64", "i64"])
def test_join_whose_build_keys_repeat(gpu, kind):
    from computeql_gb300 import ops
    lib = gpu.load_cuda()
    rng = np.random.default_rng(5)
    n, probes = 10_000_019, 3001
    unique = rng.permutation(n)
    repeated = unique % (n // 3)
    at = rng.integers(0, n, probes)
    dtype = {"u32": np.uint32, "f64": np.float64, "i64": np.int64}[kind]
    kinds = {"u32": ops.TYPE_U32, "f64": ops.TYPE_F64, "i64": ops.TYPE_I64}
    cols = [ops.Column(kinds[kind], len(a), ops.DeviceBuffer(a.nbytes, a), zone_map=False) for a in (unique.astype(dtype), repeated.astype(dtype), at.astype(dtype))]
    run = lambda b: ops.hash_join(b, cols[2])
    for b in cols[:2]:
        run(b)
    (n0, pairs), whole = nanoseconds(lib, gpu, "cql_join_unique_build", lambda: run(cols[0]))
    assert n0 == probes and np.array_equal(unique[pairs[:, 1]], at[pairs[:, 0]])
    (n1, pairs), early = nanoseconds(lib, gpu, "cql_join_unique_build", lambda: run(cols[1]))
    counts = np.bincount(repeated, minlength=n)
    assert n1 == counts[at].sum() and np.array_equal(repeated[pairs[:, 1]], at[pairs[:, 0]])
    assert early < whole / 2, (early, whole)
