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
