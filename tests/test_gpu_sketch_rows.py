"""The one-pass HyperLogLog registers (cql_hll_rows) through the C ABI: of a whole table and per value of a small-range
key, bit for bit the oracle's."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
COUNT, SUM, MAX, ACD = 0, 1, 4, 5


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


@pytest.mark.parametrize("dtype", [np.uint32, np.int32, np.float32, np.float64, np.int64, np.uint64])
@pytest.mark.parametrize("n,values", [(1, 0), (2049, 1), (70_001, 0), (70_001, 64)])
def test_sketch_registers(ops, dtype, n, values):
    """registers of a column of each type, of the whole table and per value of a small-range key, bit for bit"""
    rng = np.random.default_rng(n + values)
    v = (rng.integers(-2**31 if np.dtype(dtype).kind != "u" else 0, 2**31, n) * (1 if np.dtype(dtype).itemsize == 4 else 12345)).astype(dtype)
    w = rng.integers(0, 9, n).astype(np.uint32)
    key = (rng.integers(0, max(values, 1), n) + 3).astype(np.uint32)
    keys = [column(ops, key, (3.0, 2.0 + max(values, 1)))] if values else []
    vc, wc = column(ops, v), column(ops, w)
    res = ops.group_hash(keys, [ACD, COUNT, ACD] + ([SUM, MAX] if values else []), [vc, None, wc] + ([wc, wc] if values else []))
    regs = ops.group_hash_registers()
    assert len(regs) == 2 * res["groups"]
    assert res["groups"] == (len(np.unique(key)) if values else 1)
    for g in range(res["groups"]):
        m = key == key[int(res["repr_row"][g])] if values else np.ones(n, bool)
        assert res["counts"][g] == m.sum() == res["results"][g, 1]
        for j, a in enumerate((v, w)):
            want = oracle.hll_registers(a[m].astype(np.float64))
            assert np.array_equal(regs[2 * g + j], want)
            assert res["results"][g, 2 * j] == np.round(oracle.hll_estimate(want))
        if values:
            assert res["results"][g, 3:].tolist() == [float(w[m].sum()), float(w[m].max())]
