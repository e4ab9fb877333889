"""GROUP BY over keys whose number takes all 64 bits, with a hint of few groups: keys that differ in their top bits alone
stay apart, by the groups of the member lists (path 1)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
COUNT, SUM, MIN, MAX = 0, 1, 3, 4
N = 400_003


def values(form, groups):
    """`groups` key tuples in pairs that differ in the top bits of the keys' number"""
    half = (groups + 1) // 2
    i = np.arange(half)
    if form == "f64":                                   # x and -x: the sign bit; powers of two: the exponent's top bits
        v = (i + 1) * 0.5
        return [np.concatenate([v, -v])[:groups]]
    if form == "f64 exponents":                         # 0 and 2, and 2^k with 2^(k + 512)
        v = 2.0 ** (i - 300)
        return [np.concatenate([v, v * 2.0 ** 512, [0.0, 2.0]])[-groups:]]
    if form == "i64":                                   # no range: the keys are met as their doubles' bits
        v = i.astype(np.int64) * 3 + 1
        return [np.concatenate([v, -v])[:groups]]
    if form == "i64 0 and 2":
        return [np.array([0, 2, -2, 1 << 61, -(1 << 61)] * groups, dtype=np.int64)[:min(groups, 5)]]
    if form == "u64":
        v = (i.astype(np.uint64) << np.uint64(20)) + np.uint64(3)
        return [np.concatenate([v, v + np.uint64(1 << 63)])[:groups]]
    if form == "f32,f32":
        v = ((i + 1) * 0.25).astype(np.float32)
        return [np.concatenate([v, -v])[:groups], np.full(groups, 1.5, dtype=np.float32)]
    assert form == "u32,u32"                            # no ranges: the first key's top bit is the number's
    v = i.astype(np.uint32) * np.uint32(7)
    return [np.concatenate([v, v + np.uint32(1 << 31)])[:groups], np.full(groups, 9, dtype=np.uint32)]


RANGED = {"f64", "f64 exponents", "f32,f32"}            # (floats number by their bits, range or not)


@pytest.mark.parametrize("form", ["f64", "f64 exponents", "i64", "i64 0 and 2", "u64", "f32,f32", "u32,u32"])
@pytest.mark.parametrize("hint", [2, 50, 256, 257])
def test_top_bits_of_the_number(gpu, form, hint):
    from computeql_gb300 import ops
    rng = np.random.default_rng(hint)
    vals = values(form, 2 if hint == 2 else 40)
    pick = rng.integers(0, len(vals[0]), N)
    keys = [v[pick] for v in vals]
    kinds = {"u4": ops.TYPE_U32, "f4": ops.TYPE_F32, "f8": ops.TYPE_F64, "u8": ops.TYPE_U64, "i8": ops.TYPE_I64}
    cols = [ops.Column(kinds[k.dtype.str[1:]], N, ops.DeviceBuffer(k.nbytes, k), zone=(float(k.min()), float(k.max())) if form in RANGED else None)
            for k in keys]
    x = rng.integers(-10**6, 10**6, N).astype(np.int32)
    xc = ops.Column.from_numpy(x)
    funcs, args = [COUNT, SUM, MIN, MAX], [None, xc, xc, xc]

    def groups(path):
        r = ops.group_hash(cols, funcs, args, group_hint=hint, path=path, max_groups=N)
        rows = r["repr_row"].astype(np.int64)
        return {tuple(k[row].item() for k in keys): r["results"][g].tolist() for g, row in enumerate(rows)}, r["groups"]

    (got, n), (lists, m) = groups(0), groups(1)
    want = {}
    for g in range(len(vals[0])):
        rows = x[pick == g].astype(np.int64)
        want[tuple(v[g].item() for v in vals)] = [float(len(rows)), float(rows.sum()), float(rows.min()), float(rows.max())]
    assert n == m == len(want)
    assert got == lists == want
