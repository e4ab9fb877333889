"""The batched scan over ranks (the default form) against the register form of the same batch, query by query:
equal counts and equal sums to the bit (both add the same scaled integers), over every column type, every
comparison, literals at the types' edges, tile remainders, few and many queries, and batches whose literals do
not fit the rank form's cut tables."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REGISTERS = 4     # rows a thread: an explicit register form


@pytest.fixture(scope="module")
def ops(gpu):
    from computeql_gb300 import ops as o
    return o


def _table(n, seed):
    r = np.random.default_rng(seed)
    t = {"u": r.integers(0, 1 << 32, n, dtype=np.uint32), "i": r.integers(-(1 << 31), 1 << 31, n).astype(np.int32),
         "f": r.normal(size=n).astype(np.float32), "d": r.normal(size=n) * 1e3, "w": r.integers(-(1 << 40), 1 << 40, n)}
    t["v"] = r.lognormal(3.0, 1.0, n)
    for name, special in (("u", [0, 1, 2**32 - 1]), ("i", [0, -1, 2**31 - 1, -2**31])):
        at = r.integers(0, n, 4 * len(special))
        t[name][at] = np.resize(np.array(special, dtype=t[name].dtype), len(at))
    return t


def _special_floats(t):
    """compared, never summed: signed zeros, infinities and NaN of both signs"""
    for name, kind in (("f", np.float32), ("d", np.float64)):
        x = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, -np.nan, np.finfo(kind).tiny, np.finfo(kind).max, -np.finfo(kind).max], dtype=kind)
        t[name][: len(x)] = x[: len(t[name])]
        t[name][-len(x):] = x[-len(t[name][-len(x):]):]
    return t


LITERALS = {"u": ["0", "1", "4294967295", "4294967296", "-1", "2147483648", "1000000.5"],
            "i": ["0", "-1", "2147483647", "-2147483648", "2147483648", "-0.5", "12345"],
            "f": ["0.0", "-0.0", "0.1", "-1.25", "1e300", "-1e300", "0.5"],
            "d": ["0.0", "-0.0", "0.1", "-125.5", "1e308", "-1e308", "3.0"]}


def _queries(count, seed, sums, shapes=24):
    """conditions of one to four comparisons over all columns, operators and literals, in that many shapes"""
    r = np.random.default_rng(seed)
    skeletons = []
    for _ in range(min(count, shapes)):
        parts = [(r.integers(6), "uifd"[r.integers(4)]) for _ in range(int(r.integers(1, 5)))]
        joins = [(["and", "or"][r.integers(2)], int(r.integers(3))) for _ in parts[1:]]
        skeletons.append((parts, joins))
    out = []
    for q in range(count):
        parts, joins = skeletons[q % len(skeletons)]
        text = [f"({['=', '!=', '<', '>', '<=', '>='][op]} {c} {LITERALS[c][r.integers(len(LITERALS[c]))]})" for op, c in parts]
        for join, at in joins:
            a, b = text.pop(0), text.pop(0)
            text.insert(min(at, len(text)), f"({join} {a} {b})")
        out.append((text[0], sums[q % len(sums)]))
    return out


def _agree(ops, cols, qs):
    progs = [ops.Program(w, cols) for w, _ in qs]
    names = [s for _, s in qs]
    c, s, _ = ops.batch_aggregate(progs, names)
    c4, s4, _ = ops.batch_aggregate(progs, names, REGISTERS)
    assert np.array_equal(c, c4), [(w, int(a), int(b)) for (w, _), a, b in zip(qs, c, c4) if a != b][:4]
    assert np.array_equal(s.view(np.uint64), s4.view(np.uint64)), [(w, n, a, b) for (w, n), a, b in zip(qs, s, s4) if a != b][:4]
    return progs, c, s


def _columns(ops, t):
    return {n: ops.Column.from_numpy(a) for n, a in t.items()}


@pytest.mark.parametrize("rows", [1, 3, 127, 2047, 2048, 2049, 100_003])
@pytest.mark.parametrize("queries", [2, 17, 60])
def test_forms_agree(ops, rows, queries):
    t = _special_floats(_table(rows, rows))
    cols = _columns(ops, t)
    _agree(ops, cols, _queries(queries, queries + rows, ["v", "w", "u", "i", None]))


def test_ranks_run_by_default(ops):
    cols = _columns(ops, _table(5000, 1))
    progs = [ops.Program(w, cols) for w, _ in _queries(20, 3, ["v"])]
    assert "cql_rk" in ops.batch_source(progs, ["v"] * 20)[0]
    assert "cql_rk" not in ops.batch_source(progs, ["v"] * 20, REGISTERS)[0]


@pytest.mark.parametrize("queries", [40, 400])
def test_large_table_with_six_planes(ops, queries):
    """from 2^15 rows an accumulator the summands take six bytes; the oracle counts the matches"""
    from tests.where_shapes import oracle_mask
    t = _table(5_000_001, 9)
    cols = _columns(ops, t)
    qs = _queries(queries, 8, ["v", "d", "f", "i", "w", None])
    progs, c, _ = _agree(ops, cols, qs)
    for i in range(0, queries, 13):
        assert c[i] == oracle_mask(progs[i], t).sum(), qs[i]


@pytest.mark.parametrize("queries", [30, 100, 300, 700])
def test_many_cuts(ops, queries):
    """each query brings cuts of its own: launches of fewer queries, and the register form where a few
    queries already bring too many"""
    t = _table(70_001, 4)
    cols = _columns(ops, t)
    qs = [(f"(and (>= d {k * 1.5 - 300}) (< u {k * 1000003 % 4294967296}))", "v") for k in range(queries)]
    qs += [(f"(or (and (> d {k}.25) (< d {k}.5)) (and (> d -{k}.5) (< d -{k}.25)))", "w") for k in range(queries // 30)]
    _agree(ops, cols, qs)


def test_value_outside_its_range(ops):
    """summed values far outside the column's stated range, or NaN, do not fit the planes: the batch runs in
    the register form"""
    t = _table(30_000, 6)
    t["v"][12_345] = 1e12
    t["v"][23_456] = np.nan
    cols = _columns(ops, t)
    cols["v"].zone = (0.0, 100.0)
    progs = [ops.Program(w, cols) for w, _ in _queries(12, 5, ["v"])]
    c, s, _ = ops.batch_aggregate(progs, ["v"] * 12)
    c8, s8, _ = ops.batch_aggregate(progs, ["v"] * 12, 8 | (1 << 24))
    assert np.array_equal(c, c8) and np.array_equal(s.view(np.uint64), s8.view(np.uint64))


def test_catalog_prepared_for_both_forms(ops):
    """a catalog's batches whose cuts fit or do not fit take kernels compiled when it was prepared"""
    from computeql_gb300 import native
    t = _table(20_000, 7)
    cols = _columns(ops, t)
    few = [(f"(> d {k}.5)", "v") for k in range(40)]
    many = [(f"(> d {k}.5)", "v") for k in range(400)]
    cat = ops.BatchCatalog()
    p_few, p_many = ([ops.Program(w, cols) for w, _ in qs] for qs in (few, many))
    C = native.C
    ptrs = (C.c_void_p * 40)(*[C.addressof(p.prog) for p in p_few])
    sums = np.full(40, p_few[0].index("v"), dtype=np.int32)
    assert native.load_ops().cqlops_batch_prepare(cat.h, ptrs, 40, p_few[0]._cols, len(p_few[0].columns), native.ptr(sums), 8)
    n = C.c_uint64()
    native.load_cuda().cqlcuda_generated_kernel_stats(C.byref(n), None)
    before = n.value
    for progs in (p_few, p_many):
        c, s, _ = cat.aggregate(progs, ["v"] * len(progs), 8)
        native.load_cuda().cqlcuda_generated_kernel_stats(C.byref(n), None)
        assert n.value == before
        for q in (0, 17, 39, len(progs) - 1):
            m = t["d"] > q + 0.5
            assert c[q] == m.sum() and abs(s[q] - t["v"][m].sum()) <= 1e-12 * t["v"].sum()
    cat.close()


@pytest.mark.parametrize("rows", [3, 4099])
def test_bool_column(ops, rows):
    """a column of one byte a row, compared and summed"""
    r = np.random.default_rng(rows)
    b, v = r.integers(0, 2, rows, dtype=np.uint8), r.random(rows)
    cols = {"b": ops.Column(6, rows, ops.DeviceBuffer(rows, b), zone=(0.0, 1.0), zone_map=False), "v": ops.Column.from_numpy(v)}
    qs = [("(= b 1)", "v"), ("(and (!= b 1) (< v 0.25))", "v"), ("(or (>= b 1) (> v 0.5))", "b")]
    _, c, s = _agree(ops, cols, qs)
    want = [b == 1, (b != 1) & (v < 0.25), (b >= 1) | (v > 0.5)]
    assert [int(x) for x in c] == [int(w.sum()) for w in want] and s[2] == b[want[2]].sum()


def test_new_literals_compile_nothing(ops):
    """a batch of several launches and known shapes, with other literals and so other launches, reuses its kernel"""
    from computeql_gb300 import native
    t = _table(20_000, 12)
    cols = _columns(ops, t)
    n = native.C.c_uint64()
    compiled = []
    for seed in (1, 2, 3):
        r = np.random.default_rng(seed)
        qs = [(w, "v") for k in range(200) for w in (f"(> d {r.normal() * 1e3:.6f})", f"(and (< u {r.integers(1 << 32)}) (<= d {r.normal():.6f}))")]
        progs = [ops.Program(w, cols) for w, _ in qs]
        c, _, shapes = ops.batch_aggregate(progs, ["v"] * len(qs))
        assert shapes == 2 and c[0] == (t["d"] > float(qs[0][0].split()[-1][:-1])).sum()
        native.load_cuda().cqlcuda_generated_kernel_stats(native.C.byref(n), None)
        compiled.append(n.value)
    assert compiled[0] == compiled[1] == compiled[2]
