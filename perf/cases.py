"""The queries whose speed is measured, each one call (or the few calls) of the operator layer that answers it.

The tables are resident in device memory, as an engine keeps them; a pass runs one query and brings its answer to
the host. Column shapes are those of the repository's benchmark tables: u32 attributes uniform below 2^20, i64 values
uniform within 2^40 of zero, f64 measures lognormal(3, 1), a region of 50 values, dictionary strings of 200 values
drawn with Zipf weights (s = 1.1), users and sessions by the million. A group-by's answer is put in order with the
keys' values, as a query that shows it does. Row sets are cut to a LIMIT a little below what the filter keeps.

Operators ("op" of a case):

  filter_sum       SELECT COUNT(*), SUM/MIN/MAX(m1), SUM/MIN/MAX(u1) WHERE region/word = .. AND u0 BETWEEN .. AND m0 > ..
  filter_rows      the row numbers WHERE (u0 in a range) OR (another column above a limit) LIMIT .., and the count of all
  group_dense      SELECT key, COUNT, SUM[, MIN, MAX](u32) GROUP BY a u32 key of few to 25000 values
  group_measures   SELECT key, SUM, AVG, MIN, MAX of two measures GROUP BY a key of at most 64 values
  group_two_keys   SELECT region, code, COUNT, SUM, AVG, MAX GROUP BY a u32 region and an i64 code
  group_having     SELECT user, COUNT, SUM(measure) GROUP BY user HAVING SUM > .. ORDER BY SUM DESC LIMIT 500, users by
                   the million
  distinct         SELECT APPROX_COUNT_DISTINCT(session) of the table or by region
  join_pairs       the (probe row, build row) pairs of an equi-join, one probe row in ten with a match
  join_sum         SELECT segment, COUNT, SUM(u32) FROM fact JOIN dim GROUP BY segment, dim keys spread over 32 bits, the
                   dim table's columns resident or on the host alone
  order_by         the row numbers ORDER BY one or two keys
  projection       SELECT * WHERE u0 > .. LIMIT ..: the filter's rows of every column of a wide table
  batch            Q dashboard queries SELECT COUNT(*), SUM(f64) WHERE .. over one table, in one call
"""
import math
import statistics

import numpy as np
import torch

from computeql_gb300 import native, ops

REGIONS, WORDS, U32_RANGE, I64_RANGE, TOP = 50, 200, 1 << 20, 1 << 40, 500


# ---------------------------------------------------------------------------------------------
# the cases

def listed():
    return [
        # the smallest call of a serving loop: one filter-aggregate over a 1M-row table, latency and launches count
        {"name": "filter_sum_1m", "op": "filter_sum", "rows": 1_000_000, "text": True},
        # a row set for the operators after it, through a generated kernel for an OR of an integer and a float range
        {"name": "filter_rows_50m", "op": "filter_rows", "rows": 50_000_003, "column": "f64", "keep": 0.02},
        # the billion-row report: 10k groups, whole numbers
        {"name": "group_dense_1b", "op": "group_dense", "rows": 1_000_000_000, "groups": 10_000, "extremes": False, "narrow": 0},
        # measures by a small attribute, the commonest group-by over floats
        {"name": "group_measures_10m", "op": "group_measures", "rows": 10_000_000, "groups": REGIONS, "measure": "f64"},
        # two keys of different types, a few hundred groups
        {"name": "group_two_keys_10m", "op": "group_two_keys", "rows": 10_000_000, "codes": 20, "measure": "f64"},
        # revenue by user: a million groups over floats, the large ones kept
        {"name": "group_having_10m", "op": "group_having", "rows": 10_000_000, "users": 1_000_000, "measure": "f64"},
        # distinct sessions of an event table
        {"name": "distinct_10m", "op": "distinct", "rows": 10_000_000, "sessions": 4_000_000, "by_region": False},
        # an equi-join whose pairs feed the next operator
        {"name": "join_pairs_10m", "op": "join_pairs", "rows": 10_000_000, "build": 1_000_000, "key": "u32", "left": False},
        # a fact table joined to a dimension by a sparse key and summed by a dimension attribute
        {"name": "join_sum_50m", "op": "join_sum", "rows": 50_000_000, "dims": 100_003, "resident": True},
        # a ranking: a float measure descending, then an integer
        {"name": "order_by_20m", "op": "order_by", "rows": 20_000_000, "keys": "f64 desc,u32"},
        # the detail view: 1 % of a wide table's rows, every column
        {"name": "projection_10m", "op": "projection", "rows": 10_000_000, "columns": 28, "keep": 0.01},
        # a dashboard's queries over one table
        {"name": "batch_50m", "op": "batch", "rows": 50_000_000, "queries": 64},
    ]


def _spread(rng, lo, hi):
    """a whole number between lo and hi, spread over their logarithm"""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["filter_sum", "filter_rows", "group_dense", "group_measures", "group_two_keys", "group_having", "distinct",
                     "join_pairs", "join_sum", "order_by", "projection", "batch"])
    if op == "filter_sum":
        return {"op": op, "rows": _spread(rng, 30_000, 100_000_000), "text": rng.random() < 0.5}
    if op == "filter_rows":
        return {"op": op, "rows": _spread(rng, 100_000, 50_000_000), "column": rng.choice(["f64", "f32", "i64", "u32"]),
                "keep": rng.choice([0.001, 0.02, 0.2])}
    if op == "group_dense":
        return {"op": op, "rows": _spread(rng, 100_000, 900_000_000), "groups": _spread(rng, 5, 25_000), "extremes": rng.random() < 0.3,
                "narrow": rng.choice([0, 0, 2])}
    if op == "group_measures":
        return {"op": op, "rows": _spread(rng, 100_000, 60_000_000), "groups": rng.randint(2, 64),
                "measure": rng.choice(["f64", "f64", "f32", "decimal"])}
    if op == "group_two_keys":
        return {"op": op, "rows": _spread(rng, 100_000, 20_000_000), "codes": _spread(rng, 3, 400),
                "measure": rng.choice(["f64", "f64", "decimal", "u32"])}
    if op == "group_having":
        rows = _spread(rng, 1_000_000, 20_000_000)
        return {"op": op, "rows": rows, "users": _spread(rng, 100_000, rows // 4), "measure": rng.choice(["f64", "f64", "u32"])}
    if op == "distinct":
        rows = _spread(rng, 100_000, 50_000_000)
        return {"op": op, "rows": rows, "sessions": _spread(rng, 20_000, rows), "by_region": rng.random() < 0.5}
    if op == "join_pairs":
        rows = _spread(rng, 100_000, 10_000_000)
        return {"op": op, "rows": rows, "build": _spread(rng, 1000, max(2000, rows // 4)), "key": rng.choice(["u32", "u32", "i64"]),
                "left": rng.random() < 0.25}
    if op == "join_sum":
        rows = _spread(rng, 100_000, 100_000_000)
        return {"op": op, "rows": rows, "dims": _spread(rng, 1000, min(1_000_000, rows // 4)), "resident": rng.random() < 0.7}
    if op == "order_by":
        return {"op": op, "rows": _spread(rng, 50_000, 20_000_000), "keys": rng.choice(["f64 desc,u32", "u32", "i64", "f64", "f32 desc", "u32,i64 desc"])}
    if op == "projection":
        return {"op": op, "rows": _spread(rng, 100_000, 20_000_000), "columns": rng.randint(6, 28), "keep": rng.choice([0.001, 0.01, 0.05])}
    return {"op": op, "rows": _spread(rng, 300_000, 50_000_000), "queries": rng.randint(8, 64)}


# ---------------------------------------------------------------------------------------------
# tables: torch tensors drawn from the seed

def _u32(g, n, below):
    return torch.randint(0, below, (n,), dtype=torch.int32, device="cuda", generator=g)


def _i64(g, n, within=I64_RANGE):
    return torch.randint(-within, within, (n,), dtype=torch.int64, device="cuda", generator=g)


def _measure(g, n):
    return torch.randn(n, dtype=torch.float64, device="cuda", generator=g).add_(3.0).exp_()


def _number(g, n, kind):
    """a column of the given kind: lognormal floats, prices in cents, or uniform whole numbers"""
    if kind == "f64":
        return _measure(g, n)
    if kind == "f32":
        return _measure(g, n).float()
    if kind == "decimal":
        cents = _u32(g, n, 1_000_000).double()
        return cents.div_(torch.full_like(cents, 100.0))     # a division, not a product with 1 / 100
    if kind == "i64":
        return _i64(g, n)
    return _u32(g, n, U32_RANGE)


def _zipf(g, n, values):
    w = torch.arange(1, values + 1, dtype=torch.float64, device="cuda") ** -1.1
    cdf = torch.cumsum(w / w.sum(), 0)
    return torch.searchsorted(cdf, torch.rand(n, dtype=torch.float64, device="cuda", generator=g)).clamp_(max=values - 1).int()


def _distinct_keys(g, n):
    """n different 32-bit words in a random order: an odd multiple of the row number, and an offset"""
    mul = int(torch.randint(1 << 20, 1 << 30, (1,), generator=g, device="cuda")) * 2 + 1
    add = int(torch.randint(0, 1 << 31, (1,), generator=g, device="cuda"))
    k = (torch.arange(n, dtype=torch.int64, device="cuda") * mul + add) & 0xFFFFFFFF
    return torch.where(k >= 1 << 31, k - (1 << 32), k).int()   # the words, as torch's signed type holds them


def _table(case, seed):
    """the case's columns, by name"""
    g = torch.Generator(device="cuda").manual_seed(seed * 2654435761 % (1 << 62) + 1)
    op, n = case["op"], case["rows"]
    if op == "filter_sum":
        return {"region": _u32(g, n, REGIONS), "word": _zipf(g, n, WORDS), "u0": _u32(g, n, U32_RANGE), "m0": _measure(g, n),
                "m1": _measure(g, n), "u1": _u32(g, n, U32_RANGE)}
    if op == "filter_rows":
        return {"u0": _u32(g, n, U32_RANGE), "v": _number(g, n, case["column"])}
    if op == "group_dense":
        return {"key": _u32(g, n, case["groups"]), "u0": _u32(g, n, 10_000)}
    if op == "group_measures":
        return {"key": _u32(g, n, case["groups"]), "m0": _number(g, n, case["measure"]), "m1": _number(g, n, case["measure"])}
    if op == "group_two_keys":
        code = torch.randint(0, case["codes"], (n,), dtype=torch.int64, device="cuda", generator=g) * 1_000_003 - (1 << 33)
        return {"region": _u32(g, n, REGIONS), "code": code, "m0": _number(g, n, case["measure"])}
    if op == "group_having":
        return {"user": _u32(g, n, case["users"]), "m0": _number(g, n, case["measure"])}
    if op == "distinct":
        return {"region": _u32(g, n, REGIONS), "session": _u32(g, n, case["sessions"]) + _u32(g, 1, 1 << 30)}
    if op == "join_pairs":
        # ten times as many key values as build rows: a probe row matches one time in ten
        span = 10 * case["build"]
        keys, matches = torch.randperm(span, device="cuda", generator=g), n // 10
        build = keys[: case["build"]]
        at = torch.randint(case["build"], span, (n,), dtype=torch.int64, device="cuda", generator=g)
        at[:matches] = torch.randint(0, case["build"], (matches,), dtype=torch.int64, device="cuda", generator=g)
        probe = keys[at][torch.randperm(n, device="cuda", generator=g)]
        if case["key"] == "i64":
            return {"build": build * 1_000_003 - (1 << 40), "probe": probe * 1_000_003 - (1 << 40)}
        return {"build": build.int(), "probe": probe.int()}
    if op == "join_sum":
        key = _distinct_keys(g, case["dims"])
        pick = torch.randint(0, case["dims"], (n,), dtype=torch.int64, device="cuda", generator=g)
        return {"dim_key": key, "segment": _u32(g, case["dims"], 20), "fact_key": key[pick], "u0": _u32(g, n, 10_000)}
    if op == "order_by":
        kinds = [k.split()[0] for k in case["keys"].split(",")]
        return {f"k{i}": _number(g, n, kind) for i, kind in enumerate(kinds)}
    if op == "projection":
        kinds = ["u32", "u32", "f64", "u32", "i64", "u32", "f64"]
        return {f"c{i}": _number(g, n, kinds[i % len(kinds)]) for i in range(case["columns"])}
    # batch: 4 u32 below 2^16 and 4 f64 in [0, 1)
    t = {f"u{i}": _u32(g, n, 1 << 16) for i in range(4)}
    t.update({f"d{i}": torch.rand(n, dtype=torch.float64, device="cuda", generator=g) for i in range(4)})
    return t


class _DeviceArray:
    def __init__(self, pointer, count, kind):
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": kind, "data": (pointer, False), "version": 3}


def _buffer(t):
    """a device buffer of the framework with the tensor's values"""
    size = t.numel() * t.element_size()
    buf = ops.DeviceBuffer((size + 15) & ~15)
    kind = {1: "|u1", 2: "<i2", 4: "<i4", 8: "<i8"}[t.element_size()]
    raw = {1: torch.uint8, 2: torch.int16, 4: torch.int32, 8: torch.int64}[t.element_size()]
    there = torch.as_tensor(_DeviceArray(native.load_cuda().cqlcuda_buffer_device_pointer(buf.handle), t.numel(), kind), device="cuda")
    there.copy_(t.view(raw))
    torch.cuda.synchronize()
    return buf


def _column(t, unsigned=True, narrow=0):
    ctype = {torch.int32: ops.TYPE_U32 if unsigned else ops.TYPE_I32, torch.int64: ops.TYPE_I64, torch.float32: ops.TYPE_F32,
             torch.float64: ops.TYPE_F64}[t.dtype]
    lo, hi = (x.item() for x in t.aminmax())
    if ctype == ops.TYPE_U32 and lo < 0:
        lo, hi = 0, 0xFFFFFFFF            # words past 2^31 - 1
    zone = (float(lo), float(hi))
    if narrow == 2 and hi - lo < 65536:
        return ops.Column(ctype, t.numel(), _buffer((t - lo).to(torch.int16)), width=2, base=lo, zone=zone)
    return ops.Column(ctype, t.numel(), _buffer(t), zone=zone)


# ---------------------------------------------------------------------------------------------
# what a program has in hand before the call

def _words():
    return [f"word{i:03d}" for i in range(WORDS)]


def _quantile(p):
    """the value a lognormal(3, 1) measure is above with probability p"""
    return math.exp(3.0 + statistics.NormalDist().inv_cdf(1.0 - p))


def _rng(seed):
    return np.random.default_rng(seed + 77)


def _filter_sum_literals(seed):
    r = _rng(seed)
    lo = int(r.integers(0, U32_RANGE // 4))
    return {"region": int(r.integers(0, REGIONS)), "word": int(r.integers(0, 8)), "lo": lo, "hi": lo + U32_RANGE // 2,
            "m": round(_quantile(0.4 + 0.3 * float(r.random())), 3)}


def _filter_rows_literals(case, seed):
    lo = int(_rng(seed).integers(0, U32_RANGE // 2))
    half = case["keep"] / 2      # each side of the OR keeps half
    limit = {"f64": _quantile(half), "f32": _quantile(half), "i64": int(I64_RANGE * (1 - 2 * half)), "u32": int(U32_RANGE * (1 - half))}
    return lo, lo + max(1, int(U32_RANGE * half)), limit[case["column"]]


def _having_limit(case):
    per_user = case["rows"] / case["users"]
    mean, sd = (math.exp(3.5), math.sqrt((math.e - 1) * math.exp(7))) if case["measure"] == "f64" else (U32_RANGE / 2, U32_RANGE / math.sqrt(12))
    return per_user * mean + 2.6 * math.sqrt(per_user * (mean * mean + sd * sd))


# a dashboard's WHERE shapes over 4 u32 and 4 f64 columns, ? standing for a literal: short ranges, chains, ORs
_SHAPES = [
    "(< u0 ?)", "(and (>= u1 ?) (< d0 ?))", "(and (> d1 ?) (<= d1 ?))", "(or (< u2 ?) (> d2 ?))",
    "(and (and (>= u0 ?) (<= u1 ?)) (> d3 ?))", "(and (or (< u3 ?) (> d0 ?)) (<= d1 ?))", "(and (and (> u1 ?) (> u2 ?)) (and (< d2 ?) (< d3 ?)))",
    "(or (and (< u0 ?) (< d0 ?)) (and (> u3 ?) (> d3 ?)))", "(> d2 ?)", "(and (and (> d0 ?) (> d1 ?)) (or (< u2 ?) (and (> u3 ?) (< d3 ?))))",
]


def _batch_queries(case, seed):
    """(where, shape, literals, summed column) per query"""
    r = _rng(seed)
    out = []
    for q in range(case["queries"]):
        shape = _SHAPES[q % len(_SHAPES)]
        parts, literals = shape.split("?"), []
        where = parts[0]
        for before, after in zip(parts, parts[1:]):
            column = before.split()[-1]
            lit = int(r.integers(0, 1 << 16)) if column[0] == "u" else round(float(r.random()), 6)
            literals.append(lit)
            where += repr(lit) + after
        out.append((where, shape, literals, f"d{q % 4}"))
    return out


def prepare(case, seed):
    op, t = case["op"], _table(case, seed)
    s = {"op": op, "case": case}
    if op == "filter_sum":
        lit = _filter_sum_literals(seed)
        cols = {k: _column(t[k]) for k in ("region", "u0", "m0", "m1", "u1")}
        test = f"(= region {lit['region']})"
        if case["text"]:
            cols["word"] = ops.StringColumn.from_codes(t["word"].cpu().numpy().view(np.uint32), _words())
            test = f"(= word '{_words()[lit['word']]}')"
            del cols["region"]
        s["program"] = ops.Program(f"(and (and {test} (> m0 {lit['m']})) (and (>= u0 {lit['lo']}) (<= u0 {lit['hi']})))", cols)
    elif op == "filter_rows":
        lo, hi, limit = _filter_rows_literals(case, seed)
        cols = {k: _column(v) for k, v in t.items()}
        s["program"] = ops.Program(f"(or (and (>= u0 {lo}) (< u0 {hi})) (> v {limit!r}))", cols)
    elif op == "group_dense":
        s.update(key=_column(t["key"], narrow=case["narrow"]), u0=_column(t["u0"]))
    elif op in ("group_measures", "group_two_keys", "distinct", "projection"):
        s.update({k: _column(v) for k, v in t.items()})
        if op == "projection":
            s["selection"] = ops.DeviceBuffer(case["rows"] * 4)
    elif op == "group_having":
        s.update({k: _column(v) for k, v in t.items()})
        s["out"] = ops.HashOutputs(case["users"], 1)
    elif op == "join_pairs":
        s.update(build=_column(t["build"]), probe=_column(t["probe"]))
    elif op == "join_sum":
        s.update(fact_key=_column(t["fact_key"]), u0=_column(t["u0"]), dim_key=t["dim_key"].cpu().numpy().view(np.uint32),
                 segment=t["segment"].cpu().numpy().astype(np.float64))
        s["columns"] = {"dim_key_col": _column(t["dim_key"]), "dim_group_col": _column(t["segment"])} if case["resident"] else {}
    elif op == "order_by":
        s["keys"] = [_column(v) for v in t.values()]
        s["desc"] = [1 if k.endswith("desc") else 0 for k in case["keys"].split(",")]
        s["out"] = np.zeros(case["rows"], dtype=np.uint32)
    else:
        cols = {k: _column(v) for k, v in t.items()}
        queries = _batch_queries(case, seed)
        s["programs"] = [ops.Program(q[0], cols) for q in queries]
        s["sums"] = [q[3] for q in queries]
    return s


# ---------------------------------------------------------------------------------------------
# one query

def _kept(case):
    """filter_rows: a little below the part of the rows that one side of its OR or both keep"""
    return 0.98 * (case["keep"] - case["keep"] ** 2 / 4)


def _limit(expected):
    """a LIMIT that a filter expected to keep so many rows reaches"""
    return max(1, int(expected - 8 * math.sqrt(expected)))


def _answer(keys, r, by=None):
    """a group-by's answer with its keys' values, in key order (or the order `by` gives)"""
    values = ops.gather_rows(keys, rows=r["repr_row"].astype(np.uint32))
    order = np.lexsort(values[::-1]) if by is None else by
    return {"keys": [v[order] for v in values], "counts": r["counts"][order], "results": r["results"][order]}


def run(s):
    op, case = s["op"], s["case"]
    if op == "filter_sum":
        return ops.fused_aggregate(s["program"], ["m1", "u1"])
    if op == "filter_rows":
        count, rows, _ = ops.scan_filter(s["program"], want_rows=True, max_rows=_limit(case["rows"] * _kept(case)))
        return count, rows.view(np.int32)
    if op == "group_dense":
        u = s["u0"]
        if case["extremes"]:
            return ops.group_dense(s["key"], [ops.FUNC_COUNT, ops.FUNC_SUM, ops.FUNC_MIN, ops.FUNC_MAX], [None, u, u, u])[1:]
        lo, counts, sums, _, _ = ops.group_dense(s["key"], [ops.FUNC_COUNT, ops.FUNC_SUM], [None, u])
        return lo, counts, sums
    if op == "group_measures":
        m0, m1 = s["m0"], s["m1"]
        r = ops.group_hash([s["key"]], [ops.FUNC_SUM, ops.FUNC_AVG, ops.FUNC_MIN, ops.FUNC_MAX], [m0, m1, m1, m1], group_hint=case["groups"])
        return _answer([s["key"]], r)
    if op == "group_two_keys":
        keys, m = [s["region"], s["code"]], s["m0"]
        r = ops.group_hash(keys, [ops.FUNC_COUNT, ops.FUNC_SUM, ops.FUNC_AVG, ops.FUNC_MAX], [None, m, m, m],
                           group_hint=REGIONS * case["codes"], max_groups=REGIONS * case["codes"])
        return _answer(keys, r)
    if op == "group_having":
        r = ops.group_hash([s["user"]], [ops.FUNC_SUM], [s["m0"]], group_hint=case["users"], out=s["out"])
        kept = np.flatnonzero(ops.having("v0 > lit[0]", [r["results"][:, 0]], [_having_limit(case)]) != 0)
        top = kept[np.argsort(-r["results"][kept, 0], kind="stable")[:TOP]]
        return _answer([s["user"]], {k: r[k][top] for k in ("repr_row", "counts", "results")}, np.arange(len(top)))
    if op == "distinct":
        if not case["by_region"]:
            return ops.group_hash([], [ops.FUNC_ACD], [s["session"]])["results"]
        return _answer([s["region"]], ops.group_hash([s["region"]], [ops.FUNC_ACD], [s["session"]], group_hint=REGIONS, max_groups=REGIONS))
    if op == "join_pairs":
        count, pairs = ops.hash_join(s["build"], s["probe"], left=case["left"])
        return count, pairs.view(np.int32)
    if op == "join_sum":
        r = ops.join_aggregate(s["fact_key"], [ops.FUNC_COUNT, ops.FUNC_SUM], [None, s["u0"]], s["dim_key"], group_values=[s["segment"]],
                               **s["columns"])
        return r["dim_row"], r["results"]
    if op == "order_by":
        return ops.sort_rows(s["keys"], s["desc"], out=s["out"]).view(np.int32)
    if op == "projection":
        columns = [s[f"c{i}"] for i in range(case["columns"])]
        n = ops.scan_select(columns[:1], [(0, ops.CMP_GT, int(U32_RANGE * (1 - case["keep"])))], s["selection"])
        return ops.gather_rows(columns, selection=s["selection"], count=min(n, _limit(case["rows"] * case["keep"])))
    return ops.batch_aggregate(s["programs"], s["sums"])[:2]


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without

def work(case):
    """The columns a query reads once and its answer written once; flops: the comparisons and additions."""
    op, n = case["op"], case["rows"]
    size = {"f64": 8, "i64": 8, "decimal": 8, "f32": 4, "u32": 4}
    if op == "filter_sum":
        return {"bytes": n * (4 + 4 + 8 + 8 + 4), "flops": 10 * n}
    if op == "filter_rows":
        return {"bytes": n * (4 + size[case["column"]]) + 4 * n * _kept(case), "flops": 3 * n}
    if op == "group_dense":
        return {"bytes": n * ((case["narrow"] or 4) + 4) + case["groups"] * 40, "flops": (4 if case["extremes"] else 2) * n}
    if op == "group_measures":
        return {"bytes": n * (4 + 2 * size[case["measure"]]) + case["groups"] * 40, "flops": 5 * n}
    if op == "group_two_keys":
        return {"bytes": n * (4 + 8 + size[case["measure"]]) + REGIONS * case["codes"] * 50, "flops": 4 * n}
    if op == "group_having":
        return {"bytes": n * (4 + size[case["measure"]]) + case["users"] * 24, "flops": 2 * n}
    if op == "distinct":
        return {"bytes": n * (8 if case["by_region"] else 4), "flops": n}
    if op == "join_pairs":
        pairs = n if case["left"] else n / 10
        return {"bytes": (n + case["build"]) * size[case["key"]] + 8 * pairs, "flops": n}
    if op == "join_sum":
        return {"bytes": n * 8 + case["dims"] * 8, "flops": 2 * n}
    if op == "order_by":
        return {"bytes": n * (sum(size[k.split()[0]] for k in case["keys"].split(",")) + 4), "flops": n}
    if op == "projection":
        kinds = ["u32", "u32", "f64", "u32", "i64", "u32", "f64"]
        row = sum(size[kinds[i % len(kinds)]] for i in range(case["columns"]))
        return {"bytes": 4 * n + 2 * n * case["keep"] * row, "flops": n}
    return {"bytes": n * (4 * 4 + 4 * 8) + case["queries"] * 16, "flops": 4 * n * case["queries"]}


# ---------------------------------------------------------------------------------------------
# the same answers in 64 bits

def _grouped(key, groups, m0, m1=None):
    """per present group: its number, rows, sum of m0, and of m1 (m0 by default) sum, minimum and maximum"""
    m0 = m0.double()
    m1 = m0 if m1 is None else m1.double()
    key = key.long()
    z = torch.zeros(groups, dtype=torch.float64, device=key.device)
    count = torch.bincount(key, minlength=groups)
    mn = torch.full_like(z, math.inf).scatter_reduce_(0, key, m1, "amin")
    mx = torch.full_like(z, -math.inf).scatter_reduce_(0, key, m1, "amax")
    some = torch.nonzero(count).flatten()
    return some, count[some], torch.bincount(key, m0, groups)[some], torch.bincount(key, m1, groups)[some], mn[some], mx[some]


def _sum_min_max(m):
    m = m.double()
    return m.sum().item(), m.min().item(), m.max().item()


def exact(case, seed):
    op = case["op"]
    if op in ("filter_rows", "group_dense", "distinct", "join_pairs", "order_by"):
        return None          # row numbers and whole numbers; a sketch's estimate
    t = _table(case, seed)
    if op == "filter_sum":
        lit = _filter_sum_literals(seed)
        mask = t["word"] == lit["word"] if case["text"] else t["region"] == lit["region"]
        mask &= (t["m0"] > lit["m"]) & (t["u0"] >= lit["lo"]) & (t["u0"] <= lit["hi"])
        if not mask.any():
            return None
        per = [_sum_min_max(t[c][mask]) for c in ("m1", "u1")]
        return (float(mask.sum().item()), *([p[i] for p in per] for i in range(3)))
    if op == "group_measures":
        some, count, s0, s1, mn, mx = _grouped(t["key"], case["groups"], t["m0"], t["m1"])
        return {"keys": [None], "counts": None, "results": torch.stack([s0, s1 / count, mn, mx], 1)}
    if op == "group_two_keys":
        code = torch.div(t["code"] + (1 << 33), 1_000_003, rounding_mode="floor")
        some, count, s0, _, _, mx = _grouped(t["region"].long() * case["codes"] + code, REGIONS * case["codes"], t["m0"])
        return {"keys": [None, None], "counts": None, "results": torch.stack([count.double(), s0, s0 / count, mx], 1)}
    if op == "group_having":
        some, _, s0, _, _, _ = _grouped(t["user"], case["users"], t["m0"])
        return {"keys": [None], "counts": None, "results": s0[s0 > _having_limit(case)].sort(descending=True).values[:TOP].reshape(-1, 1)}
    if op == "join_sum":
        order = torch.argsort(t["dim_key"])
        dim = order[torch.searchsorted(t["dim_key"][order], t["fact_key"])]
        some, count, s0, _, _, _ = _grouped(t["segment"][dim], 20, t["u0"])
        first = torch.full((20,), 1 << 40, device="cuda").scatter_reduce_(0, t["segment"][dim].long(), dim, "amin")
        met = torch.argsort(first[some])
        return None, torch.stack([count.double(), s0], 1)[met]
    if op == "projection":
        rows = torch.nonzero(t["c0"] > int(U32_RANGE * (1 - case["keep"]))).flatten()[: _limit(case["rows"] * case["keep"])]
        return [c[rows] if c.dtype == torch.float64 else None for c in t.values()]
    sums = []
    for _, shape, literals, column in _batch_queries(case, seed):
        mask = _evaluate(shape.replace("(", " ( ").replace(")", " ) ").split(), t, iter(literals))
        sums.append(t[column][mask].sum().item())
    return None, np.array(sums)


def _evaluate(tokens, t, literals):
    """the mask of a shape's s-expression, its literals in order"""
    tokens.pop(0)
    op = tokens.pop(0)
    if op in ("and", "or"):
        a = _evaluate(tokens, t, literals)
        b = _evaluate(tokens, t, literals)
        tokens.pop(0)
        return a & b if op == "and" else a | b
    column, _, _ = t[tokens.pop(0)], tokens.pop(0), tokens.pop(0)
    x = next(literals)
    return {"<": column < x, "<=": column <= x, ">": column > x, ">=": column >= x}[op]
