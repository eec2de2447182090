"""The calls whose speed is followed: what a query engine on top of this library
has it do, over the range of sizes it meets.

A case is one query step through the public entry points: a grouped aggregation
with its result ordered by key, an equi-join, a sort or radix partition, a
filter, a dictionary encoding, or a batch of string pipelines.  Results are read
where the library left them (torch tensors over its buffers, no copies).

Two things are ordered here because the library leaves them in any order: the
groups of HASH and PARTITION group-bys (ordered by key, as a query's ORDER BY
has it, with the library's argsort and gather), and the groups of the batched
pipelines (ordered by their sums).  The partition-hash join, whose pairs come in
no fixed order, is left out for that reason.
"""
import ctypes as C
import math

import torch

import eiger_b200 as gx
from eiger_b200 import batch, selector

I64, F64 = torch.int64, torch.float64
KEY_TYPES = {"int32": torch.int32, "int64": torch.int64, "float32": torch.float32, "float64": torch.float64,
             "int16": torch.int16}

# Aggregation lists: requests, and the value columns (type) that they read.
AGGS = {
    "sum_count": ([(0, gx.SUM), (0, gx.COUNT_ALL)], ["int64"]),
    "seven": ([(0, gx.SUM), (0, gx.MIN), (0, gx.MAX), (1, gx.SUM), (1, gx.MIN), (1, gx.MAX), (0, gx.COUNT_ALL)],
              ["int64", "float64"]),
    "mixed": ([(1, gx.SUM), (0, gx.MAX), (0, gx.COUNT_ALL)], ["int64", "float64"]),
    "average": ([(0, gx.AVG), (1, gx.SUM)], ["int32", "float64"]),
}
ALGOS = {"auto": gx.AUTO_ALGO, "learned": gx.AUTO_ALGO, "hash": gx.HASH, "sort": gx.SORT, "partition": gx.PARTITION}


def listed():
    return [
        # A dashboard query over a few thousand rows: latency, launches and host work.
        dict(name="groupby_small", op="groupby", rows=5_003, groups=61, key="int32", skew=0.0, aggs="sum_count",
             algo="auto"),
        # SUM and COUNT of 2^20 rows over 1024 keys, the small hash group-by of the tests and the smoke run.
        dict(name="groupby_1m", op="groupby", rows=1 << 20, groups=1024, key="int32", skew=0.0, aggs="sum_count",
             algo="hash"),
        # The benchmark's step: 2^28 rows, 2^16 groups, SUM/MIN/MAX of two columns and COUNT, learned selector.
        dict(name="groupby_headline", op="groupby", rows=1 << 28, groups=1 << 16, key="int32", skew=0.0,
             aggs="seven", algo="learned"),
        # Many groups, 8-byte keys with Zipf 1.0 frequencies, an aggregation list without a compiled plan.
        dict(name="groupby_keys64_zipf", op="groupby", rows=50_000_021, groups=3_000_000, key="int64", skew=1.0,
             aggs="mixed", algo="auto"),
        # A fact table joined to a dimension with dense keys: the benchmark's 2^24 x 2^28 row-id join.
        dict(name="join_dense", op="join", build=1 << 24, probe=1 << 28, key="int32", spread=1, copies=1, skew=0.0,
             form="rowids", algo="sort"),
        # A table join on sparse 8-byte keys, a payload column on each side.
        dict(name="join_sparse_table", op="join", build=1_000_003, probe=30_000_001, key="int64", spread=1_000_003,
             copies=1, skew=0.0, form="table", algo="sort"),
        # ORDER BY a 4-byte key with row ids at the benchmark's size.
        dict(name="sort_pairs", op="sort", form="pairs", rows=1 << 28, key="int32", value="int64", order="asc"),
        # The row order of a small float64 column, descending (a top-n list).
        dict(name="argsort_small", op="sort", form="argsort", rows=100_003, key="float64", value="int64",
             order="desc"),
        # Radix partition of 8-byte keys with 4-byte payloads into 256 parts (a shuffle).
        dict(name="partition_pairs", op="partition", rows=50_000_017, key="int64", value="int32", first=0, bits=8),
        # WHERE date BETWEEN on the benchmark's rows: two 8-byte columns and the date kept for 40%.
        dict(name="filter_date", op="filter", rows=1 << 28, columns=3, predicates=1, keep=0.4),
        # Order-preserving dictionary codes of a 4-byte column with 2^16 values.
        dict(name="dictionary_ordered", op="dictionary", rows=100_000_007, values=1 << 16, key="int32",
             mode="ordered"),
        # Uneven string pipelines (encode, date range, SUM and COUNT) in one launch.
        dict(name="batch_strings", op="batch", instances=128, min_log2=12, max_log2=22, values=10_000, keep=0.4),
    ]


def _log_int(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))


def draw(rng):
    op = rng.choice(["groupby", "groupby", "groupby", "join", "join", "sort", "sort", "partition", "filter",
                     "dictionary", "batch"])
    if op == "groupby":
        rows = _log_int(rng, 1 << 10, 1 << 27)
        return dict(op=op, rows=rows, groups=_log_int(rng, 1, max(1, rows // 2)), key=rng.choice(["int32", "int64"]),
                    skew=rng.choice([0.0, 0.0, 1.0]), aggs=rng.choice(sorted(AGGS)),
                    algo=rng.choice(["auto", "auto", "learned", "sort", "partition"]))
    if op == "join":
        probe = _log_int(rng, 1 << 11, 1 << 27)
        algo = rng.choice(["sort", "sort", "hash"])
        return dict(op=op, build=_log_int(rng, 1 << 10, max(1 << 10, min(probe // 2, 1 << 24))), probe=probe,
                    key=rng.choice(["int32", "int64"]), spread=rng.choice([1, 8, 100]),
                    copies=1 if algo == "hash" else rng.choice([1, 1, 2]), skew=rng.choice([0.0, 0.0, 1.0]),
                    form=rng.choice(["rowids", "table"]), algo=algo)
    if op == "sort":
        return dict(op=op, form=rng.choice(["pairs", "pairs", "keys", "argsort"]), rows=_log_int(rng, 1 << 10, 1 << 27),
                    key=rng.choice(["int32", "int32", "int64", "float32", "float64", "int16"]),
                    value=rng.choice(["int32", "int64"]), order=rng.choice(["asc", "desc"]))
    if op == "partition":
        return dict(op=op, rows=_log_int(rng, 1 << 10, 1 << 27), key=rng.choice(["int32", "int64"]),
                    value=rng.choice(["int32", "int64"]), first=rng.choice([0, 0, 5]), bits=rng.randint(4, 12))
    if op == "filter":
        return dict(op=op, rows=_log_int(rng, 1 << 10, 1 << 27), columns=rng.randint(1, 4),
                    predicates=rng.randint(1, 2), keep=round(rng.uniform(0.05, 0.95), 3))
    if op == "dictionary":
        rows = _log_int(rng, 1 << 10, 1 << 27)
        return dict(op=op, rows=rows, values=_log_int(rng, 4, max(4, min(rows // 4, 1 << 22))),
                    key=rng.choice(["int32", "int64"]), mode=rng.choice(["ordered", "hash", "ready"]))
    return dict(op=op, instances=_log_int(rng, 4, 128), min_log2=12, max_log2=rng.randint(14, 20),
                values=_log_int(rng, 100, 10_000), keep=round(rng.uniform(0.1, 0.9), 3))


# --------------------------------------------------------------------------- inputs

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _ranks(n, groups, skew, g):
    """n ranks in [0, groups): uniform, or with P(rank r) close to 1 / (r + 1)."""
    if skew == 0.0:
        return torch.randint(0, groups, (n,), device="cuda", dtype=I64, generator=g)
    u = torch.rand(n, device="cuda", dtype=F64, generator=g)
    return (torch.exp(u * math.log(groups + 1.0)) - 1.0).long().clamp_(0, groups - 1)


def _all_ranks(n, groups, skew, g):
    """The same with every rank taken at least once (groups <= n), so that a result has `groups` rows."""
    r = _ranks(n, groups, skew, g)
    step = n // groups
    at = torch.arange(groups, device="cuda") * step
    at += torch.randint(0, step, (groups,), device="cuda", generator=g)
    r[at] = torch.randperm(groups, device="cuda", generator=g)
    return r


def _scattered(n, seed):
    """A permutation of 0..n-1 without long runs: i * odd + shift modulo n."""
    a = 2 * int(n * 0.3) + 1 + 2 * (seed % 1009)
    while math.gcd(a, n) != 1:
        a += 1
    return (torch.arange(n, device="cuda") * a + seed) % n


def _stride(groups, key):
    """Keys of consecutive ranks lie this far apart: the keys span their type."""
    return max(1, ((1 << 31) - 1) // groups) if key == "int32" else max(1, (1 << 62) // groups)


def _group_inputs(case, seed):
    g = _generator(seed)
    n = case["rows"]
    ranks = _all_ranks(n, case["groups"], case["skew"], g)
    key = ((ranks - case["groups"] // 2) * _stride(case["groups"], case["key"])).to(KEY_TYPES[case["key"]])
    vals = []
    for t in AGGS[case["aggs"]][1]:
        if t == "float64":
            vals.append(torch.rand(n, device="cuda", dtype=F64, generator=g))
        else:
            vals.append(torch.randint(0, (1 << 31) - 1, (n,), device="cuda", dtype=KEY_TYPES[t], generator=g))
    return ranks, key, vals


def _any_values(n, kind, g):
    """Values over the whole range of a type (floats: normal)."""
    t = KEY_TYPES[kind]
    if t.is_floating_point:
        return torch.randn(n, device="cuda", dtype=t, generator=g)
    lim = torch.iinfo(t)
    return torch.randint(lim.min, lim.max, (n,), device="cuda", dtype=t, generator=g)


def prepare(case, seed):
    op = case["op"]
    s = dict(case=case)
    if op == "groupby":
        if case["algo"] == "learned":
            selector.install()
        _, s["key"], s["vals"] = _group_inputs(case, seed)
    elif op == "join":
        g = _generator(seed)
        nb, t, step = case["build"], KEY_TYPES[case["key"]], case["spread"]
        unique = max(1, nb // case["copies"])
        step = min(step, ((1 << 31) - 1) // (3 * unique)) if case["key"] == "int32" else step
        ids = torch.randperm(unique, device="cuda", generator=g)
        if case["copies"] > 1:
            ids = torch.cat([ids] * case["copies"])[:nb]
        s["build_key"] = (ids * max(1, step)).to(t)
        ranks = _ranks(case["probe"], unique, case["skew"], g)
        ranks[3::10] += unique  # one probe row of ten has no match
        s["probe_key"] = (ranks * max(1, step)).to(t)
        if case["form"] == "table":
            s["build_pay"] = _any_values(s["build_key"].numel(), "int64", g)
            s["probe_pay"] = _any_values(case["probe"], "int64", g)
    elif op in ("sort", "partition"):
        g = _generator(seed)
        s["key"] = _any_values(case["rows"], case["key"], g)
        if case.get("form", "pairs") == "pairs":
            s["value"] = torch.arange(case["rows"], device="cuda", dtype=KEY_TYPES[case["value"]])
    elif op == "filter":
        g = _generator(seed)
        n = case["rows"]
        width = max(1, round(case["keep"] * 2557))
        lo = (2557 - width) // 2
        # Days [lo, lo + width) for the share `keep` of the rows, at scattered places.
        place, inside = _scattered(n, seed), int(case["keep"] * n)
        day = torch.randint(0, 1 << 30, (n,), device="cuda", dtype=I64, generator=g)
        day = torch.where(place < inside, lo + day % width, (lo + width + day % max(1, 2557 - width)) % 2557)
        cols = [day.to(torch.int32)]
        for kind in ("int64", "float64", "int32")[: case["columns"] - 1]:
            cols.append(_any_values(n, kind, g))
        s["columns"] = cols
        s["predicates"] = [gx.predicate(0, gx.CMP_BETWEEN, lo, lo + width)]
        if case["predicates"] > 1:  # keeps half of those
            if len(cols) > 1:
                last = torch.where(cols[-1] >= 0, cols[-1], -1 - cols[-1])
                cols[-1] = torch.where(place < inside // 2, last, -1 - last)
            s["predicates"].append(gx.predicate(len(cols) - 1, gx.CMP_GE, 0))
    elif op == "dictionary":
        g = _generator(seed)
        ranks = _all_ranks(case["rows"], case["values"], 0.0, g)
        step = _stride(case["values"], case["key"])
        s["column"] = ((ranks - case["values"] // 2) * step).to(KEY_TYPES[case["key"]])
        if case["mode"] == "ready":  # every value but one of eight
            r = torch.randperm(case["values"], device="cuda", generator=g)[: max(1, case["values"] * 7 // 8)]
            s["dictionary"] = ((r - case["values"] // 2) * step).to(KEY_TYPES[case["key"]])
    else:
        s["instances"], _ = batch.make_instances(case["instances"], seed, case["min_log2"], case["max_log2"],
                                                 case["values"], keep=case["keep"])
        s["plan"] = batch.Plan(s["instances"], case["values"])
        res = (gx.BatchResult * case["instances"])()
        gx.check(gx.lib.gx_batch_results(s["plan"].handle, res))
        s["sums"] = [_over(r.sum, case["values"], gx.INT64, s["plan"]) for r in res]
        s["counts"] = [_over(r.count, case["values"], gx.INT64, s["plan"]) for r in res]
    return s


# --------------------------------------------------------------------------- calls

_TYPESTR = {gx.INT8: "|i1", gx.INT16: "<i2", gx.INT32: "<i4", gx.INT64: "<i8", gx.UINT8: "|u1", gx.FLOAT32: "<f4",
            gx.FLOAT64: "<f8"}


class _Buffer:
    """Device memory of the library as torch sees it, with what owns it."""

    def __init__(self, ptr, n, gx_type, owner):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=(n,), typestr=_TYPESTR[gx_type], data=(ptr, False), strides=None,
                                             version=3)


class _Column:
    """An owned result column, returned to the library's pool when dropped."""

    def __init__(self):
        self.c = gx.OwnedColumn()

    def view(self):
        return gx.ColumnView(self.c.data, self.c.size, self.c.type, 0)

    def tensor(self):
        return _over(self.c.data, self.c.size, self.c.type, self)

    def __del__(self):
        if self.c.data and gx.lib is not None:
            gx.lib.gx_free(self.c.data, None)


def _over(ptr, n, gx_type, owner):
    if not n:
        return torch.empty(0, dtype=gx.torch_dtype(gx_type), device="cuda")
    return torch.as_tensor(_Buffer(ptr, n, gx_type, owner), device="cuda")


def _table(t):
    cols = [t.column(i) for i in range(t.num_columns)]
    return [_over(v.data, v.size, v.type, t) for v in cols]


def _ordered(t):
    """A result table's columns in the order of column 0."""
    stream = gx._stream_ptr(None)
    key, at = _Column(), _Column()
    gx.check(gx.lib.gx_argsort(t.column(0), 0, -1, gx.ASCENDING, None, 0, stream, C.byref(key.c), C.byref(at.c)))
    out = [key.tensor()]
    for i in range(1, t.num_columns):
        c = _Column()
        gx.check(gx.lib.gx_gather(at.view(), t.column(i), stream, C.byref(c.c)))
        out.append(c.tensor())
    return out


def _sort_pairs(key, value, order, first=0, end=-1):
    k, v = _Column(), _Column()
    gx.check(gx.lib.gx_sort_column_pair(gx.view(key), gx.view(value), first, end, order, None, 0,
                                        gx._stream_ptr(None), C.byref(k.c), C.byref(v.c)))
    return [k.tensor(), v.tensor()]


def _encode(s, ordered):
    codes, n = _Column(), C.c_int64()
    fn = gx.lib.gx_dictionary_encode_with_order if ordered else gx.lib.gx_dictionary_encode
    gx.check(fn(gx.view(s["column"]), gx.INT32, 0, 0.25, gx._stream_ptr(None), C.byref(codes.c), C.byref(n)))
    return codes, int(n.value)


def run(s):
    case = s["case"]
    op = case["op"]
    if op == "groupby":
        hint = gx.make_hint(ALGOS[case["algo"]],
                            selector=gx.SELECT_LEARNED if case["algo"] == "learned" else gx.SELECT_HEURISTIC)
        t = gx.groupby([s["key"]], s["vals"], AGGS[case["aggs"]][0], hint)
        return _table(t) if case["algo"] == "sort" else _ordered(t)
    if op == "join":
        hint = gx.make_join_hint(gx.JOIN_SORT if case["algo"] == "sort" else gx.JOIN_HASH)
        if case["form"] == "rowids":
            return _table(gx.inner_eq_join_rowids(s["build_key"], s["probe_key"], hint))
        return _table(gx.inner_eq_join([s["build_key"], s["build_pay"]], [s["probe_key"], s["probe_pay"]], hint))
    if op == "sort":
        order = gx.ASCENDING if case["order"] == "asc" else gx.DESCENDING
        if case["form"] == "pairs":
            return _sort_pairs(s["key"], s["value"], order)
        k, i = _Column(), _Column()
        if case["form"] == "keys":
            gx.check(gx.lib.gx_sort_column(gx.view(s["key"]), 0, -1, order, None, 0, gx._stream_ptr(None),
                                           C.byref(k.c)))
            return [k.tensor()]
        gx.check(gx.lib.gx_argsort(gx.view(s["key"]), 0, -1, order, None, 0, gx._stream_ptr(None), C.byref(k.c),
                                   C.byref(i.c)))
        return [k.tensor(), i.tensor()]
    if op == "partition":
        k, v = _Column(), _Column()
        gx.check(gx.lib.gx_partition_column_pair(gx.view(s["key"]), gx.view(s["value"]), case["first"],
                                                 case["first"] + case["bits"], None, 0, gx._stream_ptr(None),
                                                 C.byref(k.c), C.byref(v.c)))
        return [k.tensor(), v.tensor()]
    if op == "filter":
        return _table(gx.select(s["columns"], s["predicates"]))
    if op == "dictionary":
        if case["mode"] == "ready":
            codes = _Column()
            gx.check(gx.lib.gx_dictionary_encode_with_dict(gx.view(s["column"]), gx.view(s["dictionary"]), gx.INT32,
                                                           gx._stream_ptr(None), C.byref(codes.c)))
            return [codes.tensor()]
        codes, n = _encode(s, case["mode"] == "ordered")
        if case["mode"] == "ordered":
            return [codes.tensor(), n]
        # Hash codes come in no fixed order: what is asked of them is the rows of each value.
        t = gx.groupby([codes.view()], [s["column"]], [(0, gx.ANY), (0, gx.COUNT_ALL)], gx.make_hint(gx.HASH, n))
        v = [t.column(i) for i in range(3)]
        k, c = _Column(), _Column()
        gx.check(gx.lib.gx_sort_column_pair(v[1], v[2], 0, -1, gx.ASCENDING, None, 0, gx._stream_ptr(None),
                                            C.byref(k.c), C.byref(c.c)))
        return [k.tensor(), c.tensor(), n]
    s["plan"].run()
    return _sort_pairs(torch.cat(s["sums"]), torch.cat(s["counts"]), gx.DESCENDING)


# --------------------------------------------------------------------------- what a pass cannot do without

def _size(kind):
    return torch.empty(0, dtype=KEY_TYPES[kind]).element_size()


def work(case):
    op = case["op"]
    if op == "groupby":
        reqs, cols = AGGS[case["aggs"]]
        row = _size(case["key"]) + sum(_size(t) for t in cols)
        return {"bytes": case["rows"] * row + case["groups"] * (_size(case["key"]) + 8 * len(reqs)), "flops": 0}
    if op == "join":
        kw = _size(case["key"])
        pay = 8 if case["form"] == "table" else 0
        matches = 0.9 * case["probe"] * case["copies"]
        out = 16 if case["form"] == "rowids" else kw + 16
        return {"bytes": (case["build"] + case["probe"]) * (kw + pay) + matches * out, "flops": 0}
    if op == "sort":
        read = _size(case["key"]) + (_size(case["value"]) if case["form"] == "pairs" else 0)
        written = read + (8 if case["form"] == "argsort" else 0)
        return {"bytes": case["rows"] * (read + written), "flops": 0}
    if op == "partition":
        return {"bytes": case["rows"] * 2 * (_size(case["key"]) + _size(case["value"])), "flops": 0}
    if op == "filter":
        row = sum((4, 8, 8, 4)[: case["columns"]])
        kept = case["keep"] * (0.5 if case["predicates"] > 1 and case["columns"] > 1 else 1.0)
        return {"bytes": case["rows"] * row * (1.0 + kept), "flops": 0}
    if op == "dictionary":
        return {"bytes": case["rows"] * (_size(case["key"]) + 4), "flops": 0}
    # Dates and offsets of every row, strings (20 bytes on average) and amounts of the kept ones.
    a, b = case["min_log2"], case["max_log2"]
    rows = case["instances"] * (2.0 ** b - 2.0 ** a) / ((b - a) * math.log(2.0))
    return {"bytes": rows * (12 + case["keep"] * 28) + 16 * case["instances"] * case["values"], "flops": 0}


def tolerance(case):
    # Keys, counts, integer aggregates, row ids and moved values are the same
    # bits whatever the order of the work.  float64 sums differ by their order:
    # up to 1.3e-13 of the result against torch's sums of few, large groups.
    if case["op"] == "groupby" and "float64" in AGGS[case["aggs"]][1]:
        return {"rel": 5e-13}
    # Equal sums of different counts may come in either order: 1.3e-5 of the
    # values differed between two runs.
    if case["op"] == "batch":
        return {"rel": 0.0, "differ": 5e-5}
    return "exact"


def exact(case, seed):
    """The grouped aggregates in 64 bits by torch; the other cases compute nothing in floating point."""
    if case["op"] != "groupby":
        return None
    ranks, key, vals = _group_inputs(case, seed)
    n = case["groups"]
    count = torch.bincount(ranks, minlength=n)
    present = torch.nonzero(count).squeeze(1)
    out = [((present - n // 2) * _stride(n, case["key"])).to(key.dtype)]
    for col, kind in AGGS[case["aggs"]][0]:
        v = vals[col]
        if kind == gx.COUNT_ALL:
            r = count
        elif kind in (gx.SUM, gx.AVG):
            wide = v.double() if v.is_floating_point() else v.long()
            r = torch.zeros(n, dtype=wide.dtype, device="cuda").index_add_(0, ranks, wide)
            if kind == gx.AVG:
                r = r.double() / count
        else:
            r = torch.zeros(n, dtype=v.dtype, device="cuda").scatter_reduce_(
                0, ranks, v, "amin" if kind == gx.MIN else "amax", include_self=False)
        out.append(r[present])
    return out
