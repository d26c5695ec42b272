"""Performance cases of the public entry points: what a query engine calls this library for.

A case is a dict of plain values. Its "kind" is the entry point:

  group   groupby() of one key column: filter, then sums, means, minima, maxima and the row count
          of every group, ordered by the key (the reference's own group-by tests end in `.sort`)
  pair    groupby() of two key columns with many groups, ordered by both keys
  q1      groupby() of two Bool keys with expression aggregates and a date filter (a few groups
          over many rows: the shape of TPC-H query 1)
  filter  filter_columns(): every column compacted by a predicate
  order   sort_columns(): a table ordered by some of its columns, whole or its first rows
  batch   groupby_batched(): many independent queries in one call, their results collected into
          one table ordered by query and key with sort_columns()

Every output column comes back whole, values and validity bitmap. Rows are in a defined order, so
that two runs give the same rows at the same places.
"""

import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "polars-metal_b200"))

from polars_b200 import _abi as A  # noqa: E402
from polars_b200 import datagen  # noqa: E402
from polars_b200 import ColumnData, filter_columns, groupby, groupby_batched, sort_columns  # noqa: E402
from polars_b200._native import prepare_batched  # noqa: E402

DEV = "cuda"
FLOATS = {"f64": torch.float64, "f32": torch.float32}
INTS = {"i64": torch.int64, "i32": torch.int32}


# ------------------------------------------------------------------------------- the cases
def listed():
    return [
        # a dashboard's query over a small table: launches, synchronisations and the host's own work
        {"name": "group 20k", "kind": "group", "rows": 20_000, "groups": 1000, "zipf": 0.0, "key": "i64",
         "key_nulls": 0.0, "float": "f64", "int": "i64", "nulls": 0.01, "filter": "one", "inputs": "device",
         "output": "host"},
        # the small benchmark workload: 1M rows, 1000 groups, results as host arrays
        {"name": "group 1m", "kind": "group", "rows": 1_000_000, "groups": 1000, "zipf": 0.0, "key": "i64",
         "key_nulls": 0.0, "float": "f64", "int": "i64", "nulls": 0.01, "filter": "one", "inputs": "device",
         "output": "host"},
        # columns that live in host memory, as an engine's data frame holds them
        {"name": "group 3m from host", "kind": "group", "rows": 3_000_001, "groups": 20_000, "zipf": 0.5,
         "key": "i32", "key_nulls": 0.0, "float": "f32", "int": "i64", "nulls": 0.02, "filter": "one",
         "inputs": "host", "output": "host"},
        # an ordinary fact table: nullable keys, 32-bit values, no filter, an odd row count
        {"name": "group 10m ragged", "kind": "group", "rows": 9_999_991, "groups": 200_000, "zipf": 0.7,
         "key": "i64", "key_nulls": 0.02, "float": "f32", "int": "i32", "nulls": 0.05, "filter": "none",
         "inputs": "device", "output": "device"},
        # the headline workload: 100M rows, Zipf(1.1) keys over 1M values, two-part filter
        {"name": "group 100m", "kind": "group", "rows": 100_000_000, "groups": 1_000_000, "zipf": 1.1,
         "key": "i32", "key_nulls": 0.0, "float": "f64", "int": "i64", "nulls": 0.05, "filter": "two",
         "inputs": "device", "output": "device"},
        # a few groups over many rows, sums of products (the reference's benchmark has it at 10M rows)
        {"name": "q1 10m", "kind": "q1", "rows": 10_000_000, "float": "f64", "output": "host"},
        # composite keys of medium and of the benchmark's high cardinality (200M rows, 49M groups)
        {"name": "pair 12m", "kind": "pair", "rows": 12_345_678, "pool": 60_000, "output": "device"},
        {"name": "pair 200m", "kind": "pair", "rows": 200_000_000, "pool": 781_250, "output": "device"},
        # a top-level filter of narrow and nullable columns, and of the headline table
        {"name": "filter 4m mixed", "kind": "filter", "rows": 4_000_037, "table": "mixed", "keep": 0.2,
         "nulls": 0.1, "output": "device"},
        {"name": "filter 100m", "kind": "filter", "rows": 100_000_000, "table": "wide", "keep": 0.63,
         "nulls": 0.05, "output": "device"},
        # a whole table ordered by a float column with nulls, ties broken by an integer column
        {"name": "order 20m", "kind": "order", "rows": 20_000_000, "by": "float,int", "float": "f64",
         "descending": True, "nulls": 0.03, "limit": 0, "output": "device"},
        # independent queries of uneven sizes and skews in one call
        {"name": "batch 32", "kind": "batch", "queries": 32, "rows": 32_000_000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["group", "group", "group", "pair", "q1", "filter", "order", "batch"])
    if kind == "group":
        rows = _log(rng, 10_000, 60_000_000)
        where = "host" if rows < 4_000_000 and rng.random() < 0.25 else "device"
        return {"kind": kind, "rows": rows, "groups": _log(rng, 10, max(11, min(2_000_000, rows // 8))),
                "zipf": rng.choice([0.0, round(rng.uniform(0.2, 1.3), 2)]), "key": rng.choice(["i32", "i64"]),
                "key_nulls": rng.choice([0.0, 0.0, 0.02]), "float": rng.choice(["f64", "f32"]),
                "int": rng.choice(["i64", "i32"]), "nulls": rng.choice([0.0, round(rng.uniform(0.01, 0.2), 2)]),
                "filter": rng.choice(["none", "one", "two"]), "inputs": where,
                "output": "host" if rows < 5_000_000 else "device"}
    if kind == "pair":
        rows = _log(rng, 300_000, 60_000_000)
        return {"kind": kind, "rows": rows, "pool": _log(rng, 300, max(301, rows // 200)), "output": "device"}
    if kind == "q1":
        return {"kind": kind, "rows": _log(rng, 100_000, 60_000_000), "float": rng.choice(["f64", "f32"]),
                "output": "host"}
    if kind == "filter":
        return {"kind": kind, "rows": _log(rng, 50_000, 80_000_000), "table": rng.choice(["mixed", "wide"]),
                "keep": round(rng.uniform(0.02, 0.95), 2), "nulls": rng.choice([0.0, 0.1]), "output": "device"}
    if kind == "order":
        rows = _log(rng, 20_000, 30_000_000)
        return {"kind": kind, "rows": rows, "by": rng.choice(["float", "int", "float,int", "int,float"]),
                "float": rng.choice(["f64", "f32"]), "descending": rng.random() < 0.5,
                "nulls": rng.choice([0.0, 0.03]), "limit": rng.choice([0, 0, 100]), "output": "device"}
    return {"kind": kind, "queries": rng.randint(8, 32), "rows": _log(rng, 1_000_000, 32_000_000)}


# ------------------------------------------------------------------------------- inputs
def _col(name):
    return {"kind": "Column", "name": name}


def _cmp(op, name, kind, value):
    return {"kind": "Compare", "op": op, "lhs": _col(name), "rhs": {"kind": kind, "value": value}}


GROUP_FILTERS = {"none": None, "one": datagen.PRED_SMALL, "two": datagen.PRED_HASH}
GROUP_AGGS = [("Sum", "v1", "v1_sum"), ("Mean", "v1", "v1_mean"), ("Min", "v2", "v2_min"), ("Max", "v2", "v2_max"),
              ("Sum", "v3", "v3_sum"), ("Max", "v3", "v3_max"), ("Len", None, "count")]
Q1_DAY = 2300  # of 2557 days
PRICE_CUT = {"kind": "Binary", "op": "Mul", "lhs": _col("price"),
             "rhs": {"kind": "Binary", "op": "Sub", "lhs": {"kind": "LiteralF64", "value": 1.0}, "rhs": _col("disc")}}
Q1_AGGS = [("Sum", "qty", "qty_sum"), ("Sum", "price", "price_sum"), ("Sum", PRICE_CUT, "cut_sum"),
           ("Mean", "qty", "qty_mean"), ("Mean", "disc", "disc_mean"), ("Len", None, "count")]


def _spread(rows, count, phase):
    """`count` of the positions `rows`, evenly spread, from a random phase on."""
    step = rows.numel() // count
    return rows[torch.arange(count, device=DEV) * step + phase % step]


def _rand_int(g, hi):
    return int(torch.randint(0, hi, (1,), generator=g, device=DEV))


def _keys(n, groups, zipf, g, dtype, where=None):
    """Keys 0 .. groups-1, every one of them among the rows `where` (a mask; all rows without it), so
    that the number of groups does not hang on the seed."""
    if zipf > 0:
        key = datagen.zipf_keys(n, groups, zipf, g, DEV, dtype)
    else:
        key = torch.randint(0, groups, (n,), generator=g, device=DEV, dtype=dtype)
    rows = torch.arange(n, device=DEV) if where is None else torch.nonzero(where).flatten()
    key[_spread(rows, groups, _rand_int(g, 1 << 30))] = torch.randperm(groups, generator=g, device=DEV).to(dtype)
    return key


def _table(case, seed):
    """The case's input columns: name -> (values, bool validity or None, dtype tag), on the GPU."""
    g = datagen._gen(seed, DEV)
    n, kind = case["rows"], case["kind"]

    def rand():
        return torch.rand(n, generator=g, device=DEV)

    def randn(dtype):
        return torch.randn(n, generator=g, device=DEV, dtype=dtype)

    def valid(frac):
        return None if frac <= 0 else rand() >= frac

    def ints(lo, hi, dtype):
        return torch.randint(lo, hi, (n,), generator=g, device=DEV, dtype=dtype)

    if kind == "group":
        f, i = FLOATS[case["float"]], INTS[case["int"]]
        cols = {"v1": (randn(f), valid(case["nulls"]), None), "v2": (randn(f), valid(case["nulls"]), None),
                "v3": (ints(0, 1_000_000_000 if i is torch.int64 else 1_000, i), valid(case["nulls"]), None)}
        key_ok = valid(case["key_nulls"])
        keep = None if GROUP_FILTERS[case["filter"]] is None else _exact_keep(GROUP_FILTERS[case["filter"]], cols)
        if key_ok is not None:
            keep = key_ok if keep is None else keep & key_ok
        return {"key": (_keys(n, case["groups"], case["zipf"], g, INTS[case["key"]], keep), key_ok, None), **cols}
    if kind == "pair":
        # `pool` distinct values in [0, 2^40) times 64
        step = (1 << 40) // case["pool"]
        values = torch.arange(case["pool"], device=DEV) * step
        values += torch.randint(0, step, (case["pool"],), generator=g, device=DEV)
        pair = _keys(n, case["pool"] * 64, 0.0, g, torch.int64)
        return {"k1": (values[pair >> 6], None, None), "k2": ((pair & 63).to(torch.int32), None, None),
                "v": (rand(), None, None), "vi": (ints(-(1 << 40), 1 << 40, torch.int64), None, None)}
    if kind == "q1":
        f = FLOATS[case["float"]]
        price = (rand() * 104_000 + 900).to(f)
        return {"flag": (rand() < 0.5, None, A.BOOL), "status": (rand() < 0.5, None, A.BOOL),
                "qty": (ints(1, 51, torch.int64), None, None), "price": (price, None, None),
                "disc": (ints(0, 11, torch.int32).to(f) / 100, None, None), "day": (ints(0, 2557, torch.int32), None, None)}
    if kind == "filter" and case["table"] == "wide":
        cols = {"key": (datagen.zipf_keys(n, 1_000_000, 1.1, g, DEV, torch.int32), None, None),
                "v1": (randn(torch.float64), valid(case["nulls"]), None),
                "v2": (randn(torch.float64), valid(case["nulls"]), None),
                "v3": (ints(0, 1_000_000_000, torch.int64), valid(case["nulls"]), None)}
        # a few rows too many pass the filter: those fail it after all, so that every seed keeps as many
        t, kept = _wide_filter(case)
        rows = torch.nonzero(_exact_keep(_filter_predicate(case), cols)).flatten()
        if rows.numel() > kept:
            cols["v1"][0][_spread(rows, rows.numel() - kept, _rand_int(g, 1 << 30))] = t - 1.0
        return cols
    if kind == "filter":
        # (u < keep) or (small == 7) for a fixed number of rows, whatever the seed
        keep = torch.zeros(n, dtype=torch.bool, device=DEV)
        keep[torch.randperm(n, generator=g, device=DEV)[: max(1, int(n * case["keep"]))]] = True
        small = ints(-100, 100, torch.int8)
        small = torch.where(~keep & (small == 7), small + 1, small)
        small_ok = valid(case["nulls"])
        by_small = (small == 7) if small_ok is None else (small == 7) & small_ok
        u = torch.where(keep & ~by_small, rand() * case["keep"] * 0.999, case["keep"] + 0.001 + rand())
        u_ok = None if case["nulls"] <= 0 else valid(case["nulls"]) | (keep & ~by_small)
        return {"u": (u, u_ok, None), "flag": (rand() < 0.5, None, A.BOOL), "small": (small, small_ok, None),
                "short": (ints(-30_000, 30_000, torch.int16), None, None),
                "id": (ints(0, 1 << 40, torch.int64), None, None),
                "x": (randn(torch.float64), valid(case["nulls"]), None)}
    if kind == "order":
        # the float column has many ties, as measurements of limited resolution do
        val = (randn(FLOATS[case["float"]]) * 1000).round() / 1000
        return {"float": (val, valid(case["nulls"]), None), "int": (ints(-50_000, 50_000, torch.int32), None, None),
                "id": (torch.arange(n, device=DEV), None, None), "x": (rand(), valid(case["nulls"]), None)}
    raise ValueError(kind)


def _wide_filter(case):
    """Threshold on v1 of the wide table's filter, and the rows that pass it."""
    n, ok = case["rows"], (1 - case["nulls"]) ** 2 * 6 / 7
    p = max(0.01, min(0.99, case["keep"] / ok))
    t = round(-math.sqrt(2) * float(torch.erfinv(torch.tensor(2 * p - 1, dtype=torch.float64))), 3)
    p = ok * 0.5 * math.erfc(t / math.sqrt(2))
    return t, max(1, int(n * p - 6 * math.sqrt(n)))


def _filter_predicate(case):
    if case["table"] == "mixed":
        return {"kind": "Or", "lhs": _cmp("Lt", "u", "LiteralF64", case["keep"]),
                "rhs": _cmp("Eq", "small", "LiteralI64", 7)}
    return {"kind": "And", "lhs": _cmp("Gt", "v1", "LiteralF64", _wide_filter(case)[0]), "rhs": datagen.PRED_HASH["rhs"]}


def _batch(case, seed):
    """Queries of the batched benchmark's distribution: uneven rows, cardinalities and skews. The
    shapes belong to the case, the values to the seed. Per query (key, values, validity)."""
    rows, card, zipf = datagen.batch_sizes(case["queries"], case["rows"] + case["queries"])
    rows = np.maximum(1000, (rows * (case["rows"] / rows.sum())).astype(np.int64))
    card = np.maximum(1, np.minimum(card, rows // 2))
    g = datagen._gen(seed, DEV)
    out = []
    for n, k, s in zip(rows.tolist(), card.tolist(), zipf.tolist()):
        v = torch.randn(n, generator=g, device=DEV, dtype=torch.float64)
        ok = torch.rand(n, generator=g, device=DEV) >= 0.01
        out.append((_keys(n, k, s, g, torch.int32, ok & (v > -1.0)), v, ok))
    return out


def prepare(case, seed):
    if case["kind"] == "batch":
        queries = [({"key": ColumnData(k), "v": ColumnData(v, datagen.pack_bits(ok))}, ["key"], datagen.AGGS_BATCH,
                    datagen.PRED_BATCH) for k, v, ok in _batch(case, seed)]
        torch.cuda.synchronize()
        return {"case": case, "queries": prepare_batched(queries, output="device")}
    cols = {}
    for name, (data, valid, dtype) in _table(case, seed).items():
        n = data.numel()
        data = datagen.pack_bits(data) if dtype == A.BOOL else data
        valid = None if valid is None else datagen.pack_bits(valid)
        if case.get("inputs") == "host":
            data, valid = data.cpu().numpy(), None if valid is None else valid.cpu().numpy()
        cols[name] = ColumnData(data, valid, dtype=dtype, length=n)
    torch.cuda.synchronize()  # the library's stream does not wait for torch's
    return {"case": case, "cols": cols}


# ------------------------------------------------------------------------------- one pass
class _Device:
    """A device buffer of a result, for torch.as_tensor."""

    def __init__(self, addr, n, typestr):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (addr, False), "version": 3}


TYPES = {A.BOOL: "|u1", A.I8: "|i1", A.I16: "<i2", A.I32: "<i4", A.I64: "<i8", A.U8: "|u1", A.U32: "<i4", A.F32: "<f4",
         A.F64: "<f8"}


def _tensor(addr, n, typestr):
    return torch.as_tensor(_Device(addr, n, typestr), device=DEV) if n else torch.empty(0, device=DEV)


def _outputs(res, output):
    n, nb = res.n_groups, (res.n_groups + 7) // 8
    out = {"rows": n}
    for name, dt, data, valid in zip(res.names, res.dtypes, res.data, res.validity):
        if output == "device":
            data = _tensor(data, nb if dt == A.BOOL else n, TYPES[dt])
            valid = _tensor(valid, nb, "|u1")
        elif dt == A.U32:
            data = data.view(np.int32)
        out[name] = {"data": data, "valid": valid}
    return out


def run(state):
    case = state["case"]
    kind, output = case["kind"], case.get("output")
    if kind == "group":
        res = groupby(state["cols"], ["key"], GROUP_AGGS, GROUP_FILTERS[case["filter"]], output=output,
                      sort={"by": "key"})
    elif kind == "pair":
        res = groupby(state["cols"], ["k1", "k2"], PAIR_AGGS, output=output, sort={"by": ["k1", "k2"]})
    elif kind == "q1":
        res = groupby(state["cols"], ["flag", "status"], Q1_AGGS, _cmp("Le", "day", "LiteralI64", Q1_DAY),
                      output=output, sort={"by": ["flag", "status"]})
    elif kind == "filter":
        res = filter_columns(state["cols"], _filter_predicate(case), output=output)
    elif kind == "order":
        res = sort_columns(state["cols"], case["by"].split(","), descending=case["descending"], nulls_last=True,
                           limit=case["limit"] or None, output=output)
    else:
        return _run_batch(state)
    return _outputs(res, output)


PAIR_AGGS = [("Sum", "v", "v_sum"), ("Min", "v", "v_min"), ("Max", "v", "v_max"), ("Sum", "vi", "vi_sum"),
             ("Min", "vi", "vi_min"), ("Max", "vi", "vi_max"), ("Len", None, "count")]


def _run_batch(state):
    results = groupby_batched(state["queries"])
    # the report: one table of all queries' groups (the buffers are free again after the copies)
    parts = [results[i] for i in range(len(results))]
    counts = torch.tensor([r.n_groups for r in parts])
    cols = {"query": ColumnData(torch.repeat_interleave(torch.arange(len(parts), dtype=torch.int32), counts).to(DEV))}
    for c, name in enumerate(parts[0].names):
        dt = parts[0].dtypes[c]
        # every aggregate is of a column with some valid row per kept group: no nulls to carry over
        cols[name] = ColumnData(torch.cat([_tensor(r.data[c], r.n_groups, TYPES[dt]) for r in parts]))
    torch.cuda.current_stream().synchronize()
    return _outputs(sort_columns(cols, ["query", "key"], output="device"), "device")


# ------------------------------------------------------------------------------- needed work
def work(case):
    n, kind = case["rows"], case["kind"]
    sizes = {"i64": 8, "i32": 4, "f64": 8, "f32": 4}
    if kind == "group":
        f, i, k = sizes[case["float"]], sizes[case["int"]], sizes[case["key"]]
        per_row = k + 2 * f + i + (3 / 8 if case["nulls"] else 0) + (1 / 8 if case["key_nulls"] else 0)
        return {"bytes": n * per_row + case["groups"] * (k + 4 * f + 2 * i + 4 + 1), "flops": 6.0 * n}
    if kind == "pair":
        return {"bytes": n * 24.0 + case["pool"] * 64.0 * (12 + 12 + 24 + 4 + 9 / 8), "flops": 6.0 * n}
    if kind == "q1":
        return {"bytes": n * (2 / 8 + 8 + 2 * sizes[case["float"]] + 4), "flops": 8.0 * n}
    if kind == "filter":
        row = 28 + (3 / 8 if case["nulls"] else 0)
        if case["table"] == "mixed":
            row = 4 + 1 / 8 + 1 + 2 + 8 + 8 + (3 / 8 if case["nulls"] else 0)
        return {"bytes": n * row * (1 + case["keep"]), "flops": 2.0 * n}
    if kind == "order":
        row = sizes[case["float"]] + 4 + 8 + 4 + (2 / 8 if case["nulls"] else 0)
        by = sum(sizes[case["float"]] if b == "float" else 4 for b in case["by"].split(","))
        out = row * n if not case["limit"] else row * case["limit"]
        return {"bytes": (row if not case["limit"] else by) * n + out, "flops": 1.0 * n}
    return {"bytes": n * 12.125, "flops": 4.0 * n}


# ------------------------------------------------------------------------------- 64-bit results
def exact(case, seed):
    """The floating outputs of run() in 64 bits, as plain torch gives them; None for the others."""
    kind = case["kind"]
    if kind == "batch":
        return _exact_batch(case, seed)
    cols = {k: (d, v) for k, (d, v, _) in _table(case, seed).items()}
    if kind == "filter":
        keep = _exact_keep(_filter_predicate(case), cols)
        return _exact_rows(cols, torch.nonzero(keep).flatten())
    if kind == "order":
        n = case["rows"]
        perm = torch.arange(n, device=DEV)
        for name in reversed(case["by"].split(",")):
            d, v = cols[name]
            d = d if v is None else torch.where(v, d, torch.zeros_like(d))
            perm = perm[torch.sort(d[perm], stable=True, descending=case["descending"]).indices]
            if v is not None:
                perm = perm[torch.sort((~v[perm]).to(torch.uint8), stable=True).indices]
        return _exact_rows(cols, perm[: case["limit"] or n])
    if kind == "group":
        return _exact_group(cols, ["key"], GROUP_AGGS, GROUP_FILTERS[case["filter"]])
    if kind == "pair":
        return _exact_group(cols, ["k1", "k2"], PAIR_AGGS, None)
    cut = cols["price"][0].double() * (1.0 - cols["disc"][0].double())
    cols["cut"] = (cut, None)
    aggs = [(op, "cut" if isinstance(c, dict) else c, alias) for op, c, alias in Q1_AGGS]
    return _exact_group(cols, ["flag", "status"], aggs, _cmp("Le", "day", "LiteralI64", Q1_DAY))


def _exact_rows(cols, rows):
    return {k: {"data": d[rows].double() if d.is_floating_point() else None, "valid": None} for k, (d, _) in cols.items()}


def _exact_keep(p, cols):
    """Rows whose predicate is valid and true (the filters here: And / Or of compares)."""
    if p["kind"] in ("And", "Or"):
        a, b = _exact_keep(p["lhs"], cols), _exact_keep(p["rhs"], cols)
        return a & b if p["kind"] == "And" else a | b
    lhs = p["lhs"]
    d, v = cols[lhs["lhs"]["name"] if lhs["kind"] == "Arith" else lhs["name"]][:2]
    if lhs["kind"] == "Arith":
        d = torch.remainder(d, lhs["rhs"]["value"])
    if d.is_floating_point():
        d = d.double()
    op = {"Gt": torch.gt, "Lt": torch.lt, "Le": torch.le, "Eq": torch.eq, "Ne": torch.ne}[p["op"]]
    t = op(d, p["rhs"]["value"])
    return t if v is None else t & v


def _exact_sum(x, inv, groups):
    """Sums of x by group, from exact 64-bit integer sums of two limbs of every value."""
    top = float(x.abs().max()) if x.numel() else 0.0
    e = 34 - (math.frexp(top)[1] if top else 0)
    hi = torch.round(torch.ldexp(x, torch.tensor(e, device=x.device)))
    lo = torch.round(torch.ldexp(torch.ldexp(x, torch.tensor(e, device=x.device)) - hi, torch.tensor(34, device=x.device)))
    parts = []
    for limb in (hi, lo):
        s = torch.zeros(groups, dtype=torch.int64, device=x.device)
        parts.append(s.index_add_(0, inv, limb.to(torch.int64)).double())
        del limb
    return torch.ldexp(parts[0] + torch.ldexp(parts[1], torch.tensor(-34, device=x.device)), torch.tensor(-e, device=x.device))


def _exact_group(cols, keys, aggs, predicate):
    if predicate is not None:
        keep = _exact_keep(predicate, cols)
        cols = {k: (d[keep], None if v is None else v[keep]) for k, (d, v) in cols.items()}
    code = None
    for k in keys:  # dense codes in key order, nulls first
        d, v = cols[k]
        u, inv = torch.unique(d.to(torch.int64), return_inverse=True)
        inv = inv + 1 if v is None else torch.where(v, inv + 1, torch.zeros_like(inv))
        code = inv if code is None else code * (u.numel() + 1) + inv
    u, inv = torch.unique(code, return_inverse=True)
    groups = u.numel()
    out = {k: {"data": None, "valid": None} for k in keys}
    for op, c, alias in aggs:
        x = None
        if c is not None and (op == "Mean" or cols[c][0].is_floating_point()):
            d, v = cols[c]
            at = inv if v is None else inv[v]
            d = (d if v is None else d[v]).double()
            count = torch.bincount(at, minlength=groups).double()
            if op in ("Sum", "Mean"):
                x = _exact_sum(d, at, groups)
                if op == "Mean":
                    x = torch.where(count > 0, x / count.clamp(min=1), torch.zeros_like(x))
            else:
                x = torch.full((groups,), math.inf if op == "Min" else -math.inf, dtype=torch.float64, device=DEV)
                x = x.scatter_reduce_(0, at, d, "amin" if op == "Min" else "amax")
                x = torch.where(count > 0, x, torch.zeros_like(x))
        out[alias] = {"data": x, "valid": None}
    return out


def _exact_batch(case, seed):
    parts = []
    for k, v, ok in _batch(case, seed):
        parts.append(_exact_group({"key": (k, None), "v": (v, ok)}, ["key"], datagen.AGGS_BATCH, datagen.PRED_BATCH))
    out = {"query": {"data": None, "valid": None}, "key": {"data": None, "valid": None}}
    for _, _, alias in datagen.AGGS_BATCH:
        x = parts[0][alias]["data"]
        out[alias] = {"data": None if x is None else torch.cat([p[alias]["data"] for p in parts]), "valid": None}
    return out
