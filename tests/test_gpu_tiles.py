"""GPU parity at the sizes where a kernel's tiling can go wrong: tile edges, remainders, the smallest
and largest sizes of a dispatch range. Integer results and orders are compared bit for bit with the
oracle's; float sums as in tests/helpers.py."""

import numpy as np
import pytest

from helpers import as_dict, assert_results_match, pack
from oracle import pyoracle
from polars_b200 import _abi as A
from polars_b200 import _native as N
from test_gpu_sort import assert_same_rows

pytestmark = pytest.mark.gpu


def _sorted_both(cols: dict, by, descending, nulls_last=False, **kw):
    """(product, oracle) of the sort of columns given as name -> (values, bitmap or None)."""
    got = N.sort_columns({k: N.ColumnData(d, v) for k, (d, v) in cols.items()}, by, descending, nulls_last, **kw)
    nl = [nulls_last] * len(by)
    want = pyoracle.sort_table(cols, by, descending, nl, kw.get("drop_nulls", False), kw.get("offset", 0),
                               -1 if kw.get("limit") is None else kw["limit"])
    return as_dict(got), want


# the radix passes: tiles of 3840 keys of one word and of 3072 keys of two words; skewed digits (many
# lanes of a warp share one) and constant ones (a skipped pass)
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("n", [11519, 11520, 11521, 12287, 12288, 12289, 46080])
def test_radix_pass_tiles(n, wide):
    rng = np.random.default_rng(n)
    cols = {"a": (rng.integers(0, 3, n) * (1 << 33) + rng.integers(0, 700, n), pack(rng.random(n) > 0.1)),
            "b": (rng.integers(-2**62, 2**62, n), None), "row": (np.arange(n, dtype=np.int32), None)}
    by = ["a", "b"] if wide else ["a"]
    got, want = _sorted_both(cols, by, [True, False][: len(by)])
    assert_same_rows(got, want, f"{n} rows")


# the one-launch sort of small tables: padding to a power of two (at least 64), its largest size and
# the general path's smallest, one- and two-word keys, dropped nulls, slices
@pytest.mark.parametrize("spec", [(["a"], [False], {}), (["b", "a"], [True, False], {"nulls_last": True}),
                                  (["a"], [True], {"drop_nulls": True, "nulls_last": True, "limit": 7}),
                                  (["f", "s"], [False, True], {"offset": -20, "limit": 15})], ids=lambda s: "-".join(s[0]))
@pytest.mark.parametrize("n", [2, 33, 64, 65, 1000, 4096, 8191, 8192, 8193])
def test_small_sort(n, spec):
    by, desc, kw = spec
    rng = np.random.default_rng(n)
    f = rng.standard_normal(n).astype(np.float32)
    f[rng.random(n) < 0.2] = np.float32(-0.0)
    f[rng.random(n) < 0.1] = np.float32("nan")
    cols = {"a": (rng.integers(-40, 40, n), pack(rng.random(n) > 0.2)), "f": (f, None),
            "b": (rng.integers(-2**31, 2**31, n).astype(np.int32), pack(rng.random(n) > 0.1)),
            "s": (rng.integers(-128, 128, n).astype(np.int8), None), "row": (np.arange(n), None)}
    got, want = _sorted_both(cols, by, desc, **kw)
    assert_same_rows(got, want, f"{n} rows by {by}")


# host results: in one copy up to 4 MB of span (whole and partial bitmap bytes), a copy per buffer above
@pytest.mark.parametrize("n", [1, 31, 32, 33, 4099, 170_000, 180_000, 400_003])
def test_host_results(n):
    rng = np.random.default_rng(n)
    x, y = rng.standard_normal(n), rng.integers(-100, 100, n).astype(np.int8)
    z, ok = rng.integers(0, 2**60, n), rng.random(n) > 0.3
    keep = x > -3.0
    got = N.filter_columns({"x": x, "y": y, "z": N.ColumnData(z, pack(ok))},
                           {"kind": "Compare", "op": "Gt", "lhs": {"kind": "Column", "name": "x"},
                            "rhs": {"kind": "LiteralF64", "value": -3.0}})
    m = int(keep.sum())
    assert got.n_groups == m
    for have, want in zip(got.data, (x, y, z)):
        assert np.array_equal(have[:m], want[keep])
    assert np.array_equal(np.unpackbits(got.validity[2], bitorder="little")[:m].astype(bool), ok[keep])
    assert np.unpackbits(got.validity[0], bitorder="little")[:m].all() if m else True


# keys wider than 64 bits by their types whose values fit 64: nullable Int64 alone, column pairs, the
# extremes of the types, a span of exactly 64 bits and one of 65 (which stays on the 128-bit path)
@pytest.mark.parametrize("n", [1, 3000, 2_200_000])
@pytest.mark.parametrize("case", ["nullable", "all null", "pair", "negative", "span64", "span65", "floats"])
def test_wide_keys(case, n):
    rng = np.random.default_rng(len(case) + n)
    g = rng.integers(0, 300, n)
    ok = pack(rng.random(n) > 0.1)
    big = np.where(g % 2 == 0, np.int64(-2**63), np.int64(2**63 - 1))
    keys = {
        "nullable": {"k": (g * 7_000_000_000 - 900, ok)},
        "all null": {"k": (g, pack(np.zeros(n, bool)))},
        "pair": {"k": (g - (1 << 40), None), "j": (rng.integers(-5, 5, n).astype(np.int32), ok)},
        "negative": {"k": (-(g << 33), ok), "j": ((g % 3 - 128).astype(np.int8), None), "b": (pack(g % 5 == 0), None, A.BOOL, n)},
        "span64": {"k": (big, None), "j": (np.full(n, 9, np.int16), None)},
        "span65": {"k": (big, None), "j": ((g % 2).astype(np.int16), None)},
        "floats": {"k": ((g % 50) * 0.25 - 3.0, ok), "j": ((g % 4).astype(np.float32) - 1.5, None)},
    }[case]
    v = rng.standard_normal(n)
    cols = {**keys, "v": (v, pack(rng.random(n) > 0.05))}
    aggs = [("Sum", "v", "s"), ("Max", "v", "m"), ("Len", None, "c")]
    inv = {d: k for k, d in A.NUMPY_NAME.items()}
    data = {k: N.ColumnData(c[0], c[1], dtype=c[2], length=c[3]) if len(c) > 2 else N.ColumnData(c[0], c[1])
            for k, c in cols.items()}
    full = {k: c if len(c) > 2 else (c[0], c[1], inv[c[0].dtype.name], n) for k, c in cols.items()}
    want = pyoracle.groupby(full, list(keys), aggs, None)
    for strategy in ("auto", "global_hash"):
        got = N.groupby(data, list(keys), aggs, strategy=strategy)
        assert_results_match(as_dict(got), want, len(keys), aggs, f"{case} {strategy}")


# the staged compaction (PMB_JIT=1: at every size): stage tiles of 1024 rows, 256 with many columns;
# partial last tiles, more tiles than CTAs, nothing and everything kept, bitmap words shared by tiles
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("n", [1, 31, 255, 256, 257, 1023, 1024, 1025, 5 * 1024 + 3, 1_500_001])
@pytest.mark.parametrize("share", [0.0, 0.4, 1.0])
def test_staged_compaction(n, share, wide, monkeypatch):
    monkeypatch.setenv("PMB_JIT", "1")
    rng = np.random.default_rng(n)
    u, uok = rng.random(n), rng.random(n) > (0.0 if share == 1.0 else 0.1)
    cols = {"u": (u, pack(uok)), "b": (rng.random(n) > 0.5, None), "i8": (rng.integers(-9, 9, n).astype(np.int8), None),
            "i16": (rng.integers(-9, 9, n).astype(np.int16), rng.random(n) > 0.5), "f": (rng.random(n).astype(np.float32), None)}
    if wide:
        cols |= {f"w{i}": (rng.integers(0, 2**60, n), rng.random(n) > 0.2) for i in range(11)}
    data = {k: N.ColumnData(pack(d), None, dtype=A.BOOL, length=n) if d.dtype == bool else
            N.ColumnData(d, v if k == "u" or v is None else pack(v)) for k, (d, v) in cols.items()}
    got = N.filter_columns(data, {"kind": "Compare", "op": "Lt", "lhs": {"kind": "Column", "name": "u"},
                                  "rhs": {"kind": "LiteralF64", "value": share}})
    keep = (u < share) & uok
    m = int(keep.sum())
    assert got.n_groups == m
    for i, (k, (d, v)) in enumerate(cols.items()):
        have = np.unpackbits(got.data[i], bitorder="little")[:m].astype(bool) if d.dtype == bool else got.data[i][:m]
        assert np.array_equal(have, d[keep]), k
        ok = np.unpackbits(got.validity[i], bitorder="little")[:m].astype(bool)
        assert np.array_equal(ok, np.ones(m, bool) if v is None or k == "u" else v[keep]), k


# the selector's network in the sampling launch: the same pick and table size as selector_choose,
# whose features and network run as kernels of their own
@pytest.mark.parametrize("card,width", [(50, 4), (3000, 4), (90_000, 8), (400_000, 8), (1_500_000, 8)])
def test_selector_in_the_sampling_launch(card, width):
    rng = np.random.default_rng(card)
    n = 3_000_000
    k = rng.integers(0, card, n).astype(np.int32 if width == 4 else np.int64)
    v = rng.standard_normal(n)
    q = ({"k": k, "v": v}, ["k"], [("Sum", "v", "s"), ("Len", None, "c")])
    strategy, groups = N.selector_choose(*q)
    got = N.groupby(*q)
    assert got.strategy == strategy and got.n_groups == len(np.unique(k))
    if got.rehash_count == 0 and strategy.endswith("hash"):
        assert min(max(2 * groups, 1024), 2 * n) <= got.capacity <= max(3 * groups, 1024) + 3  # slots per estimated group


# expressions: tails of a thread's four rows and of a bitmap word, flat and deep trees, an output that
# overlaps an input (computed aside, then copied)
@pytest.mark.parametrize("jit", ["0", "1"])  # the interpreter, the run-time compiled kernel
@pytest.mark.parametrize("n", [1, 7, 31, 32, 33, 127, 128, 129, 1025, 100_003])
def test_expression_rows(n, jit, monkeypatch):
    import torch

    monkeypatch.setenv("PMB_JIT", jit)

    rng = np.random.default_rng(n)
    a, b = rng.standard_normal(n), rng.integers(-9, 9, n).astype(np.int32)
    ok = rng.random(n) > 0.3
    A_, B_ = {"kind": "Column", "name": "a"}, {"kind": "Column", "name": "b"}
    flat = {"kind": "Binary", "op": "Mul", "lhs": A_, "rhs": {"kind": "Binary", "op": "Sub", "lhs": B_, "rhs": A_}}
    deep = A_
    for _ in range(6):  # right-nested: seven entries on the stack
        deep = {"kind": "Binary", "op": "Add", "lhs": B_, "rhs": deep}
    want_deep = a.copy()
    for _ in range(6):
        want_deep = b + want_deep
    for e, want in ((flat, a * (b - a)), (deep, want_deep)):
        for dev in (False, True):
            cols = {"a": N.ColumnData(torch.from_numpy(a).cuda() if dev else a,
                                      torch.from_numpy(pack(ok)).cuda() if dev else pack(ok)),
                    "b": N.ColumnData(torch.from_numpy(b).cuda() if dev else b)}
            got = N.eval_expr(cols, e)
            data = got.data.cpu().numpy() if dev else got.data
            valid = got.validity.cpu().numpy() if dev else got.validity
            assert np.array_equal(np.unpackbits(valid, bitorder="little")[:n].astype(bool), ok)
            assert np.array_equal(data[:n][ok], want[ok])


def test_expression_in_place():
    import ctypes as C

    import torch

    n = 5000
    x = torch.randn(n + 1, dtype=torch.float64, device="cuda")
    want = (x[:n] + x[:n]).cpu().numpy()
    cols = {"x": N.ColumnData(x[:n])}
    abi, _keep = N._to_abi_columns(list(cols.values()))
    e, _k = N.compile_predicate({"kind": "Arith", "op": "Add", "lhs": {"kind": "Column", "name": "x"},
                                 "rhs": {"kind": "Column", "name": "x"}}, {"x": 0})
    valid = torch.zeros(N._bitmap_bytes(n), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    h, dt = N.default_handle(), C.c_int32()
    h.check(h._lib.pmb_eval_expr(h.raw, C.byref(e), abi, 1, x[1:].data_ptr(), valid.data_ptr(), 1, C.byref(dt)))
    assert np.array_equal(x[1:].cpu().numpy(), want)


# pageable columns staged by several threads: sizes around the pool's smallest copy and its chunks,
# bitmaps at a bit offset, several columns in a row through the same chunks
@pytest.mark.parametrize("n", [524_287, 524_288, 655_361, 4_000_003])
def test_pageable_columns(n):
    rng = np.random.default_rng(n)
    k, x = rng.integers(0, 5, n + 3), rng.integers(-2**40, 2**40, n + 3)
    ok = rng.random(n + 3) > 0.25
    big = pack(np.tile(ok, 1))
    cols = {"k": N.ColumnData(k, None, offset=3, length=n), "x": N.ColumnData(x, big, offset=3, length=n)}
    got = as_dict(N.groupby(cols, ["k"], [("Sum", "x", "s"), ("Count", "x", "c")], sort={"by": "k"}))
    kk, xx, oo = k[3:], x[3:], ok[3:]
    assert np.array_equal(got["data"][1][:5], [xx[(kk == i) & oo].sum() for i in range(5)])
    assert np.array_equal(got["data"][2][:5], [((kk == i) & oo).sum() for i in range(5)])


# groups left in the wanted order by the partitioned and the sort strategy: directions, null places,
# some of the keys, slices, one- and two-word keys, one group
ORDERS = [({"by": ["j", "k"]}, None), ({"by": ["k"], "descending": True, "offset": 5, "limit": 1000}, None),
          ({"by": ["k", "j"], "descending": [True, False], "nulls_last": [True, False], "offset": -900}, None),
          ({"by": ["j", "k"], "nulls_last": True, "drop_nulls": True, "limit": 50}, None),
          ({"by": ["k", "s"]}, None)]


@pytest.mark.parametrize("strategy", ["partitioned", "sort"])
@pytest.mark.parametrize("order", [o for o, _ in ORDERS], ids=lambda o: "-".join(map(str, o.values())))
@pytest.mark.parametrize("kind", ["narrow", "wide", "one"])
def test_ordered_groups(kind, order, strategy):
    rng = np.random.default_rng(len(kind))
    n = 120_000
    k = rng.integers(0, 3000, n) if kind != "one" else np.full(n, 7)
    k = np.where(k % 2 == 0, k, -k) * (3_000_000_000_000_000 if kind == "wide" else 1)
    j = rng.integers(-20, 20, n).astype(np.int16) if kind != "one" else np.full(n, -3, np.int16)
    w = (rng.integers(0, 2, n) * 2**30 if kind == "wide" else np.zeros(n)).astype(np.int32)
    ok = np.ones(n, bool) if kind == "one" else rng.random(n) > 0.02
    v = rng.standard_normal(n)
    cols = {"k": (k, None), "j": (j, pack(ok)), "w": (w, None), "v": (v, None)}
    data = {name: N.ColumnData(*c) for name, c in cols.items()}
    aggs = [("Min", "v", "s"), ("Len", None, "c")]
    keys = ["k", "j", "w"]
    want = pyoracle.groupby(cols, keys, aggs, None)
    # a total order: the other keys behind the wanted ones settle its ties
    got = as_dict(N.groupby(data, keys, aggs, strategy=strategy, sort=order))
    table = {nm: (d, va, dt, want["n_groups"]) for nm, d, va, dt in zip(want["names"], want["data"], want["validity"],
                                                                       want["dtypes"])}
    by = order["by"]
    flags = lambda x: [bool(x)] * len(by) if isinstance(x, bool) else list(x)  # noqa: E731
    full = pyoracle.sort_table(table, by, flags(order.get("descending", False)), flags(order.get("nulls_last", False)),
                               order.get("drop_nulls", False), order.get("offset", 0),
                               -1 if order.get("limit") is None else order["limit"])
    assert int(got["n_groups"]) == int(full["n_groups"])
    m = int(full["n_groups"])
    for name in by:
        i = keys.index(name) if name in keys else len(keys)
        g_ok = np.unpackbits(np.asarray(got["validity"][i], np.uint8), bitorder="little")[:m].astype(bool)
        f_ok = np.unpackbits(np.asarray(full["validity"][i], np.uint8), bitorder="little")[:m].astype(bool)
        assert np.array_equal(g_ok, f_ok), name
        assert np.array_equal(np.asarray(got["data"][i])[:m][f_ok], np.asarray(full["data"][i])[:m][f_ok]), name
    if not order.get("offset") and order.get("limit") is None:
        assert_results_match(got, want, len(keys), aggs, strategy)


# rows straight into the global table: block edges, one- and two-word keys that do not pack, and the
# rule's other side (a key with too many rows for it)
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("groups", [1, 3, 900])
@pytest.mark.parametrize("n", [1, 255, 256, 257, 30_000])
def test_direct_rows(n, groups, wide):
    rng = np.random.default_rng(n + groups)
    k = rng.integers(0, groups, n)
    cols = {"k": (np.where(k % 2 == 0, k, -k) * (2**52 if wide else 1), pack(rng.random(n) > 0.1)),
            "v": (rng.standard_normal(n).astype(np.float32), pack(rng.random(n) > 0.2)), "x": (rng.integers(-9, 9, n), None)}
    if wide:
        cols["j"] = ((rng.integers(0, 2, n) * (2**31 - 1)).astype(np.int32), None)
    keys = ["k", "j"] if wide else ["k"]
    aggs = [("Sum", "v", "s"), ("Min", "v", "lo"), ("Max", "x", "hi"), ("Count", "v", "c"), ("Len", None, "l")]
    pred = {"kind": "Compare", "op": "Ne", "lhs": {"kind": "Column", "name": "x"}, "rhs": {"kind": "LiteralI64", "value": 3}}
    got = N.groupby({c: N.ColumnData(*d) for c, d in cols.items()}, keys, aggs, pred)
    assert_results_match(as_dict(got), pyoracle.groupby(cols, keys, aggs, pred), len(keys), aggs)


# values carried through the partition passes (64 MB of them and more): every width, nulls, Bool values,
# a filter (row numbers with gaps), one and two passes, one- and two-word keys, a row too wide for it
@pytest.mark.parametrize("groups", [20_000, 900_000])
@pytest.mark.parametrize("case", ["narrow", "nulls", "filter", "wide key", "too wide"])
def test_carried_values(case, groups):
    rng = np.random.default_rng(groups)
    n = 5_000_011 if case == "narrow" else 3_400_003
    k = rng.integers(0, groups, n)
    cols = {"k": (k * (2**40 if case == "wide key" else 1), None), "a": (rng.integers(-100, 100, n).astype(np.int8), None),
            "c": (rng.integers(-9, 9, n), None), "f": (rng.standard_normal(n).astype(np.float32), None)}
    aggs = [("Sum", "a", "a_s"), ("Min", "f", "f_lo"), ("Sum", "f", "f_s"), ("Max", "c", "c_hi"), ("Len", None, "n")]
    keys, pred = ["k"], None
    if case != "narrow":
        cols["f"] = (cols["f"][0], pack(rng.random(n) > 0.2))
        cols["u"] = (rng.integers(0, 60_000, n).astype(np.uint16), pack(rng.random(n) > 0.5))
        aggs += [("Mean", "u", "u_m"), ("Count", "u", "u_c")]
    if case == "filter":
        pred = {"kind": "Compare", "op": "Gt", "lhs": {"kind": "Column", "name": "c"}, "rhs": {"kind": "LiteralI64", "value": -6}}
        cols["b"] = (pack(rng.random(n) > 0.5), pack(rng.random(n) > 0.1), A.BOOL, n)
        aggs += [("Sum", "b", "b_s")]
    if case == "wide key":
        cols["j"] = ((k % 7 * 2**28).astype(np.int32), None)
        keys.append("j")
    if case == "too wide":
        for i in range(3):
            cols[f"x{i}"] = (rng.integers(-2**40, 2**40, n), None)
            aggs.append(("Min", f"x{i}", f"x{i}_lo"))
    inv = {d: t for t, d in A.NUMPY_NAME.items()}
    full = {c: d if len(d) > 2 else (d[0], d[1], inv[d[0].dtype.name], n) for c, d in cols.items()}
    data = {c: N.ColumnData(d, v, dtype=t, length=m) for c, (d, v, t, m) in full.items()}
    got = N.groupby(data, keys, aggs, pred, strategy="partitioned")
    assert got.strategy == "partitioned"
    assert_results_match(as_dict(got), pyoracle.groupby(full, keys, aggs, pred), len(keys), aggs, case)


# sort columns by rank among few distinct values: one value, the most that the set takes and one more,
# special floats (whose bits come from their rows) and none, the all-ones order key (which stays whole),
# both directions and null places, slices, several rounds
@pytest.mark.parametrize("case", [("f64", 1, False, {}), ("f64", 5000, False, {}), ("clean", 700, True, {}),
                                  ("clean", 12288, True, {"nulls_last": True}), ("max", 40, True, {}),
                                  ("f64", 12289, False, {"offset": 1_000_000, "limit": 70_001}),
                                  ("i64", 300, True, {"drop_nulls": True, "nulls_last": True, "limit": 100}),
                                  ("i64", 9000, False, {"nulls_last": True}), ("rounds", 1000, False, {}),
                                  ("f32", 200, True, {}), ("clean32", 3000, False, {"nulls_last": True})],
                         ids=lambda c: f"{c[0]}-{c[1]}")
def test_ranked_sort_columns(case):
    kind, distinct, desc, kw = case
    n, rng = 12_000_001 if "32" in kind else 4_200_001, np.random.default_rng(case[1])
    if kind in ("f64", "clean", "f32", "clean32"):
        span = 36 if "32" in kind else 300
        values = rng.standard_normal(distinct) * 10.0 ** rng.integers(-span, span, distinct)
        if "32" in kind:
            values = values.astype(np.float32)
        if kind[0] == "f":  # and values whose bits are not their order key's
            values[: min(4, distinct - 1)] = [np.inf, -np.inf, np.nan, -0.0][: min(4, distinct - 1)]
    else:
        values = rng.integers(-2**63, 2**63 - 1, distinct)
        values[0] = 2**63 - 1 if kind == "max" else -2**63
    pick = rng.integers(0, max(1, distinct // 4), n)  # most rows have few of them, so that a sample promises few
    pick[:distinct] = np.arange(distinct)
    cols = {"v": (values[rng.permutation(pick)], pack(rng.random(n) > 0.05)),
            "i": (rng.integers(-50_000, 50_000, n).astype(np.int32), None), "row": (np.arange(n, dtype=np.int32), None)}
    by = ["v", "i"]
    if kind == "rounds":  # more than 128 key bits: the ranks in the last round, over rows already in an order
        cols["j"] = (rng.integers(-2**63, 2**63 - 1, n) >> rng.integers(0, 2, n) * 62, None)
        cols["w"] = (cols["j"][0][::-1].copy(), None)
        by = ["v", "j", "w", "i"]
    got, want = _sorted_both(cols, by, [desc, not desc, desc, desc][: len(by)], **kw)
    assert_same_rows(got, want, f"{distinct} {kind}")


# work items of the partitioned aggregation: a fraction of a row, and just below two and three rows, in each of
# 65,536 partitions (by the hint's estimate), every row a group of its own: half a table an item, so that the
# strategy holds; with a filter that leaves few of many rows, the values are carried
@pytest.mark.parametrize("filtered", [False, True])
@pytest.mark.parametrize("jit", ["0", "1"])
@pytest.mark.parametrize("kept", [20_000, 65_535, 130_900, 196_400])
def test_partition_runs(kept, jit, filtered, monkeypatch):
    monkeypatch.setenv("PMB_JIT", jit)
    n = 2_900_017 if filtered else kept
    rng = np.random.default_rng(kept)
    k = rng.permutation(n)
    cols = {"k": (k * 8191, None), "f": (k.astype(np.int32), None), "x": (rng.integers(-2**40, 2**40, n), None),
            "y": (rng.integers(-2**40, 2**40, n), None), "z": (rng.integers(-2**40, 2**40, n), None)}
    pred = {"kind": "Compare", "op": "Lt", "lhs": {"kind": "Column", "name": "f"}, "rhs": {"kind": "LiteralI64", "value": kept}}
    aggs = [("Max", "x", "s"), ("Min", "y", "l"), ("Max", "z", "h")]
    got = N.groupby({c: N.ColumnData(*d) for c, d in cols.items()}, ["k"], aggs, pred if filtered else None,
                    strategy="partitioned", capacity_hint=400_000)
    assert got.strategy == "partitioned" and got.n_groups == kept
    assert_results_match(as_dict(got), pyoracle.groupby(cols, ["k"], aggs, pred if filtered else None), 1, aggs)


def _table(want):
    return {nm: (d, v, dt, want["n_groups"]) for nm, d, v, dt in zip(want["names"], want["data"], want["validity"], want["dtypes"])}


# slices of groups left in the wanted order, by all keys, so that order and slice are unique: every output column
# of every row, so that a record taken from another place than its key shows
@pytest.mark.parametrize("strategy", ["partitioned", "sort"])
@pytest.mark.parametrize("order", [{"by": ["j", "k", "w"], "descending": [True, False, True], "offset": 5, "limit": 1000},
                                   {"by": ["k", "w", "j"], "nulls_last": [False, False, True], "offset": -900},
                                   {"by": ["w", "j", "k"], "descending": True, "offset": 2_000, "limit": 3}],
                         ids=lambda o: "-".join(o["by"]))
@pytest.mark.parametrize("kind", ["narrow", "wide"])
def test_ordered_slices(kind, order, strategy):
    rng = np.random.default_rng(len(kind))
    n = 120_000
    k = rng.integers(0, 3000, n)
    k = np.where(k % 2 == 0, k, -k) * (3_000_000_000_000_000 if kind == "wide" else 1)
    cols = {"k": (k, None), "j": (rng.integers(-20, 20, n).astype(np.int16), pack(rng.random(n) > 0.02)),
            "w": ((rng.integers(0, 2, n) * 2**30).astype(np.int32), None), "v": (rng.standard_normal(n), pack(rng.random(n) > 0.1))}
    keys, aggs = ["k", "j", "w"], [("Min", "v", "s"), ("Max", "v", "t"), ("Len", None, "c")]
    got = as_dict(N.groupby({c: N.ColumnData(*d) for c, d in cols.items()}, keys, aggs, strategy=strategy, sort=order))
    flags = lambda x: [bool(x)] * 3 if isinstance(x, bool) else list(x)  # noqa: E731
    want = pyoracle.sort_table(_table(pyoracle.groupby(cols, keys, aggs, None)), order["by"], flags(order.get("descending", False)),
                               flags(order.get("nulls_last", False)), False, order["offset"], order.get("limit", -1))
    assert_same_rows(got, want, f"{kind} {strategy}")


# the table of a learned estimate: three slots a predicted group (two made half of the tables too small)
@pytest.mark.parametrize("card,width", [(3000, 4), (90_000, 8), (400_000, 8)])
def test_slots_of_a_learned_estimate(card, width):
    rng = np.random.default_rng(card)
    n = 3_000_000
    q = ({"k": rng.integers(0, card, n).astype(np.int32 if width == 4 else np.int64), "v": rng.standard_normal(n)}, ["k"],
         [("Sum", "v", "s"), ("Len", None, "c")])
    strategy, groups = N.selector_choose(*q)
    got = N.groupby(*q)
    assert got.strategy == strategy
    if got.rehash_count == 0 and strategy.endswith("hash"):
        slots = min(max(3 * groups, 1024), 2 * n)
        assert got.capacity == (slots + 3) // 4 * 4


# the group-by's passes over two-word keys: tiles of 3072, its edges and remainders, the sort's digits and the
# partitions'; and with carried values (64 MB of them) over keys of one word (tiles of 3840) and of two
@pytest.mark.parametrize("strategy", ["partitioned", "sort"])
@pytest.mark.parametrize("n", [1, 2, 3071, 3072, 3073, 6143, 6144, 6145, 49_152])
def test_two_word_passes(n, strategy):
    rng = np.random.default_rng(n)
    k = rng.integers(-2**62, 2**62, n)
    cols = {"k": (k[rng.integers(0, max(1, n // 3), n)], None), "j": (rng.integers(-2**31, 2**31, n).astype(np.int32) >> 30, pack(rng.random(n) > 0.1)),
            "v": (rng.integers(-2**40, 2**40, n), None)}
    aggs = [("Sum", "v", "s"), ("Min", "v", "l"), ("Len", None, "c")]
    got = N.groupby({c: N.ColumnData(*d) for c, d in cols.items()}, ["k", "j"], aggs, strategy=strategy)
    assert got.strategy == strategy
    assert_results_match(as_dict(got), pyoracle.groupby(cols, ["k", "j"], aggs, None), 2, aggs)


@pytest.mark.parametrize("hint", [20_000, 400_000])  # one pass, two passes
@pytest.mark.parametrize("words,n", [(1, 729 * 3840 - 1), (1, 729 * 3840), (1, 729 * 3840 + 1), (2, 911 * 3072 - 1), (2, 911 * 3072),
                                     (2, 911 * 3072 + 1)])
def test_carried_tiles(words, n, hint):
    rng = np.random.default_rng(n)
    k = rng.integers(0, 15_000, n)
    cols = {"k": (k * (2**48 + 1 if words == 2 else 1), None), "x": (rng.integers(-2**40, 2**40, n), None),
            "y": (rng.integers(-2**40, 2**40, n), None), "z": (rng.integers(-2**40, 2**40, n), pack(rng.random(n) > 0.1))}
    keys = ["k"]
    if words == 2:
        cols["j"] = ((k % 5 * 2**29).astype(np.int32), None)
        keys.append("j")
    aggs = [("Sum", "x", "s"), ("Max", "y", "h"), ("Sum", "z", "t"), ("Count", "z", "c")]
    got = N.groupby({c: N.ColumnData(*d) for c, d in cols.items()}, keys, aggs, strategy="partitioned", capacity_hint=hint)
    assert got.strategy == "partitioned"
    assert_results_match(as_dict(got), pyoracle.groupby(cols, keys, aggs, None), len(keys), aggs)


# minima and maxima of Bool columns: bits, like the keys', in every strategy's last step, ordered by keys and by
# the aggregate itself
@pytest.mark.parametrize("jit", ["0", "1"])
@pytest.mark.parametrize("sort", [None, {"by": ["k"]}, {"by": ["lo", "k"]}], ids=["plain", "key", "aggregate"])
@pytest.mark.parametrize("strategy", ["smem_hash", "global_hash", "sort", "partitioned"])
@pytest.mark.parametrize("n,groups", [(1, 1), (40, 7), (5003, 1000), (60_000, 20_000)])
def test_bool_extremes(n, groups, strategy, sort, jit, monkeypatch):
    monkeypatch.setenv("PMB_JIT", jit)
    rng = np.random.default_rng(n)
    cols = {"k": (rng.integers(0, groups, n), None, A.I64, n), "b": (pack(rng.random(n) > 0.4), None, A.BOOL, n),
            "c": (pack(rng.random(n) > 0.6), pack(rng.random(n) > 0.3), A.BOOL, n)}
    aggs = [("Min", "b", "lo"), ("Max", "b", "hi"), ("Min", "c", "c_lo"), ("Max", "c", "c_hi"), ("Sum", "c", "s"), ("Len", None, "n")]
    got = as_dict(N.groupby({c: N.ColumnData(d, v, dtype=t, length=m) for c, (d, v, t, m) in cols.items()}, ["k"], aggs,
                            strategy=strategy, sort=sort))
    want = pyoracle.groupby(cols, ["k"], aggs, None)
    assert_results_match(got, want, 1, aggs, strategy)
    if sort:
        assert_same_rows(got, pyoracle.sort_table(_table(want), sort["by"], [False] * len(sort["by"]), [False] * len(sort["by"])), strategy)


def test_bool_extremes_in_a_batch():
    rng = np.random.default_rng(1)
    queries, wants = [], []
    aggs = [("Min", "b", "lo"), ("Max", "b", "hi"), ("Max", "c", "c_hi"), ("Len", None, "n")]
    for n in (1, 33, 2000, 70_000, 3, 9000):
        cols = {"k": (rng.integers(0, max(1, n // 4), n), None, A.I64, n), "b": (pack(rng.random(n) > 0.4), None, A.BOOL, n),
                "c": (pack(rng.random(n) > 0.6), pack(rng.random(n) > 0.3), A.BOOL, n)}
        queries.append(({c: N.ColumnData(d, v, dtype=t, length=m) for c, (d, v, t, m) in cols.items()}, ["k"], aggs, None))
        wants.append(pyoracle.groupby(cols, ["k"], aggs, None))
    for got, want in zip(N.groupby_batched(queries), wants):
        assert_results_match(as_dict(got), want, 1, aggs)


# which sorts go in one launch: up to 2048 rows all, up to 4096 those of one-word keys with two digits and more, up to
# 8192 those of a float of 64 bits alone (the passes of the others take less); the orders are right on both sides
@pytest.mark.parametrize("n", [2, 1024, 1025, 2048, 2049, 4096, 4097, 8192, 8193])
@pytest.mark.parametrize("case", [("int8", False, 2048), ("int16", False, 4096), ("int64", False, 4096), ("int64", True, 2048),
                                  ("float32", False, 4096), ("float64", False, 8192), ("float64", True, 4096)],
                         ids=lambda c: f"{c[0]}{'-null' * c[1]}")
def test_small_sort_rule(case, n):
    kind, nulls, largest = case
    rng = np.random.default_rng(n)
    a = rng.standard_normal(n).astype(kind) if kind[0] == "f" else rng.integers(-100, 100, n).astype(kind)
    cols = {"a": (a, pack(rng.random(n) > 0.2) if nulls else None), "row": (np.arange(n), None)}
    h = N.Handle(0)
    h.set_profiling(True)
    got = N.sort_columns({k: N.ColumnData(d, v) for k, (d, v) in cols.items()}, ["a"], [True], handle=h)
    assert ("order_small" in h.last_stats()["kernels"]) == (n <= largest)
    assert_same_rows(as_dict(got), pyoracle.sort_table(cols, ["a"], [True], [False]), f"{n} rows of {kind}")
    h.close()


# partitions with more groups than their table: the attempt ends at its first rows that find no slot, whatever
# the number of rows, and the sort strategy gives the result; one-word keys of fewer and of all 64 bits, two words
@pytest.mark.parametrize("kind", ["one word", "64 bits", "two words"])
def test_overflowing_partitions(kind):
    rng = np.random.default_rng(6)
    n = 1_500_000
    k = rng.permutation(n)
    cols = {"k": (k * 8191, None), "v": (rng.integers(0, 1000, n).astype(np.int32), None)}
    if kind == "64 bits":
        cols["k"] = (rng.integers(-2**63, 2**63 - 1, n), None)
    keys = ["k"]
    if kind == "two words":
        cols["k"] = (rng.integers(-2**63, 2**63 - 1, n), None)
        cols["j"] = ((k % 3).astype(np.int16), None)
        keys.append("j")
    aggs = [("Sum", "v", "s"), ("Max", "v", "m"), ("Len", None, "c")]
    h = N.Handle(0)
    h.set_profiling(True)
    data = {c: N.ColumnData(*d) for c, d in cols.items()}
    got = N.groupby(data, keys, aggs, strategy="partitioned", capacity_hint=5000, handle=h)
    assert got.strategy == "sort"
    assert_results_match(as_dict(got), pyoracle.groupby(cols, keys, aggs, None), len(keys), aggs)
    h.close()


# wide keys are packed from 100,000 rows on (their ranges are read), and where kernels are compiled at every size;
# on both sides one key, few and many, nulls among them
@pytest.mark.parametrize("jit", [None, "1"])
@pytest.mark.parametrize("groups", [1, 50, 20_000])
@pytest.mark.parametrize("n", [1, 500, 99_999, 100_000])
def test_packing_rule(n, groups, jit, monkeypatch):
    monkeypatch.setenv("PMB_JIT", jit) if jit else monkeypatch.delenv("PMB_JIT", raising=False)
    rng = np.random.default_rng(n + groups)
    cols = {"k": (rng.integers(0, groups, n) * 4099 - 7, pack(rng.random(n) > 0.1)), "v": (rng.standard_normal(n), None)}
    aggs = [("Sum", "v", "s"), ("Min", "v", "l"), ("Len", None, "c")]
    h = N.Handle(0)
    h.set_profiling(True)
    got = N.groupby({c: N.ColumnData(*d) for c, d in cols.items()}, ["k"], aggs, strategy="global_hash", handle=h)
    assert ("key_range" in h.last_stats()["kernels"]) == (n >= 100_000 or jit == "1")
    assert_results_match(as_dict(got), pyoracle.groupby(cols, ["k"], aggs, None), 1, aggs)
    h.close()
