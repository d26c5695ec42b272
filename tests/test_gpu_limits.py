"""GPU behaviour at the limits of a handle: streams other than its own, device memory that runs short, waits
that give up, kernels that cannot be compiled. Failures are made on the host; every call ends with the right
result or with an error, and the handle stays usable."""

import ctypes as C

import numpy as np
import pytest

from helpers import as_dict, assert_results_match, pack
from oracle import pyoracle
from polars_b200 import _native as N

pytestmark = pytest.mark.gpu


def faults(h, jit_kernels=-1, wait=False, workspace=0):
    """Failures that the calls of a handle meet from here on (pmb_debug_faults); no arguments: none."""
    h._lib.pmb_debug_faults(h.raw, C.c_int32(jit_kernels), C.c_int32(wait), C.c_int64(workspace))


def device_bytes(ptr, nbytes):
    rt = C.CDLL("libcudart.so.12")
    rt.cudaMemcpy.argtypes = [C.c_void_p, C.c_void_p, C.c_size_t, C.c_int]
    out = np.empty(nbytes, np.uint8)
    assert rt.cudaMemcpy(out.ctypes.data, ptr, nbytes, 2) == 0
    return out


STREAM_LEGACY, STREAM_PER_THREAD = 1, 2  # cudaStreamLegacy, cudaStreamPerThread


# pageable columns large enough for the staging threads: their copies come before the call's kernels
# whatever stream the handle launches on
@pytest.mark.parametrize("stream", [None, STREAM_LEGACY, STREAM_PER_THREAD, "torch"])
def test_pageable_columns_on_any_stream(stream):
    import torch

    side = torch.cuda.Stream()
    h = N.Handle(0)
    h.set_stream(side.cuda_stream if stream == "torch" else stream)
    n = 6_000_011
    for seed in range(4):  # other values each time, so that a stale chunk shows
        rng = np.random.default_rng(seed)
        k, x, ok = rng.integers(0, 5, n), rng.integers(-2**40, 2**40, n), rng.random(n) > 0.25
        got = as_dict(N.groupby({"k": k, "x": N.ColumnData(x, pack(ok))}, ["k"], [("Sum", "x", "s"), ("Count", "x", "c")],
                                sort={"by": "k"}, handle=h))
        assert np.array_equal(got["data"][1][:5], [x[(k == i) & ok].sum() for i in range(5)])
        assert np.array_equal(got["data"][2][:5], [((k == i) & ok).sum() for i in range(5)])
    h.close()


# the compiled aggregation of carried values is the only kernel that can read them: no second one is asked for
# when the tables of two CTAs an SM turn out too small (819K groups in 256 partitions, by the hint's estimate)
@pytest.mark.parametrize("kernels", [0, 1, -1])
def test_carried_values_need_one_kernel(kernels, monkeypatch):
    monkeypatch.setenv("PMB_JIT", "1")
    h = N.Handle(0)
    n, groups = 4_400_003, 819_200
    rng = np.random.default_rng(kernels + 5)
    k = np.concatenate([np.arange(groups), rng.integers(0, groups, n - groups)])
    cols = {"k": (k, None), "x": (rng.integers(-2**40, 2**40, n), None), "y": (rng.standard_normal(n), None)}
    # one aggregate more for each case: a signature that no other case has compiled
    aggs = [("Sum", "x", "s"), ("Max", "y", "hi")] + [("Min", "y", "lo")] * (kernels >= 0) + [("Max", "x", "h")] * (kernels == 0)
    faults(h, jit_kernels=kernels)
    h.set_profiling(True)
    got = N.groupby({c: N.ColumnData(*d) for c, d in cols.items()}, ["k"], aggs, strategy="partitioned", capacity_hint=100_000,
                    handle=h)
    if kernels:  # too few output rows, too small tables, and the one that holds them
        assert got.strategy == "partitioned" and h.last_stats()["kernels"]["part_agg"]["launches"] == 3
    assert_results_match(as_dict(got), pyoracle.groupby(cols, ["k"], aggs, None), 1, aggs, f"{kernels} kernels")
    h.close()


def _sort_columns(h, seed, by, n):
    rng = np.random.default_rng(seed)
    cols = {c: rng.integers(-2**62, 2**62, n) for c in "abc"} | {"s": rng.integers(0, 2**20, n).astype(np.int32)}
    return N.sort_columns(cols, by, output="device", handle=h), [8, 8, 8, 4]


def _sorted_groups(h, seed, strategy, by, n):
    rng = np.random.default_rng(seed)
    k = rng.permutation(n)  # a group a row, so that every call has the same sizes
    cols = {"k": k * (2**40 if strategy == "two words" else 1), "j": (k % 1000).astype(np.int32), "v": rng.integers(0, 2**40, n),
            "w": rng.integers(-2**40, 2**40, n)}
    keys = ["k", "j"] if strategy == "two words" else ["k"]
    # by an aggregate: the wanted order is not the keys'; the packed keys of "two words" need two
    if strategy == "two words":
        cols["k"], strategy = cols["k"] * 4001, "partitioned"
    got = N.groupby(cols, keys, [("Sum", "v", "s"), ("Max", "w", "m")], strategy=strategy, sort={"by": by}, output="device", handle=h,
                    capacity_hint=n)
    return got, [8] + [4] * (len(keys) - 1) + [8, 8]


# a wait of the sort's passes that gave up (a status that the host sets): the call ends with an error, and nothing
# that follows has used the row numbers: the device result of the call before is still there, byte for byte
@pytest.mark.parametrize("jit", ["0", "1"])
@pytest.mark.parametrize("call", [(_sort_columns, ["s"], 20_000), (_sort_columns, ["a", "s"], 20_000),
                                  (_sort_columns, ["a", "b", "c"], 20_000), (_sort_columns, ["a", "b"], 1_100_000),
                                  (_sorted_groups, "global_hash", ["s"], 30_000), (_sorted_groups, "partitioned", ["k"], 30_000),
                                  (_sorted_groups, "partitioned", ["m"], 30_000), (_sorted_groups, "two words", ["j", "k"], 30_000),
                                  (_sorted_groups, "sort", ["k"], 30_000), (_sorted_groups, "partitioned", ["k"], 4_300_000)],
                         ids=lambda c: "-".join(map(str, c[1:])))
def test_sort_that_gives_up(call, jit, monkeypatch):
    monkeypatch.setenv("PMB_JIT", jit)
    run, *args, n = call
    h = N.Handle(0)
    run(h, 1, *args, n)  # (a second call finds the workspace in one block, every later one at the same addresses)
    first, widths = run(h, 2, *args, n)
    before = [device_bytes(p, n * b) for p, b in zip(first.data, widths)]
    faults(h, wait=True)
    with pytest.raises(RuntimeError, match="timed out"):
        run(h, 3, *args, n)
    assert all(np.array_equal(device_bytes(p, n * b), was) for p, b, was in zip(first.data, widths, before))
    faults(h)
    again, _ = run(h, 2, *args, n)
    assert again.data == first.data
    assert all(np.array_equal(device_bytes(p, n * b), was) for p, b, was in zip(again.data, widths, before))
    h.close()


# an expression's column goes into memory that torch hands out while earlier work of torch's stream still writes
# to it: the call waits for that work, and what it wrote stays
@pytest.mark.parametrize("n", [1, 1000, 300_001])
def test_expression_behind_work_in_flight(n):
    import torch

    x = torch.arange(n, dtype=torch.int64, device="cuda")
    e = {"kind": "Arith", "op": "Add", "lhs": {"kind": "Column", "name": "x"}, "rhs": {"kind": "Column", "name": "x"}}
    k, key = np.arange(n) % 3, x % 3
    for _ in range(2):
        torch.cuda.synchronize()
        torch.cuda._sleep(200_000_000)  # 0.1 s
        del_me = [torch.full((n,), 7, dtype=torch.int64, device="cuda"), torch.zeros(N._bitmap_bytes(n), dtype=torch.uint8, device="cuda")]
        del del_me  # back to torch's allocator, the fills still to come
        got = N.eval_expr({"x": N.ColumnData(x)}, e)
        torch.cuda.synchronize()
        assert np.array_equal(got.data.cpu().numpy()[:n], 2 * np.arange(n))
        bits = np.unpackbits(got.validity.cpu().numpy(), bitorder="little")
        assert bits[:n].all() and not bits[n:].any()
        torch.cuda._sleep(200_000_000)
        g = N.groupby({"k": N.ColumnData(key), "x": N.ColumnData(x)}, ["k"], [("Sum", e, "s"), ("Count", e, "c")], sort={"by": "k"})
        assert [int(v) for v in g.data[1][: min(n, 3)]] == [int((2 * np.arange(n))[k == i].sum()) for i in range(min(n, 3))]
        assert [int(v) for v in g.data[2][: min(n, 3)]] == [int((k == i).sum()) for i in range(min(n, 3))]


# device outputs of an expression: this GPU's memory in place, pinned host memory by a copy, pageable memory refused
@pytest.mark.parametrize("jit", ["0", "1"])
@pytest.mark.parametrize("kind", ["device", "pinned", "pageable", "pageable validity"])
def test_expression_output_memory(kind, jit, monkeypatch):
    import torch

    monkeypatch.setenv("PMB_JIT", jit)
    n = 5003
    x = torch.arange(n, dtype=torch.int64, device="cuda")
    abi, _keep = N._to_abi_columns([N.ColumnData(x)])
    e, _k = N.compile_predicate({"kind": "Arith", "op": "Mul", "lhs": {"kind": "Column", "name": "x"},
                                 "rhs": {"kind": "Column", "name": "x"}}, {"x": 0})

    def memory(size, dtype, pageable):
        return torch.zeros(size, dtype=dtype, device="cuda" if kind != "pinned" and not pageable else None, pin_memory=kind == "pinned")

    data = memory(n, torch.int64, kind == "pageable")
    valid = memory(N._bitmap_bytes(n), torch.uint8, kind.startswith("pageable"))
    torch.cuda.synchronize()
    h, dt = N.default_handle(), C.c_int32()
    rc = h._lib.pmb_eval_expr(h.raw, C.byref(e), abi, 1, data.data_ptr(), valid.data_ptr(), 1, C.byref(dt))
    if kind.startswith("pageable"):
        with pytest.raises(ValueError, match="not CUDA memory"):
            h.check(rc)
        return
    h.check(rc)
    assert np.array_equal(data.cpu().numpy(), np.arange(n) ** 2)
    assert np.unpackbits(valid.cpu().numpy(), bitorder="little")[:n].all()


# a workspace too small for the values that the partition passes would carry: the call runs without carrying them,
# down to the least that it needs so, plain, sorted by a key and sorted by an aggregate
@pytest.mark.parametrize("sort", [None, {"by": "k"}, {"by": ["m", "k"]}], ids=["plain", "key", "aggregate"])
def test_workspace_without_carried_values(sort, monkeypatch):
    import torch

    monkeypatch.setenv("PMB_JIT", "1")
    n, groups = 4_300_003, 400_000
    rng = np.random.default_rng(3)
    k = np.concatenate([np.arange(groups), rng.integers(0, groups, n - groups)])
    cols = {"k": (k, None)} | {c: (rng.integers(-2**40, 2**40, n), None) for c in "xyz"}
    aggs = [("Sum", "x", "s"), ("Max", "y", "m"), ("Min", "z", "l")]
    want = pyoracle.groupby(cols, ["k"], aggs, None)
    data = {c: N.ColumnData(torch.from_numpy(d).cuda()) for c, (d, _) in cols.items()}
    torch.cuda.synchronize()

    def run(workspace):
        h = N.Handle(0)
        faults(h, workspace=workspace)
        try:
            got = N.groupby(data, ["k"], aggs, strategy="partitioned", capacity_hint=groups, sort=sort, handle=h)
        except MemoryError:
            return False
        finally:
            h.close()
        if sort:
            assert (np.diff(got.data[0] if sort["by"] == "k" else got.data[2]) >= 0).all()
        assert got.strategy == "partitioned"
        assert_results_match(as_dict(got), want, 1, aggs, f"{workspace} bytes")
        return True

    MB = 1 << 20
    assert run(0)
    fits = [w for w in range(640, 159, -20) if run(w * MB)]
    assert fits and fits == list(range(640, fits[-1] - 1, -20))  # whatever fits a workspace fits a larger one
    assert fits[-1] * MB < 2 * n * (12 + 24), fits  # keys, row numbers and 24 bytes of values a row, twice each


# a workspace too small for the groups' order keys (two words each, the sort column's own key one): the finished
# columns are sorted instead, down to what that needs
def test_workspace_without_order_keys(monkeypatch):
    import torch

    monkeypatch.setenv("PMB_JIT", "1")
    n = 2_000_003  # a group a row; too few values to carry
    rng = np.random.default_rng(4)
    k = rng.permutation(n)
    cols = {"k": (k * (2**42 + 1), None), "j": (k.astype(np.int32), None), "x": (rng.integers(-2**40, 2**40, n), None)}
    want = np.argsort(k)[-1000:][::-1]
    data = {c: N.ColumnData(torch.from_numpy(d).cuda()) for c, (d, _) in cols.items()}
    torch.cuda.synchronize()

    def run(workspace):
        h = N.Handle(0)
        h.set_profiling(True)
        faults(h, workspace=workspace)
        try:
            got = N.groupby(data, ["k", "j"], [("Sum", "x", "s")], strategy="partitioned", capacity_hint=n,
                            sort={"by": "j", "descending": True, "limit": 1000}, handle=h)
            kernels = h.last_stats()["kernels"]
        except MemoryError:
            return None
        finally:
            h.close()
        assert got.strategy == "partitioned" and got.n_groups == 1000
        for have, c in zip(got.data, ("k", "j", "x")):
            assert np.array_equal(have, cols[c][0][want])
        return "ordered" if "ordered_finalize" in kernels else "columns"

    MB = 1 << 20
    how = [run(w * MB) for w in range(600, 99, -4)]
    assert how[0] == run(0) == "ordered" and how[-1] is None
    assert "columns" in how and how == sorted(how, key=["ordered", "columns", None].index)


# pageable columns around what the staging threads take (columns of 4 MB, calls of 20 MB of them) and their chunks: one
# column or several, sizes that no chunk divides, the values and their places right
@pytest.mark.parametrize("cols,n", [(1, 524_287), (1, 524_288), (1, 2_621_439), (1, 2_621_440), (1, 2_621_441), (1, 5_000_011),
                                    (3, 524_288), (3, 873_813), (3, 873_815), (5, 524_287), (5, 524_288), (2, 4_194_305)])
def test_staged_column_sizes(cols, n):
    rng = np.random.default_rng(n)
    data = {f"c{i}": rng.integers(-2**62, 2**62, n) for i in range(cols)}
    data["c0"][0] = -2**62  # the one row that goes
    for _ in range(2):
        got = N.filter_columns(data, {"kind": "Compare", "op": "Gt", "lhs": {"kind": "Column", "name": "c0"},
                                      "rhs": {"kind": "LiteralI64", "value": -2**62}})
        keep = data["c0"] > -2**62
        m = int(keep.sum())
        assert got.n_groups == m
        for have, d in zip(got.data, data.values()):
            assert np.array_equal(have[:m], d[keep])


# a stream that torch is capturing into a graph (relaxed, so that other streams may run): the expression is evaluated
# at once, on the library's stream, and neither joins the capture nor ends it
def test_expression_beside_a_capture():
    import torch

    x = torch.arange(1000, dtype=torch.int64, device="cuda")
    e = {"kind": "Arith", "op": "Add", "lhs": {"kind": "Column", "name": "x"}, "rhs": {"kind": "Column", "name": "x"}}
    N.eval_expr({"x": N.ColumnData(x)}, e)  # (a capture allocates from a pool of its own, the library not at all)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="relaxed"):
        y = x + 1
        got = N.eval_expr({"x": N.ColumnData(x)}, e)
    for _ in range(2):
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, x + 1) and torch.equal(got.data[:1000], 2 * x)
        assert np.unpackbits(got.validity.cpu().numpy(), bitorder="little")[:1000].all()
