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


def faults(h, jit_kernels=-1):
    """Failures that the calls of a handle meet from here on (pmb_debug_faults); no arguments: none."""
    h._lib.pmb_debug_faults(h.raw, C.c_int32(jit_kernels))


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
