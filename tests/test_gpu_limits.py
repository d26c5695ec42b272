"""GPU behaviour at the limits of a handle: streams other than its own, device memory that runs short, waits
that give up, kernels that cannot be compiled. Failures are made on the host; every call ends with the right
result or with an error, and the handle stays usable."""

import numpy as np
import pytest

from helpers import as_dict, pack
from polars_b200 import _native as N

pytestmark = pytest.mark.gpu

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
