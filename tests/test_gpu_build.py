"""The device CSR build against numpy: arcs stably sorted by destination, rows
and sources in internal ids (integers, compared exactly), for key widths of 0
to 4 radix digits and edge counts around the kernels' tiles; the caller's edge
arrays stay as they are.  Weighted graphs through the solve, against the
oracle (1e-9 relative: the stop rule's 1e-10, far above FP64 rounding)."""
import numpy as np
import pytest
import torch

import igraph_b200 as ig
import oracle as O
from test_gpu_streamed_build import csr, device_arrays

pytestmark = pytest.mark.gpu

SIZES = [(1, 0), (1, 3), (2, 1), (5, 7), (200, 127), (200, 129), (300, 2049), (70_000, 33_000), (5000, 300_001),
         ((1 << 24) + 5, 4097)]


def edges(n, m):
    rng = np.random.default_rng(n + m)
    f = (rng.random(m) ** 3 * n).astype(np.uint32)  # hubs at the small ids, most rows empty
    t = rng.integers(0, n, m).astype(np.uint32)
    t[: m // 3] = n // 2
    return f, t


@pytest.mark.parametrize("n,m", SIZES)
@pytest.mark.parametrize("directed", [True, False])
@pytest.mark.parametrize("relabel", [0, 1])
def test_csr_matches_numpy(cuda_ok, n, m, directed, relabel):
    f, t = edges(n, m)
    df, dt, _ = device_arrays(f, t)
    try:
        ig.set_tuning("relabel", relabel)
        with ig.DeviceGraph.from_device(n, m, df.data_ptr(), dt.data_ptr(), directed) as dg:
            got = csr(dg)
    finally:
        ig.reset_tuning()
    assert np.array_equal(df.cpu().numpy().view(np.uint32), f)
    assert np.array_equal(dt.cpu().numpy().view(np.uint32), t)
    src, dst = (f, t) if directed else (np.stack([t, f], 1).ravel(), np.stack([f, t], 1).ravel())
    out = np.bincount(src, minlength=n)
    perm = np.arange(n)
    if relabel and n >= 2:
        noin = np.bincount(dst, minlength=n) == 0 if directed else np.zeros(n, bool)
        perm = np.lexsort((perm, -out, noin))
        assert np.array_equal(got["perm"], perm)
    iperm = np.empty(n, np.int64)
    iperm[perm] = np.arange(n)
    d, s = iperm[dst], iperm[src]
    order = np.argsort(d, kind="stable")
    assert np.array_equal(got["col"], s[order])
    assert np.array_equal(got["row_ptr"], np.concatenate([[0], np.cumsum(np.bincount(d, minlength=n))]))
    with np.errstate(divide="ignore"):
        inv = np.where(out[perm] > 0, 1.0 / out[perm], 0.0).astype(np.float32)
    assert np.array_equal(got["inv32"], inv)


@pytest.mark.parametrize("n,m", [(5, 7), (300, 2049), (5000, 30_001)])
@pytest.mark.parametrize("directed", [True, False])
@pytest.mark.parametrize("relabel", [0, 1])
def test_weighted_build_matches_oracle(cuda_ok, n, m, directed, relabel):
    f, t = edges(n, m)
    w = np.random.default_rng(m).random(m) + 0.25
    df, dt, dw = device_arrays(f, t, w)
    try:
        ig.set_tuning("relabel", relabel)
        with ig.DeviceGraph.from_device(n, m, df.data_ptr(), dt.data_ptr(), directed, dw.data_ptr()) as dg:
            x = dg.solve()[0]
    finally:
        ig.reset_tuning()
    ref = O.pagerank_weighted(n, f, t, directed, w)
    assert np.abs(x - ref).sum() <= 1e-9
