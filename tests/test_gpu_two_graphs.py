"""Resident graphs of different sizes used in turn: a launch limit that one of
them sets on a kernel must not be too small for the other.  Relabelled graphs,
whose hot prefix in shared memory is as long as the graph allows, so the small
graph asks for less than the large one.  The same solve on the same graph has
the same bits whatever ran in between (all reductions are fixed trees)."""
import numpy as np
import pytest

import igraph_b200 as ig

pytestmark = pytest.mark.gpu

PRECISIONS = [ig.PRECISION_FP64, ig.PRECISION_LINSYS, ig.PRECISION_FP32_REFINED, ig.PRECISION_FP64_KRYLOV]
ROUTES = {"default": {}, "launched": {"resident": 0}, "quads": {"resident": 0, "seg_kry32": 1},
          "row_blocks": {"resident": 0, "seg_kry32": 0, "seg_res64": 0, "seg_plain64": 0, "hot_cache": 32768}}


def graph(n, m, weighted):
    rng = np.random.default_rng(n)
    f = (rng.random(m) ** 3 * n).astype(np.uint32)
    t = rng.integers(0, n, m).astype(np.uint32)
    return ig.DeviceGraph.from_host(n, f, t, True, rng.random(m) + 0.5 if weighted else None)


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("route", ROUTES)
def test_large_small_large(cuda_ok, route, precision, weighted):
    opts = ig.Options(precision=precision)
    try:
        ig.set_tuning("relabel", 1)
        for k, v in ROUTES[route].items():
            ig.set_tuning(k, v)
        with graph(100_000, 1_000_000, weighted) as large, graph(3000, 30_000, weighted) as small:
            a, _ = large.solve(opts)
            b, _ = small.solve(opts)
            assert np.array_equal(large.solve(opts)[0], a)
            assert np.array_equal(small.solve(opts)[0], b)
    finally:
        ig.reset_tuning()
