"""The block-resident iterations (one persistent launch, arcs in shared
memory) against the launch-per-iteration kernels and the oracle, on the graph
shapes that reach every part of them: fewer arcs than a thread's chunk, rows
that span threads, warps and the 8192-arc tiles of a block, rows without
arcs, a hub, graphs for one block and for all of them, weights, both
numberings, teleport and start vectors, iteration caps.

Both routes add the same FP64 products and differ in the order of the row
sums only: per pass an L1 error of at most about 64 ulp of the unit mass
(7e-15), amplified by 1 / (1 - 0.85) over the iteration, so they agree to
1e-13 in L1 and take the same number of iterations."""
import numpy as np
import pytest

import igraph_b200 as ig
import oracle as O

pytestmark = pytest.mark.gpu


def _graph(case):
    """(n, from, to, directed)"""
    rng = np.random.default_rng(11)
    if case == "two":
        return 2, np.array([0], np.uint32), np.array([1], np.uint32), True
    if case == "loops":
        return 3, np.array([0, 0, 2, 2], np.uint32), np.array([0, 1, 2, 1], np.uint32), False
    if case == "star":  # one row of 15 000 arcs: two tiles of its block
        n = 5001
        return n, np.arange(1, n, dtype=np.uint32).repeat(3), np.zeros(3 * (n - 1), np.uint32), True
    if case == "empty_rows":
        f, t = O.erdos_renyi_gnm(30_000, 20_000, True, False, 5)
        return 30_000, f, t, True
    if case == "cycle":  # every arc ends a row
        n = 10_007
        f = np.arange(n, dtype=np.uint32)
        return n, f, ((f + 1) % n).astype(np.uint32), True
    if case == "er_undirected":
        f, t = O.erdos_renyi_gnm(1000, 25_000, False, False, 7)
        return 1000, f, t, False
    if case == "ba":
        n = 20_000
        f, t = O.barabasi_game_bag(n, 8, False, False, 3)
        return n, f, t, False
    if case == "dense_rows":  # rows of 300 .. 2000 arcs
        n = 700
        m = 600_000
        return n, rng.integers(0, n, m).astype(np.uint32), (rng.integers(0, n, m) ** 2 // n).astype(np.uint32), True
    if case == "streamed":  # indices too many for shared memory (weights from 1.9 M arcs on), skewed both ways
        n = 150_001
        f = (rng.random(7_300_013) ** 2 * n).astype(np.uint32)
        return n, f, (rng.random(len(f)) ** 3 * n).astype(np.uint32), True
    n = 1 << 16  # rmat: all blocks, several tiles each
    f, t = O.rmat(16, 40 * n, seed=3)
    return n, f, t, True


CASES = ["two", "loops", "star", "empty_rows", "cycle", "er_undirected", "ba", "dense_rows", "rmat", "streamed"]


def _both(n, f, t, directed, w, relabel, call):
    out = []
    for resident in (1, 0):
        ig.set_tuning("resident", resident)
        ig.set_tuning("relabel", relabel)
        try:
            with ig.DeviceGraph.from_host(n, f, t, directed, w) as dg:
                out.append(call(dg))
        finally:
            ig.reset_tuning()
    return out


@pytest.mark.parametrize("relabel", [0, 1])
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("case", CASES)
def test_power_iteration_matches_the_launched_kernels(cuda_ok, case, weighted, relabel):
    n, f, t, directed = _graph(case)
    rng = np.random.default_rng(2)
    w = rng.uniform(0.1, 3.0, len(f)) if weighted else None
    if weighted and len(f) > 10:
        w[::7] = 0.0
    reset = rng.uniform(0.0, 1.0, n) ** 8
    start = rng.uniform(0.5, 1.0, n)
    start /= start.sum()

    def call(dg):
        return [dg.solve(), dg.solve(reset=reset), dg.solve(start=start), dg.solve(ig.Options(max_iter=1)),
                dg.solve(ig.Options(max_iter=7, stop=ig.STOP_ERROR_BOUND), reset=reset)]

    a, b = _both(n, f, t, directed, w, relabel, call)
    for (xa, sa), (xb, sb) in zip(a, b):
        assert sa.iterations == sb.iterations
        assert np.abs(xa - xb).sum() <= 1e-13
        assert abs(sa.last_diff - sb.last_diff) <= 1e-13
    ref = O.pagerank_weighted(n, f, t, directed, w) if weighted else O.pagerank(n, f, t, directed)
    assert np.abs(a[0][0] - ref).max() <= 1e-10


def test_power_iteration_continues_over_launches(cuda_ok):
    # slower than one launch's iterations (d near 1 on a cycle), and capped
    n, f, t, directed = _graph("cycle")
    reset = np.zeros(n)
    reset[5] = 1.0
    opts = ig.Options(damping=0.9995, max_iter=9001)
    (xa, sa), (xb, sb) = _both(n, f, t, directed, None, 0, lambda dg: dg.solve(opts, reset=reset))
    assert sa.iterations == sb.iterations == 9001
    assert np.abs(xa - xb).sum() <= 7e-15 / (1 - 0.9995)


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("case", ["loops", "star", "cycle", "er_undirected", "ba", "dense_rows", "streamed"])
def test_eigenvector_matches_the_oracle(cuda_ok, case, weighted):
    n, f, t, _ = _graph(case)
    if case == "streamed":  # undirected: twice the arcs
        f, t = f[:4_000_001], t[:4_000_001]
    lo, hi = np.minimum(f, t), np.maximum(f, t)
    g = ig.Graph.from_edge_arrays(n, lo, hi, False)
    w = np.random.default_rng(4).uniform(0.5, 2.0, len(f)) if weighted else None
    got = []
    for resident in (1, 0):
        ig.set_tuning("resident", resident)
        try:
            got.append(ig.eigenvector_centrality_weighted(g, w, True) if weighted
                       else ig.eigenvector_centrality(g, True))
        finally:
            ig.reset_tuning()
    (xa, la), (xb, lb) = got
    assert abs(la - lb) <= 1e-10 * abs(lb)
    assert np.abs(xa - xb).max() <= 1e-10


@pytest.mark.parametrize("odd", [np.inf, np.nan, 1e308])
def test_eigenvector_with_weights_beyond_the_finite_range(cuda_ok, odd):
    # infinite and NaN components appear exactly where plain FP64 sums give them
    n, f, t, _ = _graph("er_undirected")
    g = ig.Graph.from_edge_arrays(n, np.minimum(f, t), np.maximum(f, t), False)
    w = np.ones(len(f))
    w[::500] = odd
    got = []
    for resident in (1, 0):
        ig.set_tuning("resident", resident)
        try:
            got.append(ig.eigenvector_centrality_weighted(g, w, True))
        finally:
            ig.reset_tuning()
    assert np.array_equal(np.isnan(got[0][0]), np.isnan(got[1][0]))
    ok = ~np.isnan(got[0][0])
    assert np.abs(got[0][0][ok] - got[1][0][ok]).max(initial=0.0) <= 1e-10
