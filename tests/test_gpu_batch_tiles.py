"""The last tile of a batch takes the narrowest kernel that holds its columns
(8, 16, 32 or 64 wide): every width against the oracle, and column by column
against the full-width kernel.

Tolerance: 1e-6 in L1 per column, the stop rule's 1e-8 d/(1-d) plus FP32
rounding of a vector of unit mass.  A column's arithmetic does not depend on
the width of its tile (only the FP64 order of its stop sums does), so its
iterate is bit-equal wherever the iteration counts agree.
"""
import numpy as np
import pytest

import igraph_b200 as ig
import oracle as O

pytestmark = pytest.mark.gpu


def graph(n, directed, seed):
    # dangling vertices, a hub row of n arcs, rows of every length modulo 4
    rng = np.random.default_rng(seed)
    m = 6 * n
    f = rng.integers(0, max(n - 5, 1), m).astype(np.uint32)
    t = rng.integers(0, n, m).astype(np.uint32)
    t[: n] = 1 % n
    return f, t


@pytest.mark.parametrize("n,directed", [(3, True), (37, False), (5000, True), (5000, False)])
@pytest.mark.parametrize("K", [1, 8, 9, 16, 17, 32, 33, 64, 65, 73, 97])
def test_last_tile_widths(cuda_ok, n, directed, K):
    f, t = graph(n, directed, n + K)
    rng = np.random.default_rng(K)
    seeds = [rng.integers(0, n, 1 + k % 5).astype(np.uint32) for k in range(K)]
    pad = seeds + [seeds[0]] * (64 * ((K + 63) // 64) - K)  # every tile full
    with ig.DeviceGraph.from_host(n, f, t, directed) as dg:
        X, iters, st = dg.ppr_batch(seeds, 0.85, 1e-8, 1000, 2)
        full, fiters, _ = dg.ppr_batch(pad, 0.85, 1e-8, 1000, 2)
    assert X.shape == (n, K) and st["tiles"] == (K + 63) // 64
    assert np.abs(iters.astype(int) - fiters[:K].astype(int)).max() <= 1
    same = iters == fiters[:K]
    assert np.array_equal(X[:, same], full[:, :K][:, same])
    for k in range(0, K, 7):
        r = np.zeros(n)
        np.add.at(r, seeds[k], 1.0 / len(seeds[k]))
        ref = O.personalized_pagerank(n, f, t, directed, r, 0.85)
        assert np.abs(X[:, k].astype(np.float64) - ref).sum() <= 1e-6
