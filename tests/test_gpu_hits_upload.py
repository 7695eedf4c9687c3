"""HITS on directed graphs uploads the edge list once for the graph and its
reverse; both sides of the streamed build's limit (2^23 edges), weighted and
not, and the range error.

Check: with A the (multi-edge) adjacency matrix in FP64, hub and authority
must be fixed points of h -> A a, a -> A^T h up to scale.  The iteration stops
at an L1 change of 1e-14 with maxima scaled to 1; these graphs have a large
spectral gap (random, dense), so the residual is a few hundred roundings of
8-byte sums over rows of ~3000 entries: 1e-11 of the maximum.
"""
import numpy as np
import pytest
from scipy.sparse import coo_matrix

import igraph_b200 as ig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [(1 << 23) - 1, 1 << 23, (1 << 23) + 3])
@pytest.mark.parametrize("weighted", [False, True])
def test_both_directions(cuda_ok, m, weighted):
    n = 3000
    rng = np.random.default_rng(m)
    f = (rng.random(m) ** 2 * n).astype(np.uint32)
    t = rng.integers(0, n, m).astype(np.uint32)
    g = ig.Graph.from_edge_arrays(n, f, t, True)
    w = rng.random(m) + 0.5 if weighted else np.ones(m)
    r = ig.hub_and_authority_scores_weighted(g, w) if weighted else ig.hub_and_authority_scores(g)
    A = coo_matrix((w, (f, t)), shape=(n, n)).tocsr()
    for x, y in ((r.hub, A @ r.authority), (r.authority, A.T @ r.hub)):
        assert abs(x.max() - 1) <= 1e-12
        assert np.abs(y / y.max() - x).max() <= 1e-11


@pytest.mark.parametrize("m", [100_000, 1 << 23])
def test_out_of_range_endpoint(cuda_ok, m):
    f = np.zeros(m, np.uint32)
    t = np.ones(m, np.uint32)
    t[m - 1] = 50
    out = [np.empty(50), np.empty(50)]
    with pytest.raises(Exception, match="vertex id 50 out of range"):
        ig._check(ig.lib().prg_hub_and_authority_scores(50, m, ig._ptr(f), ig._ptr(t), 1, ig._ptr(out[0]),
                                                        ig._ptr(out[1]), None))
