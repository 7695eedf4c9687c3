"""The bounded grid barriers of the block-resident iterations and of the
small-graph build, each made to wait for an arrival that never comes: after
about 1.5 s the call reports the timeout, nothing stays allocated, and the next
call on the same graph gives the same bits as before."""
import numpy as np
import pytest

import igraph_b200 as ig
from test_gpu_out_of_memory import Pool

pytestmark = pytest.mark.gpu

N, M = 4000, 30_000


def edges():
    rng = np.random.default_rng(9)
    return rng.integers(0, N, M).astype(np.uint32), rng.integers(0, N, M).astype(np.uint32)


def calls():
    f, t = edges()
    d = ig.Graph.from_edge_arrays(N, f, t, True)
    u = ig.Graph.from_edge_arrays(N, np.minimum(f, t), np.maximum(f, t), False)
    w = np.random.default_rng(1).random(M) + 0.5
    return {"pagerank": lambda: ig.pagerank(d), "weighted": lambda: ig.pagerank_weighted(d, w),
            "eigenvector": lambda: ig.eigenvector_centrality(u),
            "eigenvector_directed": lambda: ig.eigenvector_centrality_directed(d, 0).vector}


def times_out(call, hook):
    try:
        ig.set_tuning("resident_barrier_extra", hook)
        with pytest.raises(ig.DeviceTimeout, match="grid barrier timed out"):
            call()
    finally:
        ig.reset_tuning()


# hook 1: the iteration's barrier, 2: the build's (directed eigenvectors are built by the general path)
@pytest.mark.parametrize("kind,hook", [(k, h) for k in ("pagerank", "weighted", "eigenvector") for h in (1, 2)] +
                         [("eigenvector_directed", 1)])
def test_drop_in(cuda_ok, kind, hook):
    call = calls()[kind]
    ref = call()
    pool = Pool()
    before = pool.used()
    times_out(call, hook)
    pool.rt.cudaDeviceSynchronize()
    assert pool.used() == before
    assert np.array_equal(call(), ref)


def test_resident_graph(cuda_ok):
    f, t = edges()
    with ig.DeviceGraph.from_host(N, f, t, True) as dg:
        ref, _ = dg.solve()
        times_out(dg.solve, 1)
        assert np.array_equal(dg.solve()[0], ref)
