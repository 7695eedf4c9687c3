"""One-call drop-ins on small graphs (one build launch, one iteration launch)
against the resident-graph path and the oracle.

The small build must give the general build's CSR: with caller ids
(relabel = 0) the drop-in's result then has the same bits as a solve on a
resident graph, because both run the same iteration kernel.  Row lengths cover
the warp's 32-arc and 128-arc limits, the block sort (ids over several of its
ranges) and rows too long for an equal split; the oracle bounds the rest at
1e-10."""
import numpy as np
import pytest

import igraph_b200 as ig
import oracle as O

pytestmark = pytest.mark.gpu


def _graph(case):
    rng = np.random.default_rng(21)
    if case == "two":
        return 2, np.array([0, 1, 1], np.uint32), np.array([1, 1, 0], np.uint32)
    if case == "gnm":
        n = 1000
        return n, rng.integers(0, n, 25_000).astype(np.uint32), rng.integers(0, n, 25_000).astype(np.uint32)
    if case == "row_lengths":  # in-rows of 0..40, 127..129, 511..514, 1023..1025, 5000 arcs, edges shuffled
        lens = list(range(41)) + [127, 128, 129, 511, 512, 513, 514, 1023, 1024, 1025, 5000]
        t = np.repeat(np.arange(len(lens)), lens)
        rng.shuffle(t)
        return 400, rng.integers(0, 400, len(t)).astype(np.uint32), t.astype(np.uint32)
    if case == "long_hub":  # one row of 60 000 arcs, more than 2^20 arc ids
        t = np.concatenate([np.zeros(60_000, np.uint32), rng.integers(1, 90_000, 1_100_000).astype(np.uint32)])
        rng.shuffle(t)
        return 90_000, rng.integers(0, 90_000, len(t)).astype(np.uint32), t
    if case == "star":
        t = np.zeros(33_000, np.uint32)
        return 50_000, rng.integers(1, 50_000, len(t)).astype(np.uint32), t
    n = 120_011  # powerlaw: many rows, hubs of a few thousand arcs
    return n, (n * rng.random(700_003) ** 4).astype(np.uint32), (n * rng.random(700_003) ** 4).astype(np.uint32)


CASES = ["two", "gnm", "row_lengths", "long_hub", "star", "powerlaw"]


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("directed", [True, False])
@pytest.mark.parametrize("case", CASES)
def test_drop_ins_match_resident_solves(cuda_ok, case, directed, weighted):
    n, f, t = _graph(case)
    g = ig.Graph.from_edge_arrays(n, f, t, directed)
    f, t = g.edge_arrays()
    rng = np.random.default_rng(3)
    w = rng.uniform(0.0, 2.0, len(f)) * (rng.random(len(f)) < 0.9) if weighted else None
    ig.set_tuning("relabel", 0)
    try:
        with ig.DeviceGraph.from_host(n, f, t, directed, w) as dg:
            ref = dg.solve()[0]
            reset = rng.uniform(0, 1, n) ** 4
            ref_ppr = None if weighted else dg.solve(reset=reset)[0]
    finally:
        ig.reset_tuning()
    for _ in range(2):  # arrival order differs from run to run, the result must not
        got = ig.pagerank_weighted(g, w) if weighted else ig.pagerank(g)
        assert np.array_equal(got, ref)
        if not weighted:
            ppr = ig.personalized_pagerank(g, reset, 0.85)
            assert np.array_equal(ppr, ref_ppr)
    oracle = O.pagerank_weighted(n, f, t, directed, w) if weighted else O.pagerank(n, f, t, directed)
    assert np.abs(got - oracle).max() <= 1e-10


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("case", ["two", "gnm", "row_lengths", "long_hub", "powerlaw"])
def test_eigenvector_matches_the_general_path(cuda_ok, case, weighted):
    n, f, t = _graph(case)
    g = ig.Graph.from_edge_arrays(n, f, t, False)
    w = np.random.default_rng(8).uniform(0.5, 2.0, len(f)) if weighted else None
    got = []
    for resident in (1, 0):
        ig.set_tuning("resident", resident)
        try:
            got.append(ig.eigenvector_centrality_weighted(g, w, True) if weighted
                       else ig.eigenvector_centrality(g, True))
        finally:
            ig.reset_tuning()
    assert abs(got[0][1] - got[1][1]) <= 1e-10 * abs(got[1][1])
    assert np.abs(got[0][0] - got[1][0]).max() <= 1e-10


@pytest.mark.parametrize("directed", [True, False])
def test_out_of_range_endpoints_are_refused(cuda_ok, directed):
    import ctypes as C

    f, t = np.array([0, 1, 2], np.uint32), np.array([1, 7, 0], np.uint32)
    out = np.full(3, -1.0)
    rc = ig.lib().prg_pagerank(3, 3, f.ctypes.data_as(C.c_void_p), t.ctypes.data_as(C.c_void_p), int(directed),
                               out.ctypes.data_as(C.c_void_p))
    assert rc == 2 and "vertex id 7 out of range (vcount = 3)" in ig.last_error()
    assert (out == -1.0).all()


def test_refused_weights_name_the_first_edge(cuda_ok):
    # weights are checked before endpoints, the first refused edge is named
    n, f, t = _graph("gnm")
    g = ig.Graph.from_edge_arrays(n, f, t, True)
    for bad, text in ((-0.5, "-0.5"), (np.nan, "NaN"), (np.inf, "inf")):
        w = np.ones(len(f))
        w[[24_999, 777, 20_000]] = bad
        with pytest.raises(ig.InvalidArgument, match=f"weight at edge 777 must be non-negative and finite .got {text}."):
            ig.pagerank_weighted(g, w)
    w = np.ones(len(f))
    w[5] = -0.0
    assert np.isfinite(ig.pagerank_weighted(g, w)).all()
