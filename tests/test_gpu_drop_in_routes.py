"""Which way a drop-in or a solve goes, seen in the kernels it launches and the
bytes it uploads: a drop-in that the small-graph path cannot serve must cost
what the general path costs, and give its result to the bit; a graph whose
longest row would hold up one block does not iterate in the persistent kernel."""
import json

import numpy as np
import pytest

import igraph_b200 as ig
import oracle as O

pytestmark = pytest.mark.gpu


def traced(call, path):
    """(result, kernel names, bytes copied host to device)"""
    from torch.profiler import ProfilerActivity, profile

    with profile(activities=[ProfilerActivity.CUDA]) as p:
        out = call()
    p.export_chrome_trace(path)
    with open(path) as fh:
        events = json.load(fh)["traceEvents"]
    names = [e["name"] for e in events if e.get("cat") == "kernel"]
    up = sum(e["args"]["bytes"] for e in events if e.get("cat") == "gpu_memcpy" and "HtoD" in e["name"])
    assert names, "the profiler saw no kernels"
    return out, names, up


def both(call, tmp_path):
    """The call as it goes by default and over the general path alone."""
    ig.pagerank(ig.Graph.from_edge_arrays(2, np.zeros(1, np.uint32), np.ones(1, np.uint32), True))  # context, kernels
    got = traced(call, str(tmp_path / "default.json"))
    try:
        ig.set_tuning("resident", 0)
        general = traced(call, str(tmp_path / "general.json"))
    finally:
        ig.reset_tuning()
    return got, general


CALLS = {
    "pagerank": lambda g, w: ig.pagerank(g),
    "weighted": lambda g, w: ig.pagerank_weighted(g, w),
    "eigenvector": lambda g, w: ig.eigenvector_centrality(g),
    "eigenvector_weighted": lambda g, w: ig.eigenvector_centrality_weighted(g, w),
}


@pytest.mark.parametrize("kind,n,m", [("pagerank", 3_000_000, 1_000_000), ("pagerank", 2_450_000, 6_000_000),
                                      ("weighted", 3_000_000, 1_000_000), ("eigenvector", 1_400_000, 300_000),
                                      ("eigenvector_weighted", 1_400_000, 300_000)])
def test_many_vertices_are_refused_before_any_copy(cuda_ok, kind, n, m, tmp_path):
    rng = np.random.default_rng(n)
    f, t = rng.integers(0, n, m).astype(np.uint32), rng.integers(0, n, m).astype(np.uint32)
    directed = not kind.startswith("eigen")
    if not directed:
        f, t = np.minimum(f, t), np.maximum(f, t)
    g, w = ig.Graph.from_edge_arrays(n, f, t, directed), rng.random(m) + 0.5
    (x, names, up), (ref, _, ref_up) = both(lambda: CALLS[kind](g, w), tmp_path)
    assert not any("small_build_kernel" in k or "res_kernel" in k for k in names)
    assert up == ref_up
    assert np.array_equal(x, ref)


def hub_graph(n, m, longest):
    """Directed: one in-row of `longest` arcs, the others short."""
    rng = np.random.default_rng(longest)
    t = np.concatenate([np.full(longest, n // 3), rng.integers(0, n, m - longest)]).astype(np.uint32)
    rng.shuffle(t)
    return rng.integers(0, n, m).astype(np.uint32), t


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("longest,resident", [(30_000, True), (60_000, True), (90_000, False), (200_000, False)])
def test_long_rows_do_not_hold_up_one_block(cuda_ok, longest, resident, weighted, tmp_path):
    n, m = 60_000, 600_000  # 4 K arcs to a block
    f, t = hub_graph(n, m, longest)
    w = np.random.default_rng(1).random(m) + 0.5 if weighted else None
    with ig.DeviceGraph.from_host(n, f, t, True, w) as dg:
        dg.solve()
        (x, _), names, _ = traced(dg.solve, str(tmp_path / "solve.json"))
    assert any("res_kernel" in k for k in names) == resident and any("seg8_kernel" in k for k in names) != resident
    ref = O.pagerank_weighted(n, f, t, True, w) if weighted else O.pagerank(n, f, t, True)
    assert np.abs(x - ref).max() <= 1e-10  # the stop rule's tolerance
    lo, hi = np.minimum(f, t), np.maximum(f, t)
    g = ig.Graph.from_edge_arrays(n, lo, hi, False)
    call = "eigenvector_weighted" if weighted else "eigenvector"
    _, names, _ = traced(lambda: CALLS[call](g, w), str(tmp_path / "eigen.json"))
    assert any("seg8_kernel" in k for k in names) != resident


LONG = [(100_000, 99_000), (600_000, 90_000), (1_500_000, 700_000)]


@pytest.mark.parametrize("kind,m,longest", [(k, *r) for k in CALLS for r in LONG] + [("pagerank", 9_000_000, 400_000)])
def test_long_rows_upload_once(cuda_ok, kind, m, longest, tmp_path):
    # rows no plan holds, found in the build (or, with few edges a thread, by the plan)
    n = 60_000
    f, t = hub_graph(n, m, longest)
    directed = not kind.startswith("eigen")
    if not directed:
        f, t = np.minimum(f, t), np.maximum(f, t)
    g, w = ig.Graph.from_edge_arrays(n, f, t, directed), np.random.default_rng(2).random(m) + 0.5
    (x, names, up), (ref, _, ref_up) = both(lambda: CALLS[kind](g, w), tmp_path)
    assert any("small_build_kernel" in k for k in names)
    assert up == ref_up
    assert np.array_equal(x, ref)


def test_long_rows_report_what_is_wrong_with_the_input(cuda_ok):
    # the build ends early, the errors are the general path's
    n, m = 60_000, 1_500_000
    f, t = hub_graph(n, m, 700_000)
    w = np.ones(m)
    w[m - 1] = -1.0
    g = ig.Graph.from_edge_arrays(n, f, t, True)
    with pytest.raises(ig.InvalidArgument, match=f"weight at edge {m - 1} must be non-negative"):
        ig.pagerank_weighted(g, w)
    t[m - 1] = n
    with pytest.raises(Exception, match=f"vertex id {n} out of range"):
        ig._check(ig.lib().prg_pagerank(n, m, ig._ptr(f), ig._ptr(t), 1, ig._ptr(np.empty(n))))
