"""Per-call pinned slabs and streams are reused between calls: concurrent
one-call drop-ins and handles from several threads, more of them than the
pool keeps, give the results of a single call."""
import threading

import numpy as np
import pytest

import igraph_b200 as ig
import oracle as O

pytestmark = pytest.mark.gpu


def test_concurrent_calls_share_no_state(cuda_ok):
    n = 600
    f, t = O.erdos_renyi_gnm(n, 4000, True, False, 3)
    graphs, refs = [], []
    for k in range(4):
        m = 1500 + 600 * k
        graphs.append(ig.Graph.from_edge_arrays(n, f[:m], t[:m], True))
        refs.append(O.pagerank(n, f[:m], t[:m], True))
    errors = []

    def work(k):
        try:
            for _ in range(6):
                assert np.abs(ig.pagerank(graphs[k % 4]) - refs[k % 4]).max() <= 1e-10
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(12)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not errors, errors


def test_more_handles_than_the_pool_keeps(cuda_ok):
    n = 400
    f, t = O.erdos_renyi_gnm(n, 2500, True, False, 8)
    ref = O.pagerank(n, f, t, True)
    opts = ig.Options(precision=ig.PRECISION_FP64_KRYLOV)
    handles = [ig.DeviceGraph.from_host(n, f, t, True) for _ in range(40)]  # 80 slabs, 40 streams
    for dg in handles:
        assert np.abs(dg.solve()[0] - ref).max() <= 1e-10
        assert np.abs(dg.solve(opts)[0] - ref).sum() <= 1e-9
    for dg in handles:
        dg.close()
    with ig.DeviceGraph.from_host(n, f, t, True) as dg:
        assert np.abs(dg.solve()[0] - ref).max() <= 1e-10
