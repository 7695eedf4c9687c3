"""Rows without arcs on relabelled directed graphs, which the segmented FP64
kernels take between their tiles: no such rows, a few, most; fewer tiles than
warps and many rounds of tiles; unweighted and weighted.  Against the row-block
kernels, and at the smaller sizes the oracle.

Tolerance: both run the same FP64 power steps to the same stop, so entries
differ by the rounding of differently ordered sums: at most ~100 steps times a
few ulp (2e-16) each, 1e-12 relative with room for long rows.
"""
import numpy as np
import pytest

import igraph_b200 as ig
import oracle as O

pytestmark = pytest.mark.gpu


def solve(n, f, t, w, seg, opts):
    try:
        for k, v in (("relabel", 1), ("resident", 0), ("seg_plain64", seg), ("seg_res64", seg)):
            ig.set_tuning(k, v)
        with ig.DeviceGraph.from_host(n, f, t, True, w) as dg:
            assert dg.relabelled
            return dg.solve(opts)
    finally:
        ig.reset_tuning()


@pytest.mark.parametrize("n,m", [(40, 60), (5000, 300), (5000, 40_000), (300_000, 20_000), (200_000, 3_000_000)])
@pytest.mark.parametrize("heads", [1.0, 0.9, 0.05])  # share of the vertices that have in-arcs
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("linsys", [False, True])
def test_rows_without_arcs(cuda_ok, n, m, heads, weighted, linsys):
    rng = np.random.default_rng(n + m)
    f = (rng.random(m) ** 2 * n).astype(np.uint32)
    t = rng.integers(0, max(int(n * heads), 1), m).astype(np.uint32)
    w = rng.random(m) + 0.25 if weighted else None
    opts = ig.Options(precision=ig.PRECISION_LINSYS) if linsys else ig.Options()
    a, sa = solve(n, f, t, w, 1, opts)
    b, sb = solve(n, f, t, w, 0, opts)
    tol = 1e-9 if linsys else 1e-12  # (the linear solver stops on a bound of its error, not after equal steps)
    if not linsys:
        assert sa.iterations == sb.iterations
    assert np.abs(a / b - 1).max() <= tol
    if n <= 5000 and not linsys:
        ref = O.pagerank_weighted(n, f, t, True, w) if weighted else O.pagerank(n, f, t, True)
        assert np.abs(a - ref).sum() <= 1e-9
