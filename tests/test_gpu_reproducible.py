"""Krylov solves give the same bits every time.  Every reduction is a fixed
tree and every decision is taken from the same records by all blocks, so a
difference between runs means that some block read what another one of the
same launch had already changed: the FP64 vector kernels have more blocks than
fit on the chip at once, and near their precision limit the solves count steps
without progress."""
import numpy as np
import pytest

import igraph_b200 as ig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [ig.PRECISION_LINSYS, ig.PRECISION_FP64_KRYLOV, ig.PRECISION_FP32_REFINED])
@pytest.mark.parametrize("n,m", [(3000, 20_000), (1_300_000, 3_000_000), (1_300_000, 6_000_000)])
@pytest.mark.parametrize("relabel", [0, 1])
def test_krylov_solves_repeat(cuda_ok, n, m, relabel, precision):
    rng = np.random.default_rng(m)
    f = (n * rng.random(m) ** 3).astype(np.uint32)
    t = rng.integers(0, n, m).astype(np.uint32)
    opts = ig.Options(precision=precision)
    try:
        ig.set_tuning("relabel", relabel)
        with ig.DeviceGraph.from_host(n, f, t, True) as dg:
            first, st = dg.solve(opts)
            for _ in range(8):
                x, again = dg.solve(opts)
                assert again.iterations == st.iterations
                assert np.array_equal(x, first)
    finally:
        ig.reset_tuning()
