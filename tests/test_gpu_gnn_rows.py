"""Message aggregation and its transpose at the edges of their row classes (no
arcs, around the 8 lanes of a row and the 32 arcs a round takes, around the 2048
arcs from which a block sums a row), few rows and more than a round of them,
against the float64 CPU restatement.

Tolerances are the network's (BF16 operands, 8 bits of mantissa, through three
layers): 2e-2 of the gradient's norm, 1e-2 in L1 on the prediction, with so few
rows of each class that a wrong row exceeds them.
"""
import numpy as np
import pytest

import igraph_b200 as ig
import gnn_oracle as GO
import oracle as O
from igraph_b200 import warmstart as W

pytestmark = pytest.mark.gpu

LENGTHS = {
    "short": [0, 1, 2, 3, 5, 7, 8, 9],
    "lanes": [15, 16, 17, 31, 32, 33, 0, 0, 0, 0, 63, 64, 65],
    "heavy": [2047, 2048, 2049, 0, 1, 2080, 5000, 255, 256, 257],
    "last_heavy": [4, 2049],
}


@pytest.mark.parametrize("kind", LENGTHS)
@pytest.mark.parametrize("relabel", [0, 1])
def test_row_classes(cuda_ok, kind, relabel):
    import torch

    lengths = LENGTHS[kind]
    n = len(lengths) + 3
    rng = np.random.default_rng(n)
    t = np.repeat(np.arange(len(lengths)), lengths).astype(np.uint32)
    f = rng.integers(0, n, len(t)).astype(np.uint32)
    p = rng.permutation(len(t))
    f, t = f[p], t[p]
    x = O.pagerank(n, f, t, True)
    net = W.WarmStartNet(seed=3)
    w = net.params()
    w += np.random.default_rng(1).normal(0, 0.05, w.shape).astype(np.float32)
    net.set_params(w)
    try:
        ig.set_tuning("relabel", relabel)
        with ig.DeviceGraph.from_host(n, f, t, True) as dg:
            target = torch.tensor(x, dtype=torch.float64, device="cuda")
            loss, g = net.loss_grad(dg, target.data_ptr())
            start = torch.empty(n, dtype=torch.float64, device="cuda")
            net.predict(dg, start.data_ptr())
    finally:
        ig.reset_tuning()
    l_ref, g_ref, pred_ref = GO.loss_and_grad(net.params(), n, f, t, True, x)
    assert abs(loss - l_ref) <= 1e-2 * abs(l_ref) + 1e-6
    assert np.linalg.norm(g - g_ref) <= 2e-2 * np.linalg.norm(g_ref)
    assert np.abs(start.cpu().numpy() - pred_ref).sum() <= 1e-2
    net.close()
