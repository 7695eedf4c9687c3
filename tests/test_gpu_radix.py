"""The radix passes of the CSR build (digits of at most 8 bits, spread evenly)
through the graphs they sort: key widths of every digit split and arc counts
around a tile of 4096 pairs, skewed and constant heads.  Integers, exact."""
import numpy as np
import pytest

import igraph_b200 as ig
from test_gpu_streamed_build import csr, device_arrays

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [1, 6, 7, 8, 9, 13, 14, 15, 16, 17, 21, 22, 24, 25])
@pytest.mark.parametrize("m", [2, 31, 4095, 4096, 4097, 5_000_001])
@pytest.mark.parametrize("kind", ["uniform", "skewed", "constant"])
def test_sorted_rows(cuda_ok, bits, m, kind):
    n = (1 << bits) - (1 if bits > 1 else 0)
    rng = np.random.default_rng(bits * m)
    t = rng.integers(0, n, m).astype(np.uint32)
    if kind == "skewed":
        t = (rng.random(m) ** 8 * n).astype(np.uint32)
    elif kind == "constant":
        t[:] = n - 1
    f = rng.integers(0, n, m).astype(np.uint32)
    df, dt, _ = device_arrays(f, t)
    try:
        ig.set_tuning("relabel", 0)
        with ig.DeviceGraph.from_device(n, m, df.data_ptr(), dt.data_ptr(), True) as dg:
            got = csr(dg)
    finally:
        ig.reset_tuning()
    assert np.array_equal(got["col"], f[np.argsort(t, kind="stable")])
    assert np.array_equal(got["row_ptr"], np.concatenate([[0], np.cumsum(np.bincount(t, minlength=n))]))
