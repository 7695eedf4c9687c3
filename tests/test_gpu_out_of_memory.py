"""Calls that run out of device memory: the error is reported, what was
allocated is given back, and the next call works.  The free memory is cut down
to a few hundred MB, in steps, so that every large allocation of a call is the
one that fails at some step.

What may stay allocated is bounded by the vectors of a vertex set of 3000 (24 KB
each), 1 MB; the arrays in question are 4 to 16 bytes an edge, 30 MB and more.
"""
import numpy as np
import pytest

import igraph_b200 as ig

pytestmark = pytest.mark.gpu

MB = 1 << 20


class Pool:
    """The device's default memory pool, which the library allocates from."""

    def __init__(self):
        from cuda.bindings import runtime as rt

        self.rt = rt
        err, self.pool = rt.cudaDeviceGetDefaultMemPool(0)
        assert err == rt.cudaError_t.cudaSuccess

    def used(self):
        err, v = self.rt.cudaMemPoolGetAttribute(self.pool, self.rt.cudaMemPoolAttr.cudaMemPoolAttrUsedMemCurrent)
        assert err == self.rt.cudaError_t.cudaSuccess
        return int(v)

    def trim(self):
        self.rt.cudaDeviceSynchronize()
        (err,) = self.rt.cudaMemPoolTrimTo(self.pool, 0)
        assert err == self.rt.cudaError_t.cudaSuccess


def with_free_memory(pool, size, call):
    """The call with about `size` bytes of device memory free: its result, or None when that was too little."""
    import torch

    pool.trim()
    torch.cuda.empty_cache()
    hog = torch.empty(max(torch.cuda.mem_get_info()[0] - size, 0), dtype=torch.uint8, device="cuda")
    try:
        return call()
    except ig.IgraphError as e:
        assert "memory" in str(e)
        return None
    finally:
        del hog
        torch.cuda.empty_cache()


@pytest.mark.parametrize("weighted,m", [(False, 8_000_000), (False, 9_000_000), (True, 4_000_000)])
def test_hits_gives_back_what_it_allocated(cuda_ok, weighted, m):
    n = 3000
    rng = np.random.default_rng(m)
    f, t = rng.integers(0, n, m).astype(np.uint32), rng.integers(0, n, m).astype(np.uint32)
    w = rng.random(m) + 0.5
    g = ig.Graph.from_edge_arrays(n, f, t, True)
    call = (lambda: ig.hub_and_authority_scores_weighted(g, w)) if weighted else (lambda: ig.hub_and_authority_scores(g))
    ref = call()
    pool = Pool()
    before = pool.used()
    outcomes = []
    for size in range(32 * MB, 512 * MB, 8 * MB):
        r = with_free_memory(pool, size, call)
        outcomes.append(r is not None)
        assert pool.used() - before <= MB, f"{(pool.used() - before) / MB:.0f} MB kept with {size // MB} MB free"
        if r is not None:
            assert np.array_equal(r.hub, ref.hub)
            break
    assert outcomes[-1] and outcomes.count(False) >= 5


def test_drop_in_goes_where_there_is_room(cuda_ok):
    # 8-bit ids: the general build sorts in one pass and takes less memory than the small-graph path
    n, m = 200, 8_000_000
    rng = np.random.default_rng(m)
    f, t = rng.integers(0, n, m).astype(np.uint32), rng.integers(0, n, m).astype(np.uint32)
    g = ig.Graph.from_edge_arrays(n, f, t, True)
    ref = ig.pagerank(g)
    pool = Pool()
    before = pool.used()
    outcomes = []
    for size in range(96 * MB, 320 * MB, 8 * MB):
        try:
            ig.set_tuning("resident", 0)
            general = with_free_memory(pool, size, lambda: ig.pagerank(g))
        finally:
            ig.reset_tuning()
        x = with_free_memory(pool, size, lambda: ig.pagerank(g))
        outcomes.append((general is not None, x is not None))
        assert pool.used() - before <= MB
        assert x is None or np.abs(x - ref).max() <= 1e-10
    assert (False, False) in outcomes and (True, True) in outcomes
    assert (True, False) not in outcomes
