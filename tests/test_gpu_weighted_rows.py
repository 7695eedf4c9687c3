"""Row sums of weighted graphs in the tile-segmented passes: each row's sum
comes from its own arcs, whatever its neighbours in a 256-arc tile hold.  Rows
of every length around the 8 arcs of a lane and the 256 of a tile, rows that
are tiny or zero beside large ones, rows beside an infinite or NaN product.
Power steps run with resident = 0 (the persistent iteration has no tiles);
HITS of a directed graph takes the passes at every size.

Tolerance of a row of L positive products: summed in any order it is off by at
most L ulp / 2 of the row, on either side, and a few ulp for the scaling
around it: (2 L + 30) x 1.2e-16, relative to the row.
"""
import numpy as np
import pytest

import igraph_b200 as ig
import oracle as O

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 2, 7, 8, 9, 15, 16, 17, 31, 33, 63, 64, 65, 255, 256, 257, 300, 1000, 5000]


def rows(n, seed):
    """(from, to): in-rows of the lengths above and of 0 to 60 arcs."""
    rng = np.random.default_rng(seed)
    lens = np.concatenate([LENGTHS, rng.integers(0, 61, n - len(LENGTHS))])
    rng.shuffle(lens)
    t = np.repeat(np.arange(n), lens)
    return rng.integers(0, n, len(t)).astype(np.uint32), t.astype(np.uint32), lens


def tolerance(lens):
    return (2 * lens + 30) * 1.2e-16


@pytest.mark.parametrize("relabel", [0, 1])
@pytest.mark.parametrize("spread", [0, 12, 17, 40])  # decimal orders between a tile's rows
def test_power_step_rows_keep_their_digits(cuda_ok, spread, relabel):
    n = 3000
    f, t, lens = rows(n, 1)
    rng = np.random.default_rng(2)
    w = (rng.random(len(f)) + 0.5) * 10.0 ** (-spread * (t % 3).astype(float) / 2.0)
    reset = np.where(np.arange(n) % 2 == 0, rng.random(n) + 0.5, 0.0)
    try:
        ig.set_tuning("resident", 0)
        ig.set_tuning("relabel", relabel)
        with ig.DeviceGraph.from_host(n, f, t, True, w) as dg:
            x, _ = dg.solve(ig.Options(max_iter=1), reset=reset)
    finally:
        ig.reset_tuning()
    tele = reset / reset.sum()
    out = np.bincount(f, weights=w, minlength=n)
    lost = tele[out == 0].sum()
    xt = np.divide(tele, out, out=np.zeros(n), where=out > 0)
    y = np.zeros(n)
    np.add.at(y, t, w * xt[f])
    ref = 0.15 * tele + 0.85 * (y + lost * tele)
    odd = tele == 0.0  # there the result is the row's sum alone
    assert (ref[odd] > 0).sum() > 1000
    assert np.array_equal(x[odd] == 0, ref[odd] == 0)
    rel = np.abs(x - ref) / np.where(ref > 0, ref, 1.0)
    assert (rel <= tolerance(lens)).all()


@pytest.mark.parametrize("precision", [ig.PRECISION_FP64, ig.PRECISION_FP64_KRYLOV, ig.PRECISION_FP32_REFINED])
@pytest.mark.parametrize("relabel", [0, 1])
def test_vertices_the_seeds_cannot_reach_are_exactly_zero(cuda_ok, precision, relabel):
    # even vertices hold the seeds, odd ones only have arcs among themselves; ids interleave, so tiles mix them
    half, m = 2000, 60_000
    rng = np.random.default_rng(3)
    f = np.concatenate([2 * rng.integers(0, half, m), 2 * rng.integers(0, half, m) + 1])
    t = np.concatenate([2 * rng.integers(0, half, m), 2 * rng.integers(0, half, m) + 1])
    w = rng.random(2 * m) + 0.1
    reset = np.zeros(2 * half)
    reset[:20:2] = 1.0
    try:
        ig.set_tuning("resident", 0)
        ig.set_tuning("relabel", relabel)
        with ig.DeviceGraph.from_host(2 * half, f.astype(np.uint32), t.astype(np.uint32), True, w) as dg:
            x, _ = dg.solve(ig.Options(precision=precision), reset=reset)
    finally:
        ig.reset_tuning()
    assert (x[1::2] == 0).all() and x[::2].min() > 0
    assert abs(x.sum() - 1) <= 1e-9


@pytest.mark.parametrize("spread", [12, 17, 40])
@pytest.mark.parametrize("reverse", [False, True])
def test_hits_rows_keep_their_digits(cuda_ok, spread, reverse):
    # authority is one product A^T hub scaled by its maximum
    n = 3000
    f, t, lens = rows(n, 5)
    rng = np.random.default_rng(6)
    w = (rng.random(len(f)) + 0.5) * 10.0 ** (-spread * (t % 3).astype(float) / 2.0)
    if reverse:  # tiny rows in both directions
        w *= 10.0 ** (-spread * (f % 2).astype(float))
    r = ig.hub_and_authority_scores_weighted(ig.Graph.from_edge_arrays(n, f, t, True), w)
    y = np.zeros(n)
    np.add.at(y, t, w * r.hub[f])
    ref = y / y.max()
    assert np.array_equal(r.authority == 0, ref == 0)
    rel = np.abs(r.authority - ref) / np.where(ref > 0, ref, 1.0)
    assert (rel <= tolerance(lens) + tolerance(lens.max())).all()  # (its own row's error and the maximum's)


def two_components(odd):
    """Directed, ids interleaved; the even component holds the odd weights."""
    half, m = 2000, 40_000
    rng = np.random.default_rng(7)
    f = np.concatenate([2 * rng.integers(0, half, m), 2 * rng.integers(0, half, m) + 1]).astype(np.uint32)
    t = np.concatenate([2 * rng.integers(0, half, m), 2 * rng.integers(0, half, m) + 1]).astype(np.uint32)
    w = rng.random(2 * m) + 0.5
    w[: 40 if odd == 1e308 else 1] = odd
    return 2 * half, f, t, w


def same_where_finite(got, ref):
    bad = ~np.isfinite(ref)
    assert bad.any() and not bad.all()
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    assert np.abs(got[~bad] - ref[~bad]).max() <= 1e-10


@pytest.mark.parametrize("odd", [np.inf, np.nan, 1e308])
def test_hits_beside_weights_beyond_the_finite_range(cuda_ok, odd):
    n, f, t, w = two_components(odd)
    r = ig.hub_and_authority_scores_weighted(ig.Graph.from_edge_arrays(n, f, t, True), w)
    hub, auth, _, _ = O.hub_and_authority_scores_weighted(n, f, t, w, True)
    same_where_finite(r.hub, hub)
    same_where_finite(r.authority, auth)


@pytest.mark.parametrize("resident", [0, 1])
@pytest.mark.parametrize("odd", [np.inf, np.nan, 1e308])
def test_eigenvector_beside_weights_beyond_the_finite_range(cuda_ok, odd, resident):
    n, f, t, w = two_components(odd)
    lo, hi = np.minimum(f, t), np.maximum(f, t)
    try:
        ig.set_tuning("resident", resident)
        x = ig.eigenvector_centrality_weighted(ig.Graph.from_edge_arrays(n, lo, hi, False), w)
    finally:
        ig.reset_tuning()
    ref = O.eigenvector_centrality_weighted(n, lo, hi, w)[0]
    same_where_finite(x, ref)
