"""FindBin through the cell tables (AdaptiveMap.cc:34-38): the bins of a plain
lower_bound for every table size around the entry formats' limits, on grids
with many edges per cell, and at coordinates on and beside every edge."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def lower_bound_bins(edges, x):
    """FindBin of x on each dimension's edges[:-1]; NaN compares false."""
    return np.stack([np.where(np.isnan(x[:, d]), -1, np.searchsorted(edges[d, :-1], x[:, d], side="left") - 1)
                     for d in range(x.shape[1])], 1)


@pytest.mark.parametrize("bins", [2, 7, 253, 254, 255, 1000, 4094, 4095, 4096])
def test_bins_match_lower_bound(ctx_factory, bins):
    rng = np.random.default_rng(bins)
    inner = np.sort(rng.random((4, bins - 1)), axis=1)
    inner[1] = np.sort(0.3 + 1e-5 * rng.random(bins - 1))          # all edges in one cell
    inner[2] = np.sort(np.repeat(inner[2], 2)[:bins - 1])           # repeated edges
    inner[3] = np.sort(rng.random(bins - 1) ** 8)                   # peaked at 0
    edges = np.concatenate([np.zeros((4, 1)), inner, np.ones((4, 1))], 1)
    on = edges.T
    x = np.concatenate([on, np.nextafter(on, 2), np.nextafter(on, -1), rng.random((5000, 4)) ** 3,
                        np.array([[-0.5] * 4, [1.5] * 4, [np.nan] * 4, [np.inf] * 4, [-0.0] * 4])])
    ctx = ctx_factory()
    ctx.set_grids(edges[None])
    w, b = ctx.grid_weight(0, x)
    want = lower_bound_bins(edges, x)
    assert np.array_equal(b, want)
    ok = (want >= 0).all(1)
    width = np.stack([np.diff(edges[d])[want[ok, d]] for d in range(4)], 1)
    jac = np.ones(ok.sum())
    for d in range(4):
        jac = jac * (width[:, d] * float(bins))
    assert np.array_equal(w[ok], jac)
