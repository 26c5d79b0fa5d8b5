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


def test_crowded_cells_are_searched_by_bisection(ctx_factory):
    """A trained peak puts most edges, and so most points, into few cells.  The
    search among a cell's edges takes a logarithm of their number: with all
    1000 edges in one cell a coordinate between them costs at most six times
    one on equidistant edges (read one after the other: 44 times)."""
    import ctypes as C

    import torch

    bins, n = 1000, 1 << 20
    rng = np.random.default_rng(4)
    crowded = np.concatenate([[0.0], np.sort(0.3 + 1e-5 * rng.random(bins - 1)), [1.0]])
    x = torch.from_numpy(0.3 + 1e-5 * rng.random((n, 4))).cuda()
    w = torch.empty(n, dtype=torch.float64, device="cuda")
    times = []
    stream = torch.cuda.Stream()
    for row in (np.linspace(0, 1, bins + 1), crowded):
        ctx = ctx_factory()
        ctx.set_stream(stream.cuda_stream)
        ctx.set_grids(np.tile(row, (1, 4, 1)))
        span = x if row is crowded else torch.from_numpy(rng.random((n, 4))).cuda()
        torch.cuda.synchronize()
        best = np.inf
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            ctx.call("chili_gpu_grid_weight", 0, C.c_void_p(span.data_ptr()), C.c_void_p(w.data_ptr()), None, n)
            b.record(stream)
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        times.append(best)
    assert times[1] <= 6 * times[0], times
