"""Plain VEGAS: the iteration's bins on grids the staged edges shortcut and on
grids they must not, and materialised points on buffers of every alignment."""
import numpy as np
import pytest

from chili_b200 import abi, workloads
from oracle import port

pytestmark = pytest.mark.gpu


def lower_bound_bins(edges, x):
    return np.stack([np.where(np.isnan(x[:, d]), -1, np.searchsorted(edges[d, :-1], x[:, d], side="left") - 1)
                     for d in range(x.shape[1])], 1)


def fold(idx, val2, dims, bins):
    """Slot d * bins + FindBin of every dimension (Vegas.cc:30-33): FindBin = -1
    is the previous dimension's last slot, and none before the first."""
    slot = idx + bins * np.arange(dims)
    ok = slot >= 0
    return np.bincount(slot[ok], weights=np.broadcast_to(val2[:, None], slot.shape)[ok],
                       minlength=dims * bins).reshape(dims, bins)


@pytest.mark.parametrize("fused", [1, 0])
@pytest.mark.parametrize("dims,bins", [(1, 2), (4, 50), (5, 700), (6, 497), (6, 512), (16, 181), (9, 300)])
def test_iteration_bins(ctx_factory, dims, bins, fused):
    """Histogram of f^2 over FindBin of the mapped points.  Sizes on both sides
    of the 48 KB that histogram and edges share ((5, 700) stages 56 KB: not;
    (6, 497) 47.8 KB: yes; (6, 512) 49.2 KB: not; (16, 181) 46.5 KB).
    Uniforms on bin boundaries give points exactly on edges."""
    rng = np.random.default_rng(dims * 1000 + bins)
    inner = np.sort(rng.random((dims, bins - 1)), axis=1)
    inner[0] = np.sort(np.repeat(inner[0], 2)[:bins - 1])  # zero-width bins
    edges = np.concatenate([np.zeros((dims, 1)), inner, np.ones((dims, 1))], 1)
    u = rng.random((4000, dims))
    u[:bins] = (np.arange(bins) / bins)[:, None]
    u[-1] = 0.0
    p = np.array(workloads.camel_params(dims))
    ctx = ctx_factory()
    ctx.set_option("vegas_fused", fused)
    ctx.set_integrand(abi.CHILI_FUNC_CAMEL, p)
    ctx.set_grids(edges[None])
    x, jac = ctx.grid_map(0, u)
    a, b = p[2:2 + dims], p[2 + dims:2 + 2 * dims]
    s2 = p[0] * p[0]
    f = p[1] * (np.exp(-((x - a) ** 2).sum(1) / s2) + np.exp(-((x - b) ** 2).sum(1) / s2))
    val2 = (f * jac) ** 2
    idx = lower_bound_bins(edges, x)
    want = fold(idx, val2, dims, bins)
    st, tr = ctx.vegas_iterate(len(u), u=u, alpha=1.5, adapt=True, train=True)
    got = tr.reshape(dims, bins)
    # exponents of at most 711 to 18 roundings: 711 * 18 * 2.2e-16 = 3e-12, twice in f^2
    assert np.all(np.abs(got - want) <= 1e-11 * want)
    assert abs(st.sum - (f * jac).sum()) <= 1e-11 * st.sum and st.n == len(u)


def test_iteration_on_unordered_edges(ctx_factory):
    """Edges out of order: the bins of the binary search as it walks them
    (every training slot equals the separate search's, f^2 summed)."""
    dims, bins, n = 4, 50, 3000
    rng = np.random.default_rng(3)
    edges = np.tile(np.linspace(0, 1, bins + 1), (dims, 1))
    edges[0, 10:20] = edges[0, 10:20][::-1].copy()
    edges[2, 25] = 0.9
    u = rng.random((n, dims))
    p = np.array(workloads.camel_params(dims))
    ctx = ctx_factory()
    ctx.set_integrand(abi.CHILI_FUNC_CAMEL, p)
    ctx.set_grids(edges[None])
    x, jac = ctx.grid_map(0, u)
    _, idx = ctx.grid_weight(0, x)
    a, b = p[2:2 + dims], p[2 + dims:2 + 2 * dims]
    f = p[1] * (np.exp(-((x - a) ** 2).sum(1) / p[0] ** 2) + np.exp(-((x - b) ** 2).sum(1) / p[0] ** 2))
    _, tr = ctx.vegas_iterate(n, u=u, alpha=1.5, adapt=False, train=True)
    want = fold(idx, (f * jac) ** 2, dims, bins)
    assert np.all(np.abs(tr.reshape(dims, bins) - want) <= 1e-11 * want)


@pytest.mark.parametrize("ppt", [1, 2, 4])
@pytest.mark.parametrize("dims", [2, 3, 4, 6, 8, 16])
def test_points_at_every_alignment(ctx_factory, dims, ppt):
    """x and w of an n that ends inside a tile, written 0 to 3 doubles past a
    32-byte boundary: the uniforms' points bit for bit, nothing beside them."""
    import torch
    bins, n, seed, ctr = 40, 1291, 9, 5
    rng = np.random.default_rng(dims)
    edges = np.concatenate([np.zeros((dims, 1)), np.sort(rng.random((dims, bins - 1)), axis=1), np.ones((dims, 1))], 1)
    ctx = ctx_factory()
    ctx.set_option("vegas_gen_ppt", ppt)
    ctx.set_integrand(abi.CHILI_FUNC_CAMEL, workloads.camel_params(dims))
    ctx.set_grids(edges[None])
    x0, jac = ctx.grid_map(0, port.philox_uniforms(seed, ctr, n, dims))
    w0 = None
    for off in range(4):
        buf = torch.full((n * dims + 8,), -7.0, dtype=torch.float64, device="cuda")
        wb = torch.full((n + 8,), -7.0, dtype=torch.float64, device="cuda")
        x, w = buf[off:off + n * dims], wb[off:off + n]
        torch.cuda.synchronize()
        ctx.vegas_generate(n, seed=seed, counter=ctr, out=(x, w))
        ctx.synchronize()
        assert np.array_equal(x.cpu().numpy().reshape(n, dims), x0)
        w0 = w.cpu().numpy() if w0 is None else w0
        assert np.array_equal(w.cpu().numpy(), w0)
        assert (buf[:off] == -7).all() and (buf[off + n * dims:] == -7).all() and (wb[off + n:] == -7).all()
