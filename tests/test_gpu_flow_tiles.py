"""Coupling-layer kernels over several tiles per CTA: a point's result does not
depend on the tile, the pass or the call that carries it."""
import numpy as np
import pytest

from chili_b200 import abi, channels, flowspec, workloads
from oracle import flow as F

pytestmark = pytest.mark.gpu


def _context(ctx_factory, rng, n_out, batch):
    cs = workloads.channel_set(n_out)
    ctx = ctx_factory()
    ctx.set_channels(cs)
    ctx.uniform_grids(cs.nch, ctx.ndims, 50)
    ctx.set_integrand(abi.CHILI_FUNC_PROPAGATOR, channels.propagator_params())
    ctx.set_preprocess(abi.CHILI_PRE_FINITE)
    ctx.set_alpha(np.full(cs.nch, 1.0 / cs.nch))
    ctx.flow_init(abi.FlowParams.defaults(batch=batch))
    lay = flowspec.layout(ctx.ndims, cs.nch, cs.n_ext)
    p = flowspec.unflatten(ctx.flow_get_params(), lay)
    for k in p:
        if k.startswith("W3") or k.startswith("E") or k in ("A3", "c3", "c1", "c2"):
            p[k] = p[k] + rng.normal(0, 0.05, p[k].shape)
    flat = flowspec.flatten(p, lay)
    ctx.flow_set_params(flat)
    return ctx, cs, flowspec.unflatten(flat, lay), lay


@pytest.mark.parametrize("n", [1, 128, 129, 128 * 148, 128 * 148 * 2 + 77])
def test_points_do_not_depend_on_their_tile(ctx_factory, n):
    """One call against calls of 97 points (one tile each): bit for bit."""
    rng = np.random.default_rng(n)
    ctx, cs, _, _ = _context(ctx_factory, rng, 4, 40_000)
    u = rng.random((n, ctx.ndims)).astype(np.float32)
    ch = rng.integers(0, cs.nch, n)
    some = np.unique(np.concatenate([np.arange(min(n, 97)), rng.integers(0, n, 97), np.arange(max(0, n - 97), n)]))
    for fn in (ctx.flow_density, ctx.flow_sample_u):
        y, lq = fn(u, ch)
        for part in np.array_split(some, max(1, len(some) // 97)):
            yp, lp = fn(u[part], ch[part])
            assert np.array_equal(yp, y[part]) and np.array_equal(lp, lq[part])


@pytest.mark.parametrize("n", [129, 128 * 148 + 77])
def test_gradients_over_tiles(ctx_factory, n):
    """Against the oracle with its operands rounded to bf16: the bounds of the
    one-tile-per-CTA gradient test (loss 2e-4, a parameter block 4e-3 seen,
    1e-2 allowed: f32 order of summation and the spline's f32 arithmetic)."""
    rng = np.random.default_rng(n)
    ctx, cs, p, lay = _context(ctx_factory, rng, 4, 20_480)
    beta = rng.dirichlet(np.ones(cs.nch) * 5)
    ctx.flow_set_beta(beta)
    nfeat = flowspec.n_features(cs.n_ext)
    spec = F.Spec(ctx.ndims, cs.nch, nfeat)
    f = lambda a: a.astype(np.float32).astype(np.float64)
    batch = dict(u=f(rng.random((n, ctx.ndims))), ch=rng.integers(0, cs.nch, n), logf=f(rng.normal(0, 0.7, n)),
                 logbeta=f(np.log(beta)), feat=f(rng.uniform(-1, 1, (n, nfeat))),
                 logprior=f(np.log(1 / cs.nch) + rng.normal(0, 1, (n, cs.nch))))
    loss, grad = ctx.flow_loss_grad(batch["u"], batch["ch"], batch["logf"], batch["feat"], batch["logprior"])
    Lo, go, _ = F.loss_and_grads(spec, p, batch, use_bf16=True)
    assert abs(loss - Lo) <= 2e-4 * Lo
    g = flowspec.unflatten(grad, lay)
    for k in go:
        assert np.linalg.norm(g[k] - go[k]) <= 1e-2 * np.linalg.norm(go[k]) + 1e-6, k
