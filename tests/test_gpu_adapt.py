"""Adaptation kernels at the sizes where their split can go wrong: rows around
a block and at the limits (AdaptiveMap.cc:67-125), channel counts around the
warp sums' groups of eight and the block (MultiChannel.cc:109-154)."""
import numpy as np
import pytest

from chili_b200 import abi, channels, workloads
from oracle import port

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,bins", [(1, 2), (3, 3), (2, 127), (2, 128), (5, 129), (1, 4096)])
def test_rebinning(ctx_factory, dims, bins):
    rng = np.random.default_rng(bins)
    inner = np.sort(rng.random((dims, bins - 1)), axis=1)
    edges = np.concatenate([np.zeros((dims, 1)), inner, np.ones((dims, 1))], 1)
    train = rng.random(dims * bins) ** 6 * 1e-30
    train[::7] = 0.0
    train[0] = 1e-30
    ctx = ctx_factory()
    ctx.set_grids(edges[None])
    ctx.grid_adapt(0, 1.5, train)
    got, want = ctx.get_grids()[0], port.am_adapt(edges, 1.5, train)
    # pow and log round differently on the two sides: ulps of the factors,
    # summed over at most `bins` of them
    assert np.max(np.abs(got - want)) <= 1e-15 * bins


@pytest.mark.parametrize("n_out", [2, 3, 4, 6])
def test_training_of_every_channel_count(ctx_factory, n_out):
    """alpha and best weights of 2, 6, 15 and 45 channels from given sums."""
    cs = workloads.channel_set(n_out)
    ctx = ctx_factory()
    ctx.set_channels(cs)
    ctx.uniform_grids(cs.nch, ctx.ndims, 8)
    ctx.set_integrand(abi.CHILI_FUNC_PROPAGATOR, channels.propagator_params())
    rng = np.random.default_rng(n_out)
    alpha = rng.random(cs.nch) + 0.05
    alpha /= alpha.sum()
    ctx.set_alpha(alpha)
    train = rng.random(cs.nch) * 10.0 ** rng.integers(-40, -20, cs.nch)
    train[-1] = 0.0
    p = workloads.mc_params(1000)
    ctx.multichannel_train(p, np.zeros((cs.nch, ctx.ndims, 8)), train)
    a, best, diff = ctx.get_alpha()
    w = alpha * train ** p.beta
    w = np.where(w == 0, 0.0, np.maximum(w / w.sum(), p.min_alpha))
    want = w / w.sum()
    assert np.max(np.abs(a - want)) <= 1e-14
    assert np.array_equal(a, best)
    assert diff == max(abs(x - y) for i, x in enumerate(train) for y in train[i + 1:])
