"""Point-level branches decided by bounds: the eta and Delta R cuts
(CHILI_PRE_CUTS), and two-body decays into legs of exactly vanishing mass
(SChannelWeight, ChannelElements.cc:113-135)."""
import numpy as np
import pytest

from chili_b200 import abi, channels, workloads
from oracle import port

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_out,ptmin,etamax,delta_r", [
    (4, 30.0, 99.0, 0.4), (4, 10.0, 2.0, 0.7), (3, 0.0, 1.0, 0.0), (3, 20.0, 800.0, 2.5), (2, 5.0, 99.0, 3.0),
    (2, 5.0, 99.0, 3.3)])
def test_cuts_accept_the_oracles_points(ctx_factory, n_out, ptmin, etamax, delta_r):
    cs = workloads.channel_set(n_out)
    ctx = ctx_factory()
    ctx.set_channels(cs)
    ctx.uniform_grids(cs.nch, ctx.ndims, 20)
    ctx.set_integrand(abi.CHILI_FUNC_PROPAGATOR, channels.propagator_params())
    ctx.set_preprocess_cuts(1000.0, ptmin, etamax, delta_r)
    p = workloads.mc_params(2000)
    O = port.MultiChannel(cs, 20, p, abi.CHILI_FUNC_PROPAGATOR, channels.propagator_params())
    O.set_cuts(1000.0, ptmin, etamax, delta_r)
    st, info = ctx.multichannel_iterate(p, seed=5)
    u = port.philox_uniforms(5, 0, info.points_tried, ctx.ndims + 1)
    st_o, info_o = O.iterate(u)
    assert info.points_tried == info_o.points_tried
    assert (st.n, st.n_finite) == (st_o.n, st_o.n_finite)
    assert abs(st.sum - st_o.sum) <= 1e-11 * abs(st_o.sum)


def test_decays_into_exactly_massless_legs(ctx_factory):
    """Integer momenta, so that every squared mass vanishes exactly: opposite,
    orthogonal and parallel legs of the decaying pair, against the kernel that
    evaluates a channel per thread and the weight's closed form."""
    cs = workloads.channel_set(4)
    ctx = ctx_factory()
    ctx.set_channels(cs)
    pairs = [((5, 3, 4, 0), (13, 0, -5, 12)), ((65, 33, 56, 0), (13, 5, 0, -12)), ((50, 30, 40, 0), (100, 60, 80, 0)),
             ((50, 30, 40, 0), (50, -30, -40, 0))]
    others = [(85, 36, -77, 0), (85, 13, 84, 0)]
    mom = np.zeros((len(pairs), 6, 4))
    for k, (a, b) in enumerate(pairs):
        out = np.array([a, b] + others, dtype=np.float64)
        tot = out.sum(0)
        mom[k, 0] = [-(tot[0] + tot[3]) / 2, 0, 0, -(tot[0] + tot[3]) / 2]
        mom[k, 1] = [-(tot[0] - tot[3]) / 2, 0, 0, (tot[0] - tot[3]) / 2]
        mom[k, 2:] = out
    w, _ = ctx.fsmapper_weight(0, mom)  # channel 0: Z -> legs 2, 3
    assert np.isfinite(w[:2]).all() and (w[:2] != 0).all()
    assert w[2] == 0 or np.isnan(w[2])  # parallel legs: SqLam is 0
    ctx.uniform_grids(cs.nch, ctx.ndims, 10)
    ctx.set_integrand(abi.CHILI_FUNC_PROPAGATOR, channels.propagator_params())
    dens = []
    for pipeline in (0, 1):
        ctx.set_option("pipeline", pipeline)
        dens.append(ctx.multichannel_weight(mom, np.zeros(len(mom), dtype=np.int32))[1])
    assert np.array_equal(np.isfinite(dens[0]), np.isfinite(dens[1]))
    ok = np.isfinite(dens[0])
    assert np.allclose(dens[0][ok], dens[1][ok], rtol=1e-14, atol=0)
    assert np.allclose(dens[1][:2, 0], w[:2], rtol=1e-14, atol=0)
