"""Entry points that weight every point of a call (Integrand::GenerateWeight,
Integrand.hh:112-123; MultiChannel::GeneratePoint/GenerateWeight,
MultiChannel.hh:141-165): the tiled phased pass against the kernel that runs
one point per thread, at sizes around a block and around a tile."""
import ctypes as C

import numpy as np
import pytest

from chili_b200 import abi, channels, workloads

pytestmark = pytest.mark.gpu


def _context(make, n_out, pipeline):
    cs = workloads.channel_set(n_out)
    ctx = make()
    ctx.set_channels(cs)
    ctx.set_option("pipeline", pipeline)
    rng = np.random.default_rng(5)
    e = np.sort(rng.random((cs.nch, ctx.ndims, 19)) ** 1.5, axis=2)
    ctx.set_grids(np.concatenate([np.zeros(e.shape[:2] + (1,)), e, np.ones(e.shape[:2] + (1,))], 2))
    ctx.set_integrand(abi.CHILI_FUNC_PROPAGATOR, channels.propagator_params())
    a = rng.random(cs.nch) + 0.1
    ctx.set_alpha(a / a.sum())
    return ctx


def _close(got, want):
    """The same operations on the same inputs, except that a channel of two
    decays divides by 2 pi in another order: one rounding per factor, amplified
    where the channels' signed densities cancel (a median bar and equal
    non-finite patterns)."""
    assert np.array_equal(np.isfinite(got), np.isfinite(want))
    ok = np.isfinite(want)
    err = np.abs(got[ok] - want[ok]) / np.maximum(np.abs(want[ok]), 1e-300)
    assert np.percentile(err, 99) <= 1e-14 if err.size else True


@pytest.mark.parametrize("n_out,n", [(2, 1), (4, 255), (4, 257), (6, 1001), (4, 262145)])
def test_tiled_weights_and_events_match_per_thread(ctx_factory, n_out, n):
    ctxs = [_context(ctx_factory, n_out, p) for p in (0, 1)]
    events = [c.generate(n, seed=11, counter=3) for c in ctxs]
    assert np.array_equal(events[0][0], events[1][0], equal_nan=True)
    assert np.array_equal(events[0][2], events[1][2])
    _close(events[1][1], events[0][1])
    mom, _, ich = events[0]
    ich = ich.copy()
    ich[n // 2] = -1  # no channel's uniforms: zeros
    got = [c.multichannel_weight(mom, ich) for c in ctxs]
    _close(got[1][0], got[0][0])
    _close(got[1][1], got[0][1])
    assert np.array_equal(got[1][2], got[0][2], equal_nan=True)
    assert not got[1][2][n // 2].any()


def test_outputs_are_optional(ctx_factory):
    ctx = _context(ctx_factory, 4, 1)
    mom, w, ch = ctx.generate(300, seed=2)
    only = np.empty_like(mom)
    ctx.call("chili_gpu_generate", 300, 2, 0, C.c_void_p(only.ctypes.data), None, None)
    assert np.array_equal(only, mom, equal_nan=True)
    full, _, _ = ctx.multichannel_weight(mom, ch)
    alone = np.empty(300)
    ctx.call("chili_gpu_multichannel_weight", C.c_void_p(mom.ctypes.data), C.c_void_p(ch.ctypes.data),
             C.c_void_p(alone.ctypes.data), None, None, 300)
    assert np.array_equal(alone, full, equal_nan=True)


@pytest.mark.parametrize("n_out,n", [(3, 513), (4, 257), (5, 300), (6, 1001), (4, 262145)])
def test_both_routes_round_every_point_the_same(ctx_factory, n_out, n):
    """Every density, weight and event value of the tiled pass has the bits of
    the per-thread kernel: the running product of a channel's decay weights is
    divided by 2 pi once per decay (Channel.cc:111) on both, so the bound at
    every point, cancelling channel sums included, is zero."""
    ctxs = [_context(ctx_factory, n_out, p) for p in (0, 1)]
    ctxs[1].generate(n, seed=1)  # a context's first short call is not tiled
    events = [c.generate(n, seed=29, counter=7) for c in ctxs]
    for a, b in zip(*events):
        assert np.array_equal(a, b, equal_nan=True)
    for a, b in zip(*(c.multichannel_weight(events[0][0], events[0][2]) for c in ctxs)):
        assert np.array_equal(a, b, equal_nan=True)


def _grown(call):
    """Device memory that the call leaves allocated."""
    import torch

    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    call()
    torch.cuda.synchronize()
    return before - torch.cuda.mem_get_info()[0]


def _device_points(ctx, n):
    import torch

    mom, _, ich = ctx.generate(n, seed=3)
    return [torch.from_numpy(a).cuda() for a in (mom, ich, np.zeros(n))]


def _weigh(ctx, dev):
    ctx.call("chili_gpu_multichannel_weight", *(C.c_void_p(t.data_ptr()) for t in dev), None, None, dev[1].shape[0])
    ctx.synchronize()
    return dev[2].cpu().numpy()


def test_work_space_follows_the_call(ctx_factory):
    """A call of one point holds no buffers for 2^16 of them (0.25 GB for the
    2->6 set), a context's first short call holds none, and drawing points
    without weights holds none either."""
    import torch

    mb = 1 << 20
    warm = _context(ctx_factory, 6, 1)  # the kernels' code is loaded once
    one, some = _device_points(warm, 1), _device_points(_context(ctx_factory, 4, 0), 20000)
    out = torch.empty(300000, 8, 4, dtype=torch.float64, device="cuda")

    def points_alone(ctx):
        ctx.call("chili_gpu_generate", out.shape[0], 2, 0, C.c_void_p(out.data_ptr()), None, None)

    for _ in range(2):
        _weigh(warm, one)
        _weigh(_context(ctx_factory, 4, 1), some)
    points_alone(warm)
    ctx = _context(ctx_factory, 6, 1)
    assert _grown(lambda: _weigh(ctx, one)) <= 8 * mb
    assert _grown(lambda: points_alone(ctx)) <= 8 * mb
    want = _context(ctx_factory, 6, 0).generate(out.shape[0], seed=2)[0]
    assert np.array_equal(out.cpu().numpy(), want, equal_nan=True)
    ctx = _context(ctx_factory, 4, 1)
    got = []
    assert _grown(lambda: got.append(_weigh(ctx, some))) <= 8 * mb
    assert _grown(lambda: got.append(_weigh(ctx, some))) > 8 * mb  # the second one is tiled
    assert np.array_equal(got[0], got[1], equal_nan=True)


def test_two_channels_are_tiled_beyond_one_wave(ctx_factory):
    """Two channels' few items pay for the tiled pass's launches only where the
    per-thread kernel needs more than one wave; the bits are the same."""
    ctx, ref = _context(ctx_factory, 2, 1), _context(ctx_factory, 2, 0)
    for n, tiled in ((65536, False), (65537, True)):
        dev = _device_points(ref, n)
        want = _weigh(ref, dev)
        for k in range(3):
            before = ctx.launches
            assert np.array_equal(_weigh(ctx, dev), want, equal_nan=True)
            assert (ctx.launches - before > 1) == (tiled and k > 0)  # the first short call allocates nothing


def test_calls_of_changing_size_on_one_context(ctx_factory):
    """The tile's parts are laid out anew by every call."""
    ctx, ref = _context(ctx_factory, 4, 1), _context(ctx_factory, 4, 0)
    for n in (1, 64, 65, 5000, 3, 70000, 300, 262145, 2):
        got, want = ctx.generate(n, seed=n), ref.generate(n, seed=n)
        for a, b in zip(got, want):
            assert np.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("n", [1000, 70000])
def test_captured_calls_allocate_nothing_and_replay_the_same_bits(ctx_factory, n):
    """On a stream that is being captured the calls take the per-thread
    kernels, which need no buffers of the context; a replay on other inputs in
    the same buffers gives what an eager, tiled call gives."""
    import torch

    ctx = _context(ctx_factory, 4, 1)
    dev = _device_points(ctx, n)
    stream = torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)
    eager = [_weigh(ctx, dev), _weigh(ctx, dev)]
    out = [torch.zeros(n, 6, 4, dtype=torch.float64, device="cuda"), torch.zeros(n, dtype=torch.float64, device="cuda"),
           torch.zeros(n, dtype=torch.int32, device="cuda")]
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        before = ctx.launches
        ctx.call("chili_gpu_multichannel_weight", *(C.c_void_p(t.data_ptr()) for t in dev), None, None, n)
        ctx.call("chili_gpu_generate", n, 5, 9, *(C.c_void_p(t.data_ptr()) for t in out))
        assert ctx.launches - before == 2
    for seed in (3, 4):
        mom, w, ich = ctx.generate(n, seed=seed)
        dev[0].copy_(torch.from_numpy(mom))
        dev[1].copy_(torch.from_numpy(ich))
        dev[2].zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        want = eager[1] if seed == 3 else ctx.multichannel_weight(mom, ich)[0]
        assert np.array_equal(dev[2].cpu().numpy(), want, equal_nan=True)
    assert np.array_equal(eager[0], eager[1], equal_nan=True)
    for a, b in zip(out, ctx.generate(n, seed=5, counter=9)):
        assert np.array_equal(a.cpu().numpy(), b, equal_nan=True)
