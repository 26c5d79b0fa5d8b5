"""Two host threads, each with a context of its own, calling the same kernels
with tables of different sizes: a kernel's dynamic shared-memory limit belongs
to the process, so no call may lower it under another thread's launch."""
import ctypes as C
import threading

import numpy as np
import pytest
import torch

from chili_b200 import abi, channels, workloads

pytestmark = pytest.mark.gpu


def _together(calls, rounds):
    """Each call `rounds` times in a thread of its own; the errors raised."""
    start, errors = threading.Barrier(len(calls)), []

    def work(call):
        start.wait()
        try:
            for _ in range(rounds):
                call()
        except Exception as e:  # noqa: BLE001 -- reported below
            errors.append(e)

    threads = [threading.Thread(target=work, args=(c,)) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return errors


def test_channel_tables_of_two_sizes(ctx_factory):
    # 16 dimensions: 79 KB of tables at 100 bins, 157 KB at 200; device
    # buffers, so that a call is little more than its launches
    cs = workloads.channel_set(6)
    calls, checks = [], []
    for bins in (100, 200):
        ctx = ctx_factory()
        ctx.set_channels(cs)
        ctx.uniform_grids(cs.nch, ctx.ndims, bins)
        ctx.set_integrand(abi.CHILI_FUNC_PROPAGATOR, channels.propagator_params())
        mom, _, ich = ctx.generate(64, seed=5)
        want = ctx.multichannel_weight(mom, ich)[0]
        dev = [torch.from_numpy(a).cuda() for a in (mom, ich, np.zeros(64))]

        def call(ctx=ctx, dev=dev):
            ctx.call("chili_gpu_multichannel_weight", *(C.c_void_p(t.data_ptr()) for t in dev), None, None, 64)

        calls.append(call)
        checks.append((ctx, dev[2], want))
    for _ in range(20):
        assert not _together(calls, 400)
        for ctx, got, want in checks:
            ctx.synchronize()
            assert np.array_equal(got.cpu().numpy(), want, equal_nan=True)


def test_vegas_grids_of_two_sizes(ctx_factory):
    # 4 dimensions: an adapting iteration asks for 44.8 KB at 560 bins, 60.8 KB
    # at 760; materialised points stage 18 and 24 KB of edges
    calls = []
    for bins in (560, 760):
        ctx = ctx_factory()
        ctx.set_grids(np.tile(np.linspace(0, 1, bins + 1), (1, 4, 1)))
        ctx.set_integrand(abi.CHILI_FUNC_CAMEL, workloads.camel_params(4))
        calls.append(lambda ctx=ctx: ctx.vegas_iterate(1000, seed=3, adapt=True))
    for bins in (1600, 3200):  # 50 and 100 KB of edges
        ctx = ctx_factory()
        ctx.set_grids(np.tile(np.linspace(0, 1, bins + 1), (1, 4, 1)))
        ctx.set_integrand(abi.CHILI_FUNC_CAMEL, workloads.camel_params(4))
        calls.append(lambda ctx=ctx: ctx.vegas_generate(500, seed=3))
    assert not _together(calls, 1500)
