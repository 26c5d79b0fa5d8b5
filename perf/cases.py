"""The measured workloads of chili_b200: what programs call this library for.

Every case goes through the public entry points (chili_b200.gpu.Context, and
the C ABI of include/chili_gpu.h on device buffers where a program keeps its
points on the GPU).  The kinds:

vegas       one adapting Vegas iteration (plain VEGAS of the camel)
points      materialised VEGAS points (x and weight of every point)
iterate     one adapting multichannel iteration from a trained grid
weight      the combined multichannel weight of given momenta
events      weighted events: momenta, weight and channel of drawn points
unweighted  hit-or-miss unweighted events of drawn points
evaluate    uniforms through one channel (the hook of the TensorFlow and
            nanobind front ends)
batch       adapting iterations of many uneven integrands together
flow_grad   loss and gradient of the learned proposal on a training batch
flow_sample the learned proposal's sampling direction

The second half of the file restates each kind in 64-bit torch (exact()).
"""
import ctypes
import math

import numpy as np
import torch

from chili_b200 import abi, gpu, workloads

SQRTS = 1000.0
PTMIN, ETAMAX, DELTA_R = 30.0, 99.0, 0.4
MZ, GZ, MT = 91.1876, 2.4952, 10.0
# integrand of the 2->n workloads: the product of the two largest pair
# propagators from six outgoing legs on, their sum below
PAIR_SUM, PAIR_TOP2 = abi.CHILI_FUNC_PROPAGATOR, abi.CHILI_FUNC_PROPAGATOR_TOP2
# about the largest weight of an iteration on the trained grid
W_MAX = {4: 2e-18, 6: 5e-28}
# iterations of one integration before the next starts from the trained grid
# (the default of MultiChannelParams)
INTEGRATION = 10


def listed():
    return [
        # the plain-VEGAS workload: 4-d camel, 50 bins, 1e5 points; a call of
        # tens of microseconds, made ten to hundreds of times
        {"name": "vegas_camel_1e5", "kind": "vegas", "dims": 4, "bins": 50, "n": 100_000, "sigma": 0.1},
        # points of a trained VEGAS grid handed to a device-side consumer
        {"name": "vegas_points_2e7", "kind": "points", "dims": 4, "bins": 50, "n": 20_000_000, "sigma": 0.1},
        # one iteration at the reference's default ncalls (10000): latency
        {"name": "iterate_2to4_1e4", "kind": "iterate", "n_out": 4, "bins": 100, "n": 10_000},
        # the headline workload: 15 channels, 100 bins, 1e6 points
        {"name": "iterate_2to4_1e6", "kind": "iterate", "n_out": 4, "bins": 100, "n": 1_000_000},
        # the large channel set: 45 channels, 16 dimensions, 200 bins
        {"name": "iterate_2to6_1e6", "kind": "iterate", "n_out": 6, "bins": 200, "n": 1_000_000},
        # reweighting a ragged batch of momenta that are already on the GPU
        {"name": "weight_2to4_3e5", "kind": "weight", "n_out": 4, "bins": 100, "n": 300_007},
        # weighted events for a device-side consumer
        {"name": "events_2to4_1e6", "kind": "events", "n_out": 4, "bins": 100, "n": 1_000_000},
        # event generation after training: 4e6 drawn points per call
        {"name": "unweighted_2to4_4e6", "kind": "unweighted", "n_out": 4, "bins": 100, "n": 4_000_000},
        # one call of the framework front ends: a batch through one channel
        {"name": "evaluate_2to4_1e5", "kind": "evaluate", "n_out": 4, "channel": 3, "n": 100_003},
        # the 512-integrand workload's mix at an eighth of the tasks
        {"name": "batch_64", "kind": "batch", "camels": 32, "multichannels": 32, "scale": 0.5, "iterations": 2},
        # one training batch of the 6-layer flow, forward and backward
        {"name": "flow_grad_65536", "kind": "flow_grad", "n_out": 4, "layers": 6, "hidden": 128, "depth": 2,
         "n": 65_536},
        # proposal points of one sampling chunk
        {"name": "flow_sample_1e6", "kind": "flow_sample", "n_out": 4, "layers": 6, "hidden": 128, "depth": 2,
         "n": 1_000_000},
    ]


STATS = ("n", "min", "max", "sum", "sum2", "n_finite")


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["vegas", "points", "iterate", "iterate", "weight", "events", "unweighted", "evaluate",
                       "batch", "flow_grad", "flow_sample"])
    if kind in ("vegas", "points"):
        n = _log_int(rng, 10_000, 5_000_000 if kind == "vegas" else 20_000_000)
        return {"kind": kind, "dims": rng.randint(2, 8), "bins": rng.randint(20, 200), "n": n,
                "sigma": round(rng.uniform(0.1, 0.2), 4)}
    if kind == "iterate":
        # larger channel sets need more points per iteration to train on
        n_out = rng.choice([3, 4, 5, 6])
        return {"kind": kind, "n_out": n_out, "bins": rng.randint(20, 200),
                "n": _log_int(rng, {3: 10_000, 4: 10_000, 5: 40_000, 6: 100_000}[n_out], 800_000)}
    if kind in ("weight", "events"):
        return {"kind": kind, "n_out": rng.choice([3, 4, 5, 6]), "bins": rng.randint(20, 200),
                "n": _log_int(rng, 1_000, 800_000)}
    if kind == "unweighted":
        return {"kind": kind, "n_out": rng.choice([4, 6]), "bins": rng.randint(50, 200),
                "n": _log_int(rng, 20_000, 2_000_000)}
    if kind == "evaluate":
        return {"kind": kind, "n_out": rng.choice([3, 4, 5, 6]), "channel": rng.randint(0, 5),
                "n": _log_int(rng, 1_000, 3_000_000)}
    if kind == "batch":
        return {"kind": kind, "camels": rng.randint(2, 32), "multichannels": rng.randint(2, 32),
                "scale": round(math.exp(rng.uniform(math.log(0.02), math.log(0.5))), 4), "iterations": 2}
    case = {"kind": kind, "n_out": rng.choice([3, 4]), "layers": rng.randint(4, 8),
            "hidden": rng.choice([128, 128, 256]), "depth": rng.choice([2, 3])}
    return dict(case, n=_log_int(rng, 512, 65_536) if kind == "flow_grad" else _log_int(rng, 2_000, 400_000))


# ------------------------------------------------------------------ inputs
def _rng(seed):
    return np.random.default_rng(int(seed))


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _channel_set(n_out):
    return workloads.channel_set(n_out, SQRTS)


# Quantiles (at 0, .05, .25, .5, .75, .95, 1) that the trained grids of the
# 2->4 and 2->6 workloads have, by what a dimension samples.
_LEVELS = np.array([0.0, 0.05, 0.25, 0.5, 0.75, 0.95, 1.0])
_QUANTILES = {
    "pole": [0, 0.02, 0.24, 0.50, 0.76, 0.98, 1], "pair": [0, 0.29, 0.42, 0.51, 0.59, 0.70, 1],
    "pt": [0, 0.384, 0.44, 0.53, 0.64, 0.80, 1], "pt_pair": [0, 0.70, 0.88, 0.94, 0.975, 0.99, 1],
    "y": [0, 0.19, 0.365, 0.50, 0.64, 0.80, 1], "flat": [0, 0.05, 0.25, 0.5, 0.75, 0.95, 1],
    "last": [0, 0.04, 0.23, 0.50, 0.76, 0.96, 1], "cos": [0, 0.15, 0.30, 0.48, 0.68, 0.85, 1],
}


def _roles(info, decays):
    """What each uniform of a channel samples, in the channel's order."""
    roles = ["pole" if d.parent.width > 0 else "pair"
             for d in sorted(decays, key=lambda d: d.parent.key())]
    for p in info[:-1]:
        roles += ["pt_pair" if p.idx & (p.idx - 1) and len(roles) > 2 else "pt", "y", "flat"]
    return roles + ["last"] + ["cos", "flat"] * len(decays)


def _trained_grids(cs, bins, rng):
    """Monotone VEGAS grids of the shapes that training gives, each with its
    own fluctuations."""
    edges = np.empty((cs.nch, cs.ndims, bins + 1))
    for c, (info, decays) in enumerate(cs.channels):
        for d, role in enumerate(_roles(info, decays)):
            q = np.array(_QUANTILES[role]) + 0.01 * rng.uniform(-1, 1, 7)
            q[0], q[-1] = 0.0, 1.0
            widths = np.diff(np.interp(np.arange(bins + 1) / bins, _LEVELS, np.sort(q.clip(0, 1)) + 1e-4 * _LEVELS))
            widths *= rng.uniform(0.85, 1.15, bins)
            edges[c, d, 0] = 0.0
            edges[c, d, 1:] = np.cumsum(widths) / widths.sum()
            edges[c, d, -1] = 1.0
    return edges


def _trained_alpha(cs, rng):
    """Channel weights of a trained set: the pole channels lead, the pairs of
    massless currents end near the floor."""
    share = np.array([0.75 if decays and decays[0].parent.width > 0 else (0.02 if decays else 0.23)
                      for _, decays in cs.channels])
    count = {s: np.sum(share == s) for s in set(share)}
    a = share / np.array([count[s] for s in share]) * rng.uniform(0.4, 1.6, cs.nch)
    return a / a.sum()


def _integrand(n_out):
    return PAIR_TOP2 if n_out >= 6 else PAIR_SUM


def _context(case, seed, cuts=True):
    """A program's handle: channels, trained grids, channel weights, integrand."""
    cs = _channel_set(case["n_out"])
    rng = _rng(seed)
    ctx = gpu.Context()
    ctx.set_channels(cs)
    ctx.set_integrand(_integrand(case["n_out"]), [MZ, GZ, MT])
    if cuts:
        ctx.set_preprocess_cuts(SQRTS, PTMIN, ETAMAX, DELTA_R)
    else:
        ctx.set_preprocess(abi.CHILI_PRE_FINITE)
    state = {"case": case, "ctx": ctx, "cs": cs, "seed": int(seed)}
    if "bins" in case:
        grids, alpha = _trained_grids(cs, case["bins"], rng), _trained_alpha(cs, rng)
        ctx.set_grids(grids)
        ctx.set_alpha(alpha)
        state.update(grids=_dev(grids), alpha=_dev(alpha))
    return state


def _camel(case, seed):
    """Camel parameters with centres of their own and unit integral."""
    rng = _rng(seed)
    a, b = rng.uniform(0.25, 0.45, case["dims"]), rng.uniform(0.55, 0.75, case["dims"])
    return np.array(workloads.camel_params(case["dims"], case["sigma"], a, b))


def _camel_grid(case, params):
    """The grid that training on that camel ends near: half of the bins on
    each peak, over a flat share."""
    d, bins, s = case["dims"], case["bins"], params[0]
    x = np.linspace(0, 1, 2001)
    edges = np.empty((1, d, bins + 1))
    for j in range(d):
        dens = 0.2 + sum(np.exp(-((x - params[2 + j + o]) / s) ** 2) for o in (0, d)) / s
        cdf = np.concatenate([[0], np.cumsum((dens[1:] + dens[:-1]) / 2)])
        edges[0, j] = np.interp(np.arange(bins + 1) / bins, cdf / cdf[-1], x)
    edges[..., 0], edges[..., -1] = 0.0, 1.0
    return edges


def _momenta(n, n_out, seed):
    """Massless outgoing momenta inside the cuts and the beams that balance
    them, all-outgoing convention (incoming energies negative)."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))

    def rand(*shape):
        return torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)

    got, have = [], 0
    while have < n:
        m = max(4096, 2 * n)
        pt = PTMIN * (1.2 + 4 * rand(m, n_out) ** 3)
        y, phi = 2.4 * (rand(m, n_out) - 0.5), 2 * math.pi * rand(m, n_out)
        px, py = pt * torch.cos(phi), pt * torch.sin(phi)
        px[:, -1] = -px[:, :-1].sum(1)
        py[:, -1] = -py[:, :-1].sum(1)
        pt = torch.sqrt(px * px + py * py)
        out = torch.stack([pt * torch.cosh(y), px, py, pt * torch.sinh(y)], 2)
        tot = out.sum(1)
        zero = torch.zeros_like(tot[:, 0])
        plus, minus = (tot[:, 0] + tot[:, 3]) / 2, (tot[:, 0] - tot[:, 3]) / 2
        beams = [torch.stack([-plus, zero, zero, -plus], 1), torch.stack([-minus, zero, zero, minus], 1)]
        mom = torch.cat([torch.stack(beams, 1), out], 1)
        got.append(mom[_inside(mom)])
        have += len(got[-1])
    return torch.cat(got)[:n].contiguous()


def _channel_draw(n, nch, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed) + 1)
    return torch.randint(0, nch, (n,), generator=g, device="cuda", dtype=torch.int32)


def _flow_masks(dims, layers):
    """Conditioning dimensions of each layer (include/chili_gpu.h)."""
    i = np.arange(dims)
    pats = [i % 2 == 0, i % 2 == 1, i < dims // 2, i >= dims // 2, ((i + 1) // 2) % 2 == 0, ((i + 1) // 2) % 2 == 1]
    return [pats[layer % 6] for layer in range(layers)]


def _flow_shapes(case, dims, nch):
    """[(name, shape)] of the flat parameters (include/chili_gpu.h)."""
    h, out = case["hidden"], []
    for layer, m in enumerate(_flow_masks(dims, case["layers"])):
        out += [("W1_%d" % layer, (h, int(m.sum()))), ("E_%d" % layer, (nch, h))]
        out += [("W2_%d_%d" % (layer, k), (h, h)) for k in range(case["depth"] - 1)]
        out += [("W3_%d" % layer, (int((~m).sum()) * 49, h))]
    nf = case["n_out"] * (case["n_out"] - 1) // 2 + case["n_out"]
    return out + [("A1", (64, nf)), ("c1", (64,)), ("A2", (64, 64)), ("c2", (64,)), ("A3", (nch, 64)), ("c3", (nch,))]


def _flow_params(case, dims, nch, seed):
    """Weights of a partly trained flow: the initial scales, spline
    parameters away from the identity."""
    rng, flat = _rng(seed), []
    for name, shape in _flow_shapes(case, dims, nch):
        fan = shape[-1]
        if name.startswith("W3"):
            v = rng.normal(0, 0.1 / math.sqrt(fan), shape)
        elif name[0] in "Ec":
            v = rng.normal(0, 0.1, shape)
        else:
            v = rng.uniform(-1, 1, shape) * math.sqrt((4.0 if name[0] == "W" else 1.0) / fan)
        flat.append(v.reshape(-1))
    return np.concatenate(flat).astype(np.float32)


def _flow_batch(case, dims, nch, seed):
    n, n_out = case["n"], case["n_out"]
    g = torch.Generator(device="cuda").manual_seed(int(seed) + 2)
    u = torch.rand(n, dims, generator=g, device="cuda") * 0.9998 + 0.0001
    ch = _channel_draw(n, nch, seed)
    if case["kind"] == "flow_sample":
        return u, ch
    nf = n_out * (n_out - 1) // 2 + n_out
    feat = torch.randn(n, nf, generator=g, device="cuda")
    logf = torch.cos(2 * math.pi * u[:, :4] - 2.0).sum(1) - 1.0  # structure for the flow to learn
    prior = torch.log_softmax(torch.randn(n, nch, generator=g, device="cuda"), 1)
    return u, ch, logf, feat, prior


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("vegas", "points"):
        params = _camel(case, seed)
        ctx = gpu.Context()
        ctx.set_integrand(abi.CHILI_FUNC_CAMEL, params)
        state = {"case": case, "ctx": ctx, "seed": int(seed), "counter": 0}
        ctx.set_grids(_camel_grid(case, params))
        if kind == "points":
            state["out"] = (torch.empty(case["n"], case["dims"], dtype=torch.float64, device="cuda"),
                            torch.empty(case["n"], dtype=torch.float64, device="cuda"))
        else:
            state["edges"] = torch.empty(1, case["dims"], case["bins"] + 1, dtype=torch.float64, device="cuda")
        return state
    if kind == "batch":
        ctx = gpu.Context()
        ctx.batch_set(workloads.batched_tasks(int(seed), case["camels"], case["multichannels"],
                                              scale=case["scale"]))
        return {"case": case, "ctx": ctx, "seed": int(seed)}
    state = _context(case, seed, cuts=kind != "evaluate")
    ctx, cs, n = state["ctx"], state["cs"], case.get("n")
    f64 = {"dtype": torch.float64, "device": "cuda"}
    if kind == "iterate":
        params = workloads.mc_params(n)
        state.update(params=params, counter=0, passes=0, edges=torch.empty_like(state["grids"]))
        # the integration that trained these grids ran in this context: its
        # buffers and acceptance rate are in place
        ctx.multichannel_iterate(params, seed=int(seed), counter=1 << 40)
        ctx.set_grids(state["grids"])
        ctx.set_alpha(state["alpha"])
    elif kind == "weight":
        state.update(mom=_momenta(n, case["n_out"], seed), ich=_channel_draw(n, cs.nch, seed),
                     wgt=torch.empty(n, **f64), dens=torch.empty(n, cs.nch, **f64), x=torch.empty(n, cs.ndims, **f64))
    elif kind in ("events", "unweighted"):
        rows = n if kind == "events" else max(1024, n // 16)
        state.update(rows=rows, mom=torch.zeros(rows, cs.n_ext, 4, **f64), wgt=torch.zeros(rows, **f64),
                     ich=torch.zeros(rows, dtype=torch.int32, device="cuda"))
    elif kind == "evaluate":
        g = torch.Generator(device="cuda").manual_seed(int(seed))
        state.update(u=torch.rand(n, cs.ndims, generator=g, **f64), out=torch.empty(n, **f64))
    else:
        ctx.uniform_grids(cs.nch, cs.ndims, 50)
        ctx.set_alpha(_trained_alpha(cs, _rng(seed)))
        ctx.flow_init(layers=case["layers"], hidden=case["hidden"], depth=case["depth"], batch=max(128, n))
        ctx.flow_set_params(_flow_params(case, cs.ndims, cs.nch, seed))
        state["batch"] = _flow_batch(case, cs.ndims, cs.nch, seed)
        if kind == "flow_grad":
            state["grad"] = torch.empty(ctx.flow_np, dtype=torch.float32, device="cuda")
        else:
            state["u"] = torch.empty(n, cs.ndims, dtype=torch.float32, device="cuda")
            state["logq"] = torch.empty(n, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    return state


def _by_stat(stats):
    """StatsData of many tasks [..., 6] by field (the extremes of n would
    hide the sums)."""
    return {name: np.ascontiguousarray(stats[..., i]) for i, name in enumerate(STATS)}


# ------------------------------------------------------------------ one pass
def run(s):
    case, ctx = s["case"], s["ctx"]
    kind, n = case["kind"], case.get("n")
    if kind == "vegas":
        stats = ctx.vegas_iterate(n, seed=s["seed"], counter=s["counter"], alpha=1.5, adapt=True)
        s["counter"] += n
        ctx.call("chili_gpu_get_grids", _ptr(s["edges"]), 1, case["dims"], case["bins"])
        return dict(zip(STATS, np.array(stats.as_tuple())), grid=s["edges"])
    if kind == "points":
        x, w = ctx.vegas_generate(n, seed=s["seed"], out=s["out"])
        return {"x": x, "w": w}
    if kind == "iterate":
        if s["passes"] == INTEGRATION:  # the next integration
            s["passes"] = 0
            ctx.set_grids(s["grids"])
            ctx.set_alpha(s["alpha"])
        s["passes"] += 1
        stats, info = ctx.multichannel_iterate(s["params"], seed=s["seed"], counter=s["counter"])
        s["counter"] += info.points_tried
        ctx.call("chili_gpu_get_grids", _ptr(s["edges"]), *s["edges"].shape[:2], case["bins"])
        counts = (info.points_tried, info.points_accepted, info.rejected_pre, info.rejected_nan)
        return dict(zip(STATS, np.array(stats.as_tuple())), wmax=np.float64(info.weight_max), grids=s["edges"],
                    alpha=ctx.get_alpha()[0], counts=np.array(counts, dtype=np.int64))
    if kind == "weight":
        ctx.call("chili_gpu_multichannel_weight", _ptr(s["mom"]), _ptr(s["ich"]), _ptr(s["wgt"]), _ptr(s["dens"]),
                 _ptr(s["x"]), n)
        return {"weight": s["wgt"], "density": s["dens"], "x": s["x"]}
    if kind == "events":
        ctx.call("chili_gpu_generate", n, s["seed"], 0, _ptr(s["mom"]), _ptr(s["wgt"]), _ptr(s["ich"]))
        return {"momenta": s["mom"], "weight": s["wgt"], "channel": s["ich"]}
    if kind == "unweighted":
        info = ctx.generate_unweighted(n, W_MAX[case["n_out"]], seed=s["seed"], max_events=s["rows"],
                                       out=(s["mom"], s["wgt"], s["ich"]))[3]
        return {"momenta": s["mom"], "weight": s["wgt"], "channel": s["ich"], "sum": np.float64(info.sum),
                "max": np.float64(info.max), "kept": int(info.kept)}
    if kind == "evaluate":
        ctx.call("chili_gpu_evaluate_batch", case["channel"] % s["cs"].nch, _ptr(s["u"]), _ptr(s["out"]), n)
        return {"value": s["out"]}
    if kind == "batch":
        stats, _ = ctx.batch_iterate(case["iterations"], seed=s["seed"], adapt=True)
        return {"camel": _by_stat(stats[:, :case["camels"]]), "multichannel": _by_stat(stats[:, case["camels"]:])}
    if kind == "flow_grad":
        u, ch, logf, feat, prior = s["batch"]
        loss = ctypes.c_double()
        ctx.call("chili_gpu_flow_loss_grad", _ptr(u), _ptr(ch), _ptr(logf), _ptr(feat), _ptr(prior), n,
                 ctypes.byref(loss), _ptr(s["grad"]))
        return {"loss": np.float32(loss.value), "grad": s["grad"]}
    z, ch = s["batch"]
    ctx.call("chili_gpu_flow_sample_u", _ptr(z), _ptr(ch), n, _ptr(s["u"]), _ptr(s["logq"]))
    return {"u": s["u"], "logq": s["logq"]}


# ------------------------------------------------------------------ work
# FP64 operations of the path's parts, a transcendental function counted as 20
_FORWARD, _ENTRY, _CHAIN, _DECAY, _SEARCH = 60, 90, 130, 110, 12


def _forward_flops(cs):
    return cs.ndims * _FORWARD


def _weight_flops(cs):
    """All channels' densities of one point, the parts that channels share
    evaluated once."""
    entries, chains, decays = set(), set(), set()
    for info, dec in cs.channels:
        entries.update(p.key() for p in info[:-1])
        chains.add(tuple(p.key() for p in info))
        decays.update((d.parent.key(), d.child1.key()) for d in dec)
    return len(entries) * _ENTRY + len(chains) * _CHAIN + len(decays) * _DECAY + cs.nch * cs.ndims * _SEARCH


def _flow_flops(case, dims, nch):
    return 2 * sum(math.prod(shape) for name, shape in _flow_shapes(case, dims, nch) if name[0] in "WA")


def work(case):
    kind, n = case["kind"], case.get("n")
    if kind in ("vegas", "points"):
        d = case["dims"]
        per = 24 * d + 60
        out = 8 * n * (d + 1) if kind == "points" else 8 * (2 * d * (case["bins"] + 1) + 6)
        return {"bytes": out, "flops": n * per}
    if kind == "batch":
        tasks = workloads.batched_tasks(1, case["camels"], case["multichannels"], scale=case["scale"])
        flops = sum(t["ncalls"] * (24 * t["dims"] + 60 if t["kind"] == "camel" else
                                   _forward_flops(t["channels"]) + _weight_flops(t["channels"])) for t in tasks)
        return {"bytes": 48 * len(tasks) * case["iterations"], "flops": flops * case["iterations"]}
    cs = _channel_set(case["n_out"])
    if kind == "iterate":  # about 1.7 points tried per accepted one inside the cuts
        return {"bytes": 16 * cs.nch * (cs.ndims * (case["bins"] + 1) + 1),
                "flops": n * (1.7 * _forward_flops(cs) + _weight_flops(cs))}
    if kind == "weight":
        return {"bytes": n * (32 * cs.n_ext + 4 + 8 * (1 + cs.nch + cs.ndims)), "flops": n * _weight_flops(cs)}
    if kind == "events":
        return {"bytes": n * (32 * cs.n_ext + 12), "flops": n * (_forward_flops(cs) + _weight_flops(cs))}
    if kind == "unweighted":
        return {"bytes": 16 * cs.nch * cs.ndims * (case["bins"] + 1),
                "flops": n * (_forward_flops(cs) + 0.5 * _weight_flops(cs))}
    if kind == "evaluate":
        return {"bytes": 8 * n * (cs.ndims + 1), "flops": n * 2 * _forward_flops(cs)}
    flops = _flow_flops(case, cs.ndims, cs.nch)
    if kind == "flow_grad":
        nf = case["n_out"] * (case["n_out"] + 1) // 2
        return {"bytes": 4 * n * (cs.ndims + 2 + nf + cs.nch), "flops": 3 * n * flops}
    return {"bytes": 4 * n * (2 * cs.ndims + 2), "flops": n * flops}


# ------------------------------------------------- the same in 64-bit torch
def _mul_hi_lo(a, m):
    p = a * m  # 32 x 32 bits; the product's bits are right modulo 2^64
    return (p >> 32) & 0xFFFFFFFF, p & 0xFFFFFFFF


def _uniforms(key, counters, count, stream=0):
    """Philox4x32-10 uniforms [len(counters), count]: pair q of counter k is
    the block {q, lo(k), hi(k), stream} under the key {lo, hi}."""
    out = torch.empty(len(counters), count, dtype=torch.float64, device=counters.device)
    for q in range((count + 1) // 2):
        a = torch.full_like(counters, q)
        b, c, d = counters & 0xFFFFFFFF, counters >> 32, torch.full_like(counters, stream)
        k0, k1 = key & 0xFFFFFFFF, key >> 32
        for _ in range(10):
            h0, l0 = _mul_hi_lo(a, 0xD2511F53)
            h1, l1 = _mul_hi_lo(c, 0xCD9E8D57)
            a, b, c, d = h1 ^ b ^ k0, l1, h0 ^ d ^ k1, l0
            k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
        out[:, 2 * q] = ((a << 21) | (b >> 11)).double() * 2.0 ** -53
        if 2 * q + 1 < count:
            out[:, 2 * q + 1] = ((c << 21) | (d >> 11)).double() * 2.0 ** -53
    return out


def _grid_map(edges, u):
    """x and the Jacobian of uniforms through one grid [dims, bins + 1]."""
    bins = edges.shape[1] - 1
    x, jac = torch.empty_like(u), torch.ones_like(u[:, 0])
    for d in range(u.shape[1]):
        pos = u[:, d] * bins
        i = pos.long()
        size = edges[d][i + 1] - edges[d][i]
        x[:, d] = edges[d][i] + (pos - i) * size
        jac = jac * size * bins
    return x, jac


def _bins_of(edges, x):
    """Bin of every coordinate: the last edge below x."""
    return torch.stack([torch.searchsorted(edges[d][:-1].contiguous(), x[:, d].contiguous()) - 1
                        for d in range(x.shape[1])], 1).clamp(min=0)


def _camel_value(params, x):
    d = x.shape[1]
    p = torch.from_numpy(params).to(x.device)
    d1, d2 = ((x - p[2:2 + d]) ** 2).sum(1), ((x - p[2 + d:2 + 2 * d]) ** 2).sum(1)
    return p[1] * (torch.exp(-d1 / p[0] ** 2) + torch.exp(-d2 / p[0] ** 2))


def _adapt(edges, hist, alpha):
    """VEGAS rebinning of one dimension: smoothed importances, equal shares."""
    bins = len(hist)
    o = np.concatenate([[0.0], hist, [0.0]])
    s = (o[:-2] + o[1:-1] + o[2:]) / 3
    s[0], s[-1] = (hist[0] + hist[1]) / 2, (hist[-2] + hist[-1]) / 2
    r = s / s.sum()
    with np.errstate(divide="ignore", invalid="ignore"):
        imp = np.where(s > 0, ((r - 1) / np.log(r)) ** alpha, 0.0)
    cum = np.concatenate([[0.0], np.cumsum(imp)])
    want = imp.sum() / bins * np.arange(1, bins)
    k = np.searchsorted(cum, want).clip(1, bins)
    new = np.empty(bins + 1)
    new[0], new[-1] = 0.0, 1.0
    new[1:-1] = edges[k] - (edges[k] - edges[k - 1]) * (cum[k] - want) / imp[k - 1]
    return new


def _stats(values, rejected=0):
    n = len(values) + rejected
    lo, hi = float(values.min()), float(values.max())
    return np.array([n, min(lo, 0.0) if rejected else lo, max(hi, 0.0, 2.2250738585072014e-308),
                     float(values.sum()), float((values ** 2).sum()), float((values != 0).sum())])


def _exact_vegas(case, params, edges, key, counters, want_points=False):
    e = torch.from_numpy(edges[0]).cuda()
    total = []
    hist = torch.zeros(case["dims"] * case["bins"], dtype=torch.float64, device="cuda")
    for part in counters.split(1 << 21):
        x, jac = _grid_map(e, _uniforms(key, part, case["dims"]))
        v = _camel_value(params, x) * jac
        if want_points:
            total.append((x, v))
            continue
        slot = _bins_of(e, x) + case["bins"] * torch.arange(case["dims"], device="cuda")
        hist.index_add_(0, slot.reshape(-1), (v * v)[:, None].expand(-1, case["dims"]).reshape(-1))
        total.append(v)
    if want_points:
        return {"x": torch.cat([t[0] for t in total]), "w": torch.cat([t[1] for t in total])}
    return _stats(torch.cat(total)), hist.reshape(case["dims"], case["bins"]).cpu().numpy()


# four-vectors: [..., 4] as (E, px, py, pz)
def _m2(p):
    return p[..., 0] ** 2 - ((p[..., 1] ** 2 + p[..., 2] ** 2) + p[..., 3] ** 2)


def _rapidity(p):
    return torch.log((p[..., 0] + p[..., 3]) / (p[..., 0] - p[..., 3])) / 2


def _axes(p):
    """The two transverse axes of a decay of p (reference axis x): 3-vectors."""
    v = p[:, 1:]
    a = v.norm(dim=1)
    l = v / a[:, None]
    s = torch.sqrt(l[:, 1] ** 2 + l[:, 2] ** 2)
    n_perp = torch.stack([s, -l[:, 0] * l[:, 1] / s, -l[:, 0] * l[:, 2] / s], 1)
    side = torch.sign(a - p[:, 0] * l[:, 0])
    l_perp = torch.stack([torch.zeros_like(s), -side * l[:, 2] / s, side * l[:, 1] / s], 1)
    return l, l_perp, n_perp


def _boost(p, v, back):
    m = torch.sqrt(_m2(p))
    sign = 1.0 if back else -1.0
    pv = (p[:, 1:] * v[:, 1:]).sum(1)
    v0 = (p[:, 0] * v[:, 0] + sign * pv) / m
    c = (v[:, 0] + v0) / (m + p[:, 0])
    return torch.cat([v0[:, None], v[:, 1:] + sign * p[:, 1:] * c[:, None]], 1)


class _Mapping:
    """One FSMapper channel (all legs massless) in 64-bit torch."""

    def __init__(self, cs, c):
        info, decays = cs.channels[c]
        self.n_ext, self.sqrts = cs.n_ext, cs.sqrts
        self.info = [p.idx for p in info]
        self.decays = sorted(decays, key=lambda d: d.parent.key())
        by = {d.parent.key(): d for d in decays}
        self.order = [by[p.key()] for p in info if p.key() in by]  # one level of decays

    def _ptmin(self, idx):
        return PTMIN if idx & (idx - 1) == 0 else 1.0

    def _limits(self, d):
        both = [PTMIN if c.idx & (c.idx - 1) == 0 else 0.0 for c in (d.child1, d.child2)]
        return both[0] * both[1] * 2 / math.pi / math.pi * DELTA_R ** 2, self.sqrts ** 2

    def _last(self, psum):
        s = self.sqrts
        m2, yj, ptj2 = _m2(psum), _rapidity(psum), psum[:, 1] ** 2 + psum[:, 2] ** 2
        return ptj2, torch.sqrt(m2 + ptj2) / s, yj

    def generate(self, x):
        s, ir, m2 = self.sqrts, 0, {1 << i: 0.0 for i in range(self.n_ext)}
        for d in self.decays:
            u, (lo, hi) = x[:, ir], self._limits(d)
            ir += 1
            m, g = d.parent.mass, d.parent.width
            if g > 0:
                y1, y0 = math.atan((lo - m * m) / (m * g)), math.atan((hi - m * m) / (m * g))
                m2[d.parent.idx] = m * m + m * g * torch.tan(y0 + u * (y1 - y0))
            else:
                ce = 1.0 - 0.99
                m2[d.parent.idx] = (u * hi ** ce + (1 - u) * lo ** ce) ** (1 / ce)
        mom, psum, ptmax = {}, 0.0, s / 2
        for idx in self.info[:-1]:
            lo, u = self._ptmin(idx), x[:, ir]
            pt = 2 * lo * ptmax * u / (2 * lo + ptmax * (1 - u))
            e = s / 2 / pt
            e = torch.log(e + torch.sqrt(e * e - 1)).clamp(max=ETAMAX)
            sh = torch.sinh(e * (2 * x[:, ir + 1] - 1))
            ph = 2 * math.pi * x[:, ir + 2]
            mt = torch.sqrt(pt * pt + m2[idx])
            mom[idx] = torch.stack([mt * torch.sqrt(1 + sh * sh), pt * torch.cos(ph), pt * torch.sin(ph), mt * sh], 1)
            psum, ir = psum + mom[idx], ir + 3
        ptj2, mt, yj = self._last(psum)
        idx = self.info[-1]
        qt = torch.sqrt(m2[idx] + ptj2)
        ymin = -torch.log(s / qt * (1 - mt * torch.exp(-yj)))
        ymax = torch.log(s / qt * (1 - mt * torch.exp(yj)))
        sh = torch.sinh(ymin + x[:, ir] * (ymax - ymin))
        ir += 1
        mom[idx] = torch.stack([qt * torch.sqrt(1 + sh * sh), -psum[:, 1], -psum[:, 2], qt * sh], 1)
        tot, zero = mom[idx] + psum, torch.zeros_like(qt)
        pp, pm = (tot[:, 0] + tot[:, 3]) / 2, (tot[:, 0] - tot[:, 3]) / 2
        for d in self.order:
            p = mom[d.parent.idx]
            ss = _m2(p)
            rs = torch.sqrt(ss.abs())
            k, ct, ph = rs / 2, 2 * x[:, ir] - 1, 2 * math.pi * x[:, ir + 1]
            l, l_perp, n_perp = _axes(p)
            st = torch.sqrt(1 - ct * ct)
            v = l * ct[:, None] + (l_perp * torch.cos(ph)[:, None] + n_perp * torch.sin(ph)[:, None]) * st[:, None]
            q = torch.cat([k[:, None], v * k[:, None]], 1)
            mom[d.child1.idx] = _boost(p, q, True)
            mom[d.child2.idx] = p - mom[d.child1.idx]
            ir += 2
        out = [torch.stack([-pp, zero, zero, -pp], 1), torch.stack([-pm, zero, zero, pm], 1)]
        return torch.stack(out + [mom[1 << i] for i in range(2, self.n_ext)], 1)

    def invert(self, mom):
        """Density and uniforms; density 0 where the chain has no solution."""
        s, ptmax = self.sqrts, self.sqrts / 2
        p = {1 << i: mom[:, i] for i in range(self.n_ext)}
        xs, w = [], torch.ones_like(mom[:, 0, 0])
        for d in self.decays:
            p[d.parent.idx] = p[d.child1.idx] + p[d.child2.idx]
            v, (lo, hi), m, g = _m2(p[d.parent.idx]), self._limits(d), d.parent.mass, d.parent.width
            if g > 0:
                y1, y0 = math.atan((lo - m * m) / (m * g)), math.atan((hi - m * m) / (m * g))
                xs.append((torch.atan((v - m * m) / (m * g)) - y0) / (y1 - y0))
                w = w * (y0 - y1) * ((v - m * m) ** 2 + (m * g) ** 2) / (m * g)
            else:
                ce = 1.0 - 0.99
                xs.append((v ** ce - lo ** ce) / (hi ** ce - lo ** ce))
                w = w * (hi ** ce - lo ** ce) / ce * v ** 0.99
            w = w / (2 * math.pi)
        t, psum = torch.full_like(w, 2 * math.pi), 0.0
        for idx in self.info[:-1]:
            q, lo = p[idx], self._ptmin(idx)
            pt = torch.sqrt(q[:, 1] ** 2 + q[:, 2] ** 2)
            t = t / (16 * math.pi ** 3) * pt * ptmax / 2 / lo / (2 * lo + ptmax) * (2 * lo + pt) ** 2
            xs.append(pt * (ptmax + 2 * lo) / (ptmax * (pt + 2 * lo)))
            e = s / 2 / pt
            e = torch.log(e + torch.sqrt(e * e - 1)).nan_to_num(nan=ETAMAX).clamp(max=ETAMAX)
            t = t * 4 * math.pi * e
            xs.append((_rapidity(q) / e + 1) / 2)
            ph = torch.atan2(q[:, 2], q[:, 1])
            xs.append(torch.where(ph < 0, ph + 2 * math.pi, ph) / (2 * math.pi))
            psum = psum + q
        q = p[self.info[-1]]
        ptj2, mt, yj = self._last(psum)
        qt = torch.sqrt(_m2(q) + ptj2)
        ymin = -torch.log(s / qt * (1 - mt * torch.exp(-yj)))
        ymax = torch.log(s / qt * (1 - mt * torch.exp(yj)))
        fail = torch.isnan(ymin) | torch.isnan(ymax)
        t = torch.where(fail, torch.zeros_like(t), t * (ymax - ymin) / s / s)
        xs.append((_rapidity(q) - ymin) / (ymax - ymin))
        for d in self.order:
            pp, q = p[d.parent.idx], p[d.child1.idx]
            l, l_perp, n_perp = _axes(pp)
            rest = _boost(pp, q, False)[:, 1:]
            xs.append(((rest * l).sum(1) / rest.norm(dim=1) + 1) / 2)
            ph = torch.atan2((q[:, 1:] * n_perp).sum(1), (q[:, 1:] * l_perp).sum(1)) / (2 * math.pi)
            xs.append(torch.where(ph < 0, ph + 1, ph))
            w = w / (8 * math.pi)
        return w * t, torch.stack(xs, 1)


def _inside(mom):
    """The physical region and the cuts."""
    half = SQRTS / 2 * (1 + 1e-12)
    ok = (-mom[:, 0, 0] <= half) & (-mom[:, 1, 0] <= half)
    out = mom[:, 2:]
    pt = torch.sqrt(out[..., 1] ** 2 + out[..., 2] ** 2)
    eta, phi = torch.asinh(out[..., 3] / pt), torch.atan2(out[..., 2], out[..., 1])
    ok &= ((pt >= PTMIN) & (eta.abs() <= ETAMAX)).all(1)
    for i in range(out.shape[1]):
        for j in range(i + 1, out.shape[1]):
            dphi = (phi[:, i] - phi[:, j]).abs()
            dphi = torch.where(dphi > math.pi, 2 * math.pi - dphi, dphi)
            ok &= (eta[:, i] - eta[:, j]) ** 2 + dphi ** 2 >= DELTA_R ** 2
    return ok


def _propagators(mom, kind):
    out, bw = mom[:, 2:], []
    for i in range(out.shape[1]):
        for j in range(i + 1, out.shape[1]):
            bw.append(1 / ((_m2(out[:, i] + out[:, j]) - MZ * MZ) ** 2 + MZ * MZ * GZ * GZ))
    bw = torch.stack(bw, 1)
    top = torch.topk(bw, 2, dim=1)[0].prod(1) if kind == PAIR_TOP2 else bw.sum(1)
    t = _m2(mom[:, :1] + out).abs() + MT * MT
    return top / t.prod(1)


class _MultiChannel:
    def __init__(self, case, cs, grids, alpha):
        self.maps = [_Mapping(cs, c) for c in range(cs.nch)]
        self.cs, self.kind = cs, _integrand(case["n_out"])
        self.grids, self.alpha = torch.as_tensor(grids).cuda(), torch.as_tensor(alpha).cuda()

    def draw(self, key, counters):
        u = _uniforms(key, counters, self.cs.ndims + 1)
        cp = torch.cumsum(self.alpha / self.alpha.sum(), 0)
        cp[-1] = 1.0
        ich = torch.searchsorted(cp, u[:, -1].contiguous())
        mom = torch.empty(len(u), self.cs.n_ext, 4, dtype=torch.float64, device="cuda")
        for c, m in enumerate(self.maps):
            sel = (ich == c).nonzero()[:, 0]
            if len(sel):
                mom[sel] = m.generate(_grid_map(self.grids[c], u[sel, :-1])[0])
        return ich, mom

    def weight(self, mom, ich):
        """Combined weight, densities, and the chosen channel's uniforms."""
        acc, bins = 0.0, self.grids.shape[2] - 1
        dens, mine = [], torch.zeros(len(mom), self.cs.ndims, dtype=torch.float64, device="cuda")
        for c, m in enumerate(self.maps):
            d, x = m.invert(mom)
            g, vw = self.grids[c], torch.ones_like(d)
            b = _bins_of(g, x)
            for j in range(x.shape[1]):
                vw = vw * (g[j][b[:, j] + 1] - g[j][b[:, j]]) * bins
            acc = acc + self.alpha[c] / d / vw
            dens.append(d)
            mine = torch.where((ich == c)[:, None], x, mine)
        return 1 / acc, torch.stack(dens, 1), mine


def _parts(n, width):
    """Counter ranges small enough for the tensors of one part."""
    step = max(1 << 14, min(1 << 19, (1 << 26) // width))
    return [(k, min(k + step, n)) for k in range(0, n, step)]


def _exact_iterate(case, mc, seed):
    n, cs, bins = case["n"], mc.cs, case["bins"]
    hist = torch.zeros(cs.nch * cs.ndims * bins, dtype=torch.float64, device="cuda")
    train = torch.zeros(cs.nch, dtype=torch.float64, device="cuda")
    got, tried, values, at = 0, 0, [], 0
    while got < n:
        step = max(1 << 14, min(1 << 19, 2 * (n - got)))
        ich, mom = mc.draw(seed, torch.arange(at, at + step, dtype=torch.int64, device="cuda"))
        keep = _inside(mom).nonzero()[:, 0]
        if got + len(keep) >= n:
            keep = keep[:n - got]
            tried = at + int(keep[-1]) + 1
        got, at = got + len(keep), at + step
        for lo, hi in _parts(len(keep), cs.nch * cs.ndims):
            p, c = mom[keep[lo:hi]], ich[keep[lo:hi]]
            w, dens, x = mc.weight(p, c)
            v = _propagators(p, mc.kind) * w
            values.append(v)
            train += ((v * v * w)[:, None] / dens).sum(0)
            inner = mc.grids[:, :, :-1].contiguous()
            b = torch.stack([torch.searchsorted(inner[c, j], x[:, j:j + 1].contiguous())[:, 0] - 1
                             for j in range(cs.ndims)], 1).clamp(min=0)
            slot = (c[:, None] * cs.ndims + torch.arange(cs.ndims, device="cuda")) * bins + b
            hist.index_add_(0, slot.reshape(-1), (v * v)[:, None].expand(-1, cs.ndims).reshape(-1))
    v = torch.cat(values)
    par = workloads.mc_params(n)
    a = mc.alpha * train ** par.beta
    a = torch.clamp(a / a.sum(), min=par.min_alpha)
    grids, h = mc.grids.cpu().numpy().copy(), hist.reshape(cs.nch, cs.ndims, bins).cpu().numpy()
    for c in range(cs.nch):
        for d in range(cs.ndims):
            if h[c].any():
                grids[c, d] = _adapt(grids[c, d], h[c, d], par.grid_alpha)
    return dict(zip(STATS, _stats(v, tried - n)), wmax=np.float64(v.max().item()), grids=grids,
                alpha=(a / a.sum()).cpu().numpy(), counts=np.array([tried, n, tried - n, 0], dtype=np.int64))


def _exact_events(case, mc, seed):
    mom, wgt, ich = [], [], []
    total, vmax = 0.0, 0.0
    for lo, hi in _parts(case["n"], mc.cs.nch * mc.cs.ndims):
        k = torch.arange(lo, hi, dtype=torch.int64, device="cuda")
        c, p = mc.draw(seed, k)
        if case["kind"] == "unweighted":
            inside = _inside(p)
            k, c, p = k[inside], c[inside], p[inside]
        v = _propagators(p, mc.kind) * mc.weight(p, c)[0]
        if case["kind"] == "unweighted":
            total, vmax = total + float(v.sum()), max(vmax, float(v.max()))
            keep = _uniforms(seed, k, 1, stream=1)[:, 0] * W_MAX[case["n_out"]] < v.abs()
            c, p, v = c[keep], p[keep], v[keep].sign() * v[keep].abs().clamp(min=W_MAX[case["n_out"]])
        else:
            v = torch.where(torch.isfinite(v), v, torch.zeros_like(v))
        mom.append(p), wgt.append(v), ich.append(c)
    out = {"momenta": torch.cat(mom), "weight": torch.cat(wgt), "channel": torch.cat(ich).int()}
    if case["kind"] == "unweighted":
        out.update(sum=np.float64(total), max=np.float64(vmax), kept=len(out["weight"]))
        rows = max(1024, case["n"] // 16)
        for k in ("momenta", "weight", "channel"):  # the buffers' rows past the kept events stay zero
            full = torch.zeros((rows,) + out[k].shape[1:], dtype=out[k].dtype, device="cuda")
            full[:len(out[k])] = out[k][:rows]
            out[k] = full
    elif case["n_out"] >= 3:
        # points outside the physical region have no density in some
        # channels: their weights hang on rounding alone
        out["weight"] = None
    return out


def _exact_camels(case, seed):
    """The camel tasks of a batch: each a Vegas object of its own."""
    out = np.empty((case["iterations"], case["camels"], 6))
    tasks = workloads.batched_tasks(int(seed), case["camels"], case["multichannels"], scale=case["scale"])
    for t in range(case["camels"]):
        task = tasks[t]
        c = {"dims": task["dims"], "bins": task["bins"]}
        edges = np.tile(np.arange(c["bins"] + 1) / c["bins"], (1, c["dims"], 1))
        for it in range(case["iterations"]):
            k = (it << 32) + torch.arange(task["ncalls"], dtype=torch.int64, device="cuda")
            out[it, t], hist = _exact_vegas(c, np.array(task["params"]), edges, int(seed) + t, k)
            edges = np.stack([[_adapt(edges[0, d], hist[d], task["grid_alpha"]) for d in range(c["dims"])]])
    return out


def _spline(theta, v, inverse):
    """Rational-quadratic spline on [0, 1] with 16 bins: value and log slope
    of the density direction."""
    k = 16
    w = 1e-3 + (1 - k * 1e-3) * torch.softmax(theta[..., :k], -1)
    h = 1e-3 + (1 - k * 1e-3) * torch.softmax(theta[..., k:2 * k], -1)
    d = 1e-3 + torch.nn.functional.softplus(theta[..., 2 * k:])
    xk, yk = (torch.nn.functional.pad(torch.cumsum(t, -1), (1, 0)) for t in (w, h))
    i = ((yk if inverse else xk)[..., 1:k] <= v[..., None]).sum(-1, keepdim=True)
    wk, hk, x0, y0, d0 = (torch.gather(t, -1, i)[..., 0] for t in (w, h, xk, yk, d))
    d1, s = torch.gather(d, -1, i + 1)[..., 0], hk / wk
    dl = d0 + d1 - 2 * s
    if inverse:
        dy = v - y0
        a, b, c = hk * (s - d0) + dy * dl, hk * d0 - dy * dl, -s * dy
        xi = 2 * c / (-b - torch.sqrt((b * b - 4 * a * c).clamp(min=0)))
        out = x0 + xi * wk
    else:
        xi = (v - x0) / wk
    om = xi * (1 - xi)
    bb = s + dl * om
    if not inverse:
        out = y0 + hk * (s * xi * xi + d0 * om) / bb
    slope = d1 * xi * xi + 2 * s * om + d0 * (1 - xi) ** 2
    return out, 2 * torch.log(s) + torch.log(slope) - 2 * torch.log(bb)


def _bf16(t):
    return t.to(torch.bfloat16).to(t.dtype)


class _Product(torch.autograd.Function):
    """a b^T of bf16 operands (as include/chili_gpu.h defines the networks'
    products), everything else in 64 bits."""

    @staticmethod
    def forward(ctx, a, b):
        ctx.save_for_backward(_bf16(a), _bf16(b))
        return _bf16(a) @ _bf16(b).T

    @staticmethod
    def backward(ctx, g):
        a, b = ctx.saved_tensors
        return _bf16(g) @ b, _bf16(g).T @ a


def _flow(case, prm, x, ch, inverse):
    """The coupling layers in one direction: coordinates and log q."""
    logq, last = 0.0, case["hidden"] - 1
    masks = _flow_masks(x.shape[1], case["layers"])
    for layer in (reversed(range(len(masks))) if inverse else range(len(masks))):
        m = torch.from_numpy(masks[layer]).cuda()
        def lrelu(t):
            t = torch.nn.functional.leaky_relu(t, 0.01)
            return torch.cat([t[:, :last], torch.ones_like(t[:, :1])], 1)
        h = lrelu(_Product.apply(2 * x[:, m] - 1, prm["W1_%d" % layer]) + _bf16(prm["E_%d" % layer])[ch])
        for k in range(case["depth"] - 1):
            h = lrelu(_Product.apply(h, prm["W2_%d_%d" % (layer, k)]))
        theta = _Product.apply(h, prm["W3_%d" % layer]).reshape(len(x), -1, 49)
        y, lj = _spline(theta, x[:, ~m], inverse)
        z = x.clone()
        z[:, ~m] = y
        x, logq = z.clamp(0.0, 1.0), logq + lj.sum(1)
    return x, logq


def _exact_flow(case, seed):
    cs = _channel_set(case["n_out"])
    flat = torch.from_numpy(_flow_params(case, cs.ndims, cs.nch, seed)).cuda().double()
    batch = [t.double() if t.is_floating_point() else t.long() for t in _flow_batch(case, cs.ndims, cs.nch, seed)]
    grad = case["kind"] == "flow_grad"
    flat.requires_grad_(grad)
    prm, at = {}, 0
    for name, shape in _flow_shapes(case, cs.ndims, cs.nch):
        prm[name] = flat[at:at + math.prod(shape)].reshape(shape)
        at += math.prod(shape)
    us, logqs, loss = [], [], 0.0
    logbeta = torch.log(torch.from_numpy(_trained_alpha(cs, _rng(seed))).cuda())
    for lo in range(0, case["n"], 1 << 14):
        part = [t[lo:lo + (1 << 14)] for t in batch]
        u, logq = _flow(case, prm, part[0], part[1], not grad)
        if not grad:
            us.append(u), logqs.append(logq)
            continue
        _, ch, logf, feat, prior = part
        h = torch.nn.functional.leaky_relu(_Product.apply(feat, prm["A1"]) + prm["c1"], 0.01)
        h = torch.nn.functional.leaky_relu(_Product.apply(h, prm["A2"]) + prm["c2"], 0.01)
        logalpha = torch.log_softmax(_Product.apply(h, prm["A3"]) + prm["c3"] + prior, 1)
        la = torch.gather(logalpha, 1, ch[:, None])[:, 0]
        term = torch.exp(2 * la + 2 * logf - 2 * logbeta[ch] - logq).sum() / case["n"]
        term.backward(retain_graph=True)
        loss += float(term.detach())
    if not grad:
        return {"u": torch.cat(us), "logq": torch.cat(logqs)}
    return {"loss": loss, "grad": flat.grad}


def exact(case, seed):
    kind, seed = case["kind"], int(seed)
    if kind in ("flow_grad", "flow_sample"):
        return _exact_flow(case, seed)
    with torch.no_grad():
        if kind in ("vegas", "points"):
            params = _camel(case, seed)
            edges = _camel_grid(case, params)
            k = torch.arange(case["n"], dtype=torch.int64, device="cuda")
            if kind == "points":
                return _exact_vegas(case, params, edges, seed, k, want_points=True)
            stats, hist = _exact_vegas(case, params, edges, seed, k)
            grid = np.stack([[_adapt(edges[0, d], hist[d], 1.5) for d in range(case["dims"])]])
            return dict(zip(STATS, stats), grid=grid)
        if kind == "batch":
            # the multichannel tasks run outside the cuts too, where a weight
            # can hang on rounding alone: no value of theirs is exact
            return {"camel": _by_stat(_exact_camels(case, seed)), "multichannel": None}
        cs = _channel_set(case["n_out"])
        if kind == "evaluate":
            m = _Mapping(cs, case["channel"] % cs.nch)
            g = torch.Generator(device="cuda").manual_seed(seed)
            u = torch.rand(case["n"], cs.ndims, generator=g, dtype=torch.float64, device="cuda")
            mom = m.generate(u)
            v = _propagators(mom, _integrand(case["n_out"])) * m.invert(mom)[0]
            return {"value": torch.where(torch.isnan(mom[:, 0, 0]) | torch.isnan(v), torch.zeros_like(v), v)}
        rng = _rng(seed)
        grids, alpha = _trained_grids(cs, case["bins"], rng), _trained_alpha(cs, rng)
        mc = _MultiChannel(case, cs, grids, alpha)
        if kind == "iterate":
            return _exact_iterate(case, mc, seed)
        if kind in ("events", "unweighted"):
            return _exact_events(case, mc, seed)
        mom, ich = _momenta(case["n"], case["n_out"], seed), _channel_draw(case["n"], cs.nch, seed).long()
        got = [mc.weight(mom[lo:hi], ich[lo:hi]) for lo, hi in _parts(case["n"], cs.nch * cs.ndims)]
        return dict(zip(("weight", "density", "x"), (torch.cat(t) for t in zip(*got))))
