"""The work whose time this repository watches: calls a user of the engine makes,
over the range of networks it is used on.

listed()            the named cases
draw(rng)           one more case of the same ranges
prepare(case, seed) what a program holds before the call: a built, running network
run(state)          one pass through the public entry points, and its results
work(case)          the bytes and operations one pass cannot do without
exact(case, seed)   the results in 64 bits by plain numpy, where a 64-bit run means anything

A network's spikes are chaotic: after a few hundred cycles a run in 64 bits has
other spikes than any run in 32 bits, so exact() gives values for the short run
from rest and for the predictor's training only (a few steps of it: the sign a
rounded unit takes at zero sends longer trainings apart as well). The other cases'
results are reproducible to the bit (exact integer sums, fixed order of every
rounding).
"""
import math

import numpy as np
import torch

import bsim_b200 as B
from bsim_b200 import workloads as W

DT = 1.0e-4
LIF = [-0.065, -0.065, -0.065, 0.25e-9, 20e-3, 2e-3, 5e-3, 10e-3, -0.050, 0.0]
DELIVERY = {"push": B.DELIVERY_PUSH, "pull": B.DELIVERY_PULL, "auto": B.DELIVERY_AUTO, "tile": B.DELIVERY_TILE}


def listed():
    return [
        # A controller in a loop with a small network: every 1 ms of simulated time it reads the
        # state and the spike counts. The smallest call: launches and host round trips.
        {"name": "closed_loop_1k", "kind": "loop", "n": 1007, "degree": 20, "delay": 6, "settle": 100, "steps": 10},
        # The reference's CPU-sized test network (10 x 1,000, ~100 Hz, delays 1-6), with the
        # defaults of the engine: push delivery. A few microseconds per cycle.
        {"name": "standard_10k", "kind": "net", "n_pop": 10, "pop": 1000, "rate": 100, "delay": 6, "delivery": "push",
         "settle": 1000, "steps": 1000},
        # Input drives: Poisson and constant sources feeding LIF neurons, from host arrays.
        {"name": "poisson_driven_5k", "kind": "drive", "n": 5003, "degree": 60, "delay": 15, "settle": 300,
         "steps": 500},
        # Validation against the reference simulator, bit for bit: sums in its own order.
        {"name": "ordered_10k", "kind": "net", "n_pop": 10, "pop": 1000, "rate": 100, "delay": 6,
         "delivery": "ordered", "settle": 300, "steps": 300},
        # The shape of the reference's own benchmark program: all-to-all chain, 1-step delays,
        # populations that fire together.
        {"name": "all_to_all_20k", "kind": "net", "n_pop": 20, "pop": 1000, "rate": 100, "delay": 1, "p": 1.0,
         "delivery": "push", "settle": 500, "steps": 500},
        # A recorded run: every spike of 100 cycles (10 ms) of a 250,000-neuron network, read back
        # as a raster into a page-locked buffer.
        {"name": "record_250k", "kind": "record", "n_pop": 25, "pop": 10000, "rate": 500, "delay": 6, "i_max": 30e-9,
         "delivery": "tile", "settle": 2000, "steps": 100},
        # A parameter sweep: 16 networks of uneven sizes, rates and delays in one engine.
        {"name": "batched_16", "kind": "batch", "nets": 16, "mix": 7, "delivery": "tile", "settle": 300,
         "steps": 100},
        # Dense firing with long delays at a quarter of the full size, tiled delivery.
        {"name": "dense_250k", "kind": "net", "n_pop": 50, "pop": 5000, "rate": 2000, "delay": 50, "i_max": 62.5e-9,
         "delivery": "tile", "settle": 500, "steps": 200},
        # Drive that swings between ~10 Hz and ~900 Hz; push or tiled chosen per cycle.
        {"name": "square_wave_500k", "kind": "wave", "n_pop": 50, "pop": 10000, "rate": 500, "delay": 20,
         "i_max": 2.5e-9, "scale": 32.0, "half": 250, "delivery": "auto", "settle": 500, "steps": 500},
        # The headline network: 1e6 neurons, 1.19e9 synapses, ~560 Hz, tiled delivery.
        {"name": "plain_1m", "kind": "net", "n_pop": 100, "pop": 10000, "rate": 500, "delay": 6, "i_max": 30e-9,
         "delivery": "tile", "settle": 3000, "steps": 400},
        # The dense configuration at full size (2.36e9 synapses, ~2 kHz), pushed as the benchmark does.
        {"name": "dense_1m", "kind": "net", "n_pop": 50, "pop": 20000, "rate": 2000, "delay": 50, "i_max": 62.5e-9,
         "delivery": "push", "settle": 200, "steps": 40},
        # Training of the firing predictor on recorded rates (host arrays in, weights out), with the
        # benchmark's batch size.
        {"name": "predictor_training", "kind": "mlp", "n": 65001, "batch": 8192, "epochs": 1},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["loop", "net", "net", "net", "ordered", "drive", "record", "batch", "wave", "mlp"])
    if kind == "loop":
        return {"kind": "loop", "n": _log(rng, 50, 4000), "degree": rng.randint(3, 40), "delay": rng.randint(1, 16),
                "settle": 100, "steps": rng.randint(1, 20)}
    if kind == "drive":
        return {"kind": "drive", "n": _log(rng, 500, 20000), "degree": rng.randint(10, 80),
                "delay": rng.randint(1, 30), "settle": 200, "steps": rng.randint(100, 500)}
    if kind == "mlp":
        batch = rng.choice([512, 1000, 4096, 8192, 10007])  # a few steps: see exact()
        return {"kind": "mlp", "n": int(batch * rng.uniform(1.0, 9.0)), "batch": batch, "epochs": 1}
    if kind == "batch":
        return {"kind": "batch", "nets": rng.randint(3, 16), "mix": rng.randint(1, 1000), "delivery": "tile",
                "settle": 200, "steps": rng.randint(30, 100)}
    if kind == "ordered":
        return {"kind": "net", "n_pop": rng.randint(3, 12), "pop": _log(rng, 200, 1500), "rate": rng.choice([100, 500]),
                "delay": rng.randint(1, 20), "delivery": "ordered", "settle": 200, "steps": rng.randint(50, 300)}
    n_pop, pop = rng.randint(4, 60), _log(rng, 200, 12000)
    while n_pop > 4 and 0.12 * n_pop * pop * pop > 6e8:  # synapses: at most half the headline network's
        n_pop -= 1
    syn = 0.12 * n_pop * pop * pop
    steps = max(20, min(500, int(3e11 / (syn + 2e8))))
    c = {"kind": kind, "n_pop": n_pop, "pop": pop, "rate": rng.choice([100, 500, 2000]),
         "delay": rng.choice([1, rng.randint(2, 10), rng.randint(11, 60)]), "delivery": rng.choice(["push", "tile"]),
         "settle": 500, "steps": steps}
    if kind == "record":
        c.update(steps=min(steps, 100))
    if kind == "wave":
        c.update(rate=500, i_max=2.5e-9, scale=32.0, half=rng.randint(50, 250), delivery="auto")
    return c


# ---------------------------------------------------------------------------
# Networks
# ---------------------------------------------------------------------------
def _specs(case, seed):
    if case["kind"] == "batch":
        specs, _ = W.batched(case["nets"], case["mix"])
        for k, sp in enumerate(specs):  # the sizes of the mix, other networks for another seed
            sp.seed = 1000003 * (seed + 1) + k
        return specs
    sp = W.cuba(case["n_pop"], case["pop"], case["rate"], case["delay"], seed=seed + 1, i_max=case.get("i_max"))
    p = case.get("p", 0.1)
    sp.p_conn = p
    sp.w_max *= 0.1 / p  # the same mean input at another connection probability
    if case["kind"] == "wave":
        sp.drive_scale, sp.drive_half_period = case["scale"], case["half"]
    return [sp]


def _arrays(case, seed):
    """A random network as host arrays: LIF neurons, and for "drive" the first tenth of the
    neurons are Poisson sources (mean gap 40 cycles) and the next fiftieth constant ones."""
    rng = np.random.default_rng(seed)
    n, s = case["n"], case["n"] * case["degree"]
    params = np.tile(np.array(LIF, np.float32), (n, 1))
    params[:, 0] = rng.uniform(-0.065, -0.0505, n)
    params[:, 9] = rng.uniform(0.1e-9, 1.5e-9, n)
    kind = np.zeros(n, np.uint8)
    if case["kind"] == "drive":
        n_p, n_c = n // 10, n // 50
        kind[:n_p], kind[n_p:n_p + n_c] = B.NEURON_POISSON, B.NEURON_CONSTANT
        params[:n_p + n_c] = 0.0
        params[:n_p, 0], params[:n_p, 3] = rng.uniform(10.0, 70.0, n_p), 1e6
        params[n_p:n_p + n_c, 0], params[n_p:n_p + n_c, 2] = rng.uniform(0.005, 0.05, n_c), 1e6
    src, dst = rng.integers(0, n, s).astype(np.int32), rng.integers(0, n, s).astype(np.int32)
    w = np.where(rng.random(s) < 0.8, rng.uniform(0.0, 1e-10, s), -rng.uniform(0.0, 4e-10, s)).astype(np.float32)
    d = rng.integers(1, case["delay"] + 1, s).astype(np.int32)
    return params, kind, src, dst, w, d


def prepare(case, seed):
    if case["kind"] == "mlp":
        x, y = _samples(case, seed)
        return {"case": case, "x": x, "y": y, "params": B.mlp_init(seed + 1)}
    if case["kind"] in ("loop", "drive"):
        params, kind, src, dst, w, d = _arrays(case, seed)
        eng = B.Engine.from_arrays(params, src, dst, w, d, DT, kind=kind if case["kind"] == "drive" else None,
                                   input_seed=seed)
    else:
        if case["delivery"] == "ordered":
            opts = B.options(accumulate=B.ACC_ORDERED)
        else:
            opts = B.options(delivery=DELIVERY[case["delivery"]])
        eng = B.Engine.generated(_specs(case, seed), DT, opts=opts)
        if case["delivery"] == "auto":  # cost models of the two modes, as fitted once on such networks
            eng.set_predictor(None, cost_push=[53000.0, 0.0065], cost_tile=[109000.0, 0.0038])
    eng.run(case["settle"])
    state = {"case": case, "eng": eng}
    n = eng.info().n_neurons
    state["counts"] = torch.zeros(n, dtype=torch.int32).pin_memory().numpy()
    if case["kind"] == "record":
        # room for every neuron firing as often as its refractory period lets it
        state["cap"] = n * case["steps"] // {100: 20, 500: 5, 2000: 2}[case["rate"]]
        state["ids"] = torch.zeros(state["cap"], dtype=torch.int32).pin_memory().numpy()
        eng.record(case["steps"], state["cap"])
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "mlp":
        params, loss = B.mlp_train(state["params"], state["x"], state["y"], epochs=case["epochs"],
                                   batch=case["batch"], lr=2e-3, seed=1)
        return {"params": params, "loss": loss}
    eng = state["eng"]
    if case["kind"] == "record":
        eng.record(case["steps"], state["cap"])
        eng.run(case["steps"])
        rows = eng.raster(out=state["ids"])
        per_cycle = np.array([len(r) for r in rows], np.int64)
        # the buffer as a whole (its head holds the spikes): one size whatever was fired
        return {"spikes_per_cycle": per_cycle, "ids": state["ids"], "count": eng.fire_count(out=state["counts"])}
    eng.run(case["steps"])
    st = eng.state()
    st["count"] = eng.fire_count(out=state["counts"])
    return st


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def _size(sp):
    """Neurons and expected synapses of one generated network (chain and remote projections)."""
    n_proj = sp.n_pop - 1 + int(sp.remote_frac * sp.n_pop + 0.5)
    return sp.n_pop * sp.pop_size, n_proj * float(sp.pop_size) ** 2 * sp.p_conn


def work(case):
    if case["kind"] == "mlp":
        # weights of the three layers: forward, and twice as much backward; samples and weights moved once
        macs = B.MLP_IN * B.MLP_HIDDEN + B.MLP_HIDDEN * B.MLP_HIDDEN + B.MLP_HIDDEN
        batches = case["epochs"] * (case["n"] // min(case["batch"], case["n"]))
        return {"bytes": case["epochs"] * case["n"] * 4.0 * (B.MLP_IN + 1) + batches * B.MLP_PARAMS * 24.0,
                "flops": case["epochs"] * case["n"] * 6.0 * macs}
    neurons = spikes = events = 0.0  # per cycle
    if case["kind"] in ("loop", "drive"):
        neurons = case["n"]
        spikes = neurons * 40.0 * DT
        events = spikes * case["degree"]
    else:
        # mean rates of the presets, measured (Hz): the refractory period sets the order of magnitude
        hz = {100: 100.0, 500: 520.0, 2000: 2000.0}
        rates = [{20: 100.0, 5: 520.0, 2: 2000.0}[int(round(sp.tau_refrac * 1e4))] for sp in _specs(case, 0)] \
            if case["kind"] == "batch" else [450.0 if case["kind"] == "wave" else hz[case["rate"]]]
        for sp, r in zip(_specs(case, 0), rates):
            n, s = _size(sp)
            neurons += n
            spikes += n * r * DT
            events += s * r * DT
    k = case["steps"]
    # state read and written, drive, input read and cleared: 52 bytes a neuron; target and weight of
    # each delivered synapse: 8 bytes; a fired id written and read: 8 bytes
    return {"bytes": k * (52.0 * neurons + 8.0 * events + 8.0 * spikes), "flops": k * (12.0 * neurons + 2.0 * events)}


# ---------------------------------------------------------------------------
# The same results in 64 bits
# ---------------------------------------------------------------------------
def _mix64(x):
    with np.errstate(over="ignore"):
        x = x ^ (x >> np.uint64(30))
        x = x * np.uint64(0xbf58476d1ce4e5b9)
        x = x ^ (x >> np.uint64(27))
        x = x * np.uint64(0x94d049bb133111eb)
        return x ^ (x >> np.uint64(31))


def _hash3(seed, a, b):
    with np.errstate(over="ignore"):
        h = _mix64(np.uint64(seed) ^ (np.uint64(a) * np.uint64(0x9e3779b97f4a7c15)))
        return _mix64(h + b * np.uint64(0xd1b54a32d192ed03) + np.uint64(1))


def _samples(case, seed):
    """Rates of 8 past cycles and a mean in-degree, and the rate two cycles on: a slow
    oscillation per sample with noise, as population rates show."""
    rng = np.random.default_rng(seed)
    n = case["n"]
    level, phase, noise = rng.uniform(0.0, 6.0, n), rng.uniform(0.0, 2 * np.pi, n), rng.normal(0, 0.05, (n, 9))
    at = np.concatenate([-1.0 - np.arange(8), [1.0]])
    r = np.maximum(level[:, None] * (1.0 + 0.5 * np.sin(phase[:, None] + 0.15 * at)) + noise, 0.0)
    x = np.concatenate([r[:, :8], rng.uniform(0.9, 1.5, (n, 1))], 1).astype(np.float32)
    return x, r[:, 8].astype(np.float32)


def _train64(case, seed):
    H, IN = B.MLP_HIDDEN, B.MLP_IN
    x, y = (a.astype(np.float64) for a in _samples(case, seed))
    p = np.zeros(B.MLP_PARAMS)
    at = {}
    o = 0
    for name, shape in (("W1", (H, IN)), ("b1", (H,)), ("W2", (H, H)), ("b2", (H,)), ("W3", (H,)), ("b3", (1,))):
        at[name] = (o, shape)
        o += int(np.prod(shape))
    v = {k: p[a:a + int(np.prod(s))].reshape(s) for k, (a, s) in at.items()}  # views into p
    for name, fan_in, fan_out, salt in (("W1", IN, H, 1), ("W2", H, H, 2), ("W3", H, 1, 3)):
        m = int(np.prod(v[name].shape))
        u = (_hash3(seed + 1, salt, np.arange(m, dtype=np.uint64)) >> np.uint64(40)).astype(np.float32)
        a = np.sqrt(np.float32(6.0) / np.float32(fan_in + fan_out))
        v[name][...] = ((np.float32(2.0) * (u * np.float32(1.0 / 16777216.0)) - np.float32(1.0)) * a).reshape(v[name].shape)
    g, m1, m2 = np.zeros_like(p), np.zeros_like(p), np.zeros_like(p)
    gv = {k: g[a:a + int(np.prod(s))].reshape(s) for k, (a, s) in at.items()}
    lr, b1, b2 = float(np.float32(2e-3)), float(np.float32(0.9)), float(np.float32(0.999))

    def backward(xb, yb):
        z1 = xb @ v["W1"].T + v["b1"]
        h1 = np.maximum(z1, 0.0)
        h2 = np.maximum(h1 @ v["W2"].T + v["b2"], 0.0)
        e = h2 @ v["W3"] + v["b3"][0] - yb
        dy = 2.0 * e / len(e)
        dz2 = dy[:, None] * v["W3"] * (h2 > 0)
        dz1 = (dz2 @ v["W2"]) * (h1 > 0)
        gv["W3"][...], gv["b3"][...] = h2.T @ dy, dy.sum()
        gv["W2"][...], gv["b2"][...] = dz2.T @ h1, dz2.sum(0)
        gv["W1"][...], gv["b1"][...] = dz1.T @ xb, dz1.sum(0)
        return float(np.mean(e * e))

    n, bs, idx, step = case["n"], min(case["batch"], case["n"]), list(range(case["n"])), 0
    for ep in range(case["epochs"]):
        h = _hash3(1, ep, np.arange(n, dtype=np.uint64))
        js = (h % (np.arange(n, dtype=np.uint64) + np.uint64(1))).tolist()
        for i in range(n - 1, 0, -1):
            idx[i], idx[js[i]] = idx[js[i]], idx[i]
        order = np.array(idx)
        for b0 in range(0, n - bs + 1, bs):
            backward(x[order[b0:b0 + bs]], y[order[b0:b0 + bs]])
            step += 1
            m1[:] = b1 * m1 + (1.0 - b1) * g
            m2[:] = b2 * m2 + (1.0 - b2) * g * g
            p -= lr * (m1 / (1.0 - b1 ** step)) / (np.sqrt(m2 / (1.0 - b2 ** step)) + 1e-8)
    return {"params": p, "loss": backward(x, y)}


def _loop64(case, seed):
    """The membrane equations from rest, the synaptic input of a spike at t - d entering the
    currents in cycle t + 1: settle + steps cycles."""
    params, _, src, dst, w, d = _arrays(case, seed)
    P = params.astype(np.float64)
    v, rest, reset, cm, tau_m, refr, tE, tI, thr, ioff = P.T
    dt = float(np.float32(DT))
    rm = tau_m / cm
    Cm, CE, CI = np.exp(-dt / tau_m), np.exp(-dt / tE), np.exp(-dt / tI)
    v_tmp = (ioff * rm + rest) * (1.0 - Cm)
    C_E, C_I = rm * tE / (tE - tau_m) * (CE - Cm), rm * tI / (tI - tau_m) * (CI - Cm)
    r_time = (params[:, 5] / np.float32(DT)).astype(np.int32)
    v, n = v.copy(), case["n"]
    iE, iI, left, count = np.zeros(n), np.zeros(n), np.zeros(n, np.int32), np.zeros(n, np.int32)
    T, D = case["settle"] + case["steps"], case["delay"]
    inE, inI = np.zeros((T + D + 2, n)), np.zeros((T + D + 2, n))
    order = np.argsort(src, kind="stable")
    src, dst, w, d = src[order], dst[order], w[order].astype(np.float64), d[order]
    first = np.searchsorted(src, np.arange(n + 1))
    for t in range(T):
        free = left == 0
        left[~free] -= 1
        nv = Cm * v + v_tmp + iE * C_E + iI * C_I
        fire = free & (nv >= thr)
        keep = free & ~fire
        iE = np.where(free, CE * iE, iE) + np.where(keep, inE[t], 0.0)
        iI = np.where(free, CI * iI, iI) + np.where(keep, inI[t], 0.0)
        v = np.where(fire, reset, np.where(free, nv, v))
        left[fire] = r_time[fire] - 1
        count += fire
        for s in np.nonzero(fire)[0]:
            k = slice(first[s], first[s + 1])
            pos = w[k] >= 0
            np.add.at(inE, (t + d[k][pos] + 1, dst[k][pos]), w[k][pos])
            np.add.at(inI, (t + d[k][~pos] + 1, dst[k][~pos]), w[k][~pos])
    return {"v": v, "i_E": iE, "i_I": iI, "refrac": left, "count": count}


def exact(case, seed):
    if case["kind"] == "mlp":
        return _train64(case, seed)
    if case["kind"] == "loop":
        return _loop64(case, seed)
    return None
