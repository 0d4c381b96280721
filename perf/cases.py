"""The work that a user of the simulator has it do, as cases to be timed.

Two kinds of case:

  "sim"      a simulation handle (``Simulation``) advanced by one trial of ``steps`` exchange
             steps per pass.  The networks are the synthetic scaffolds that the tests and the
             benchmark use (configurations 1 and 2 and ten times 2, population sizes times a
             scale); initial potentials and stimulus streams come from the seed.  A pass hands
             back what such a program reads at the end of a trial: spike counts per population
             and step, the raster where it is recorded, the cells' potentials, conductances and
             refractory counts, and the plastic values.
  "deliver"  the standalone delivery operator on caller-owned device buffers.

Connectivity depends on the case alone, as a program runs many trials on one network.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PACKAGE = os.path.join(_ROOT, "cerebellar-scaffold-model-simulation-on-gpu_gb300")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

import scaffold_gb300 as sg  # noqa: E402

# Cells, input cells and synapses of each configuration at scale 1.
SIZES = {1: (9256, 512, 196_960), 2: (92_550, 2_400, 2_731_520)}
DT_MS = 0.1
MEAN_RATE_HZ = 7.0  # events per synapse and second that the frozen drives settle at

_SIM = dict(kind="sim", arch=2, scale=1.0, instances=1, bf16=False, driver="persistent", prop="push",
            substeps=1, steps=1000, raster=False, state=True, rates=False, plastic=False)


def _sim(**over):
    return dict(_SIM, **over)


def listed():
    return [
        # A controller that sets the mossy rate and reads the counts every millisecond: the
        # smallest call, launch and host latency.
        _sim(name="control_loop", arch=1, steps=10, state=False, rates=True),
        # A trial of 0.1 s on the 9k-cell net, the size for parameter studies.
        _sim(name="trial_9k", arch=1, steps=1000),
        # The headline: the 92k-cell scaffold, 32-bit weights.
        _sim(name="trial_92k", steps=3000),
        # The same with 16-bit weights and every spike recorded, as the reference records it.
        _sim(name="raster_92k_bf16", bf16=True, raster=True, state=False, steps=1000),
        # The default driver (per-step kernels in a graph), event-driven.
        _sim(name="graph_92k", driver="graph", steps=500),
        # The reference's exchange step: 1 ms of ten substeps, at an odd size.
        _sim(name="ms_steps_97k", scale=1.0483, substeps=10, steps=300),
        # Dense pull of every projection, the reference's own propagation.
        _sim(name="dense_92k_bf16", bf16=True, prop="pull", steps=1000),
        # Dense pull at a size whose tables pass the L2, per-step kernels.
        _sim(name="dense_1m4_graph", scale=15.0, bf16=True, driver="graph", prop="pull", steps=200),
        # Teacher-gated depression of the parallel fibres (learning).
        _sim(name="learning_92k", plastic=True, steps=4000),
        # A batch of instances of different sizes in one handle.
        _sim(name="batch_32", instances=32, bf16=True, steps=1500),
        # One ten-times scaffold.
        _sim(name="trial_925k", scale=10.0, bf16=True, steps=2000),
        # Delivery of one step's spikes for a program with its own neuron update.
        dict(name="deliver_92k", kind="deliver", cells=92_550, fan=29.5, bf16=False, active=0.005,
             slots=5),
    ]


def draw(rng):
    """One more case of the same ranges."""
    def log(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    bf16 = rng.random() < 0.5
    kind = rng.choice(["trial", "trial", "trial", "batch", "ms", "graph", "dense", "learning",
                       "deliver"])
    if kind == "deliver":
        return dict(kind="deliver", cells=int(log(2_000, 900_000)), fan=round(log(4, 60), 2), bf16=bf16,
                    active=round(log(0.0005, 0.05), 5), slots=rng.choice([5, 6, 9, 16]))
    if kind == "trial":
        scale = log(0.05, 9.0)
        steps = int(log(10, 3000)) if scale < 1.6 else int(log(50, 900))
        if rng.random() < 0.35:
            return _sim(arch=1, scale=round(log(0.1, 12.0), 4), bf16=bf16, steps=int(log(10, 2000)),
                        raster=rng.random() < 0.3)
        return _sim(scale=round(scale, 4), bf16=bf16, steps=steps, raster=scale < 3.0 and rng.random() < 0.25)
    if kind == "batch":
        arch = rng.choice([1, 2])
        n = int(log(2, 24))
        return _sim(arch=arch, instances=n, scale=round(log(0.15, 1.0), 4), bf16=bf16, steps=int(log(30, 600)))
    if kind == "ms":
        return _sim(arch=rng.choice([1, 2]), scale=round(log(0.2, 2.0), 4), bf16=bf16, substeps=10,
                    driver=rng.choice(["persistent", "persistent", "graph"]), steps=int(log(10, 300)))
    if kind == "graph":
        return _sim(scale=round(log(0.1, 4.0), 4), bf16=bf16, driver="graph", steps=int(log(10, 500)))
    if kind == "dense":
        return _sim(scale=round(log(0.1, 4.0), 4), bf16=bf16, prop="pull",
                    driver=rng.choice(["persistent", "persistent", "graph"]), steps=int(log(20, 400)))
    return _sim(scale=round(log(0.2, 1.5), 4), bf16=bf16, plastic=True,
                driver=rng.choice(["persistent", "persistent", "graph"]), steps=int(log(50, 1000)))


@functools.lru_cache(maxsize=24)
def _network(arch, scale, seed, plastic):
    net = sg.scaffold(arch, scale, seed)
    if plastic:
        names = {p.name: p.index for p in net.projections}
        net.add_plasticity(names["granule_to_purkinje"], sg.STDP_TEACHER,
                           teacher=names["basket_to_purkinje"], window=50, a2_ji=-0.01)
    return net


def _scales(case):
    n = case["instances"]
    if n == 1:
        return [case["scale"]]
    return [case["scale"] * s for s in sg.batched_scales(range(1, n + 1))]


def _networks(case):
    return [_network(case["arch"], s, 1 + k, case["plastic"]) for k, s in enumerate(_scales(case))]


def prepare(case, seed):
    return _prepare_deliver(case, seed) if case["kind"] == "deliver" else _prepare_sim(case, seed)


def _prepare_sim(case, seed):
    nets = _networks(case)
    sim = sg.Simulation(
        nets, [seed * 64 + 1 + k for k in range(len(nets))], dt_ms=DT_MS, substeps=case["substeps"],
        weight_type=sg.WEIGHT_BF16 if case["bf16"] else sg.WEIGHT_FP32,
        exec_mode=sg.EXEC_PERSISTENT if case["driver"] == "persistent" else sg.EXEC_GRAPH,
        default_prop=sg.PROP_ELL if case["prop"] == "pull" else sg.PROP_AUTO,
        chunk_steps=min(case["steps"], 1000), raster=case["raster"])
    rates = np.random.default_rng(seed).uniform(2.0, 8.0, (64, 1)) if case["rates"] else None
    plastic = None
    if case["plastic"]:
        plastic = next(p.index for p in nets[0].projections if p.name == "granule_to_purkinje")
    return {"case": case, "sim": sim, "rates": rates, "pass": 0, "plastic": plastic}


def _prepare_deliver(case, seed):
    n, gen = case["cells"], torch.Generator(device="cuda").manual_seed(seed)
    dev = torch.device("cuda")
    # Out-degrees: most cells a few dozen synapses, one in 400 about a thousand (Golgi cells).
    deg = torch.poisson(torch.full((n,), 0.9 * case["fan"], device=dev), generator=gen)
    big = torch.rand(n, device=dev, generator=gen) < 0.0025
    deg = torch.where(big, deg + 40.0 * case["fan"], deg).to(torch.int64)
    row = torch.zeros(n + 1, dtype=torch.int64, device=dev)
    row[1:] = deg.cumsum(0)
    total = int(row[-1])
    post = torch.randint(0, n, (total,), device=dev, generator=gen)
    delay = torch.randint(1, 5, (total,), device=dev, generator=gen)
    channel = (torch.rand(total, device=dev, generator=gen) < 0.2).to(torch.int64)
    word = post | (delay << 27) | (channel << 31)
    word = torch.where(word >= 1 << 31, word - (1 << 32), word).to(torch.int32)
    weight = torch.rand(total, device=dev, generator=gen) * 2.0**16 + 2.0**15
    flags = (torch.rand((8, n), device=dev, generator=gen) < case["active"]).to(torch.uint8)
    return {"case": case, "flags": flags, "row": row.to(torch.int32), "syn": word,
            "weight": weight.to(torch.bfloat16) if case["bf16"] else weight,
            "ring": torch.zeros((case["slots"], n, 2), dtype=torch.int32, device=dev), "pass": 0}


def run(state):
    case, k = state["case"], state["pass"]
    state["pass"] += 1
    if case["kind"] == "deliver":
        flags = state["flags"][k % 8]
        rc = sg.lib().sgb_deliver_spikes(
            flags.data_ptr(), case["cells"], state["row"].data_ptr(), state["syn"].data_ptr(),
            state["weight"].data_ptr(), 1 if case["bf16"] else 0, state["ring"].data_ptr(), case["slots"], k,
            torch.cuda.current_stream().cuda_stream)
        if rc:
            raise RuntimeError("sgb_deliver_spikes returned %d" % rc)
        return state["ring"]
    sim = state["sim"]
    if state["rates"] is not None:
        sim.set_input_freq(0, state["rates"][k % 64])
    counts, raster = sim.loop_n_steps(case["steps"], counts=True, raster=case["raster"])
    out = {"counts": counts}
    if raster is not None:
        # A trial's raster goes into a table of fixed size, one row per trial.
        table = np.full(_raster_rows(case), 0xFFFFFFFF, np.uint32)
        table[: raster[0].size] = raster[0]
        out["raster_ids"], out["raster_offsets"] = table, raster[1]
    if case["state"]:
        out["u"], out["g"], out["ref"] = sim.state()
    if state["plastic"] is not None:
        out["plastic"] = sim.plastic_values(0, state["plastic"])
    return out


def _raster_rows(case):
    return int(65536 + 3e-3 * case["steps"] * sum(_scales(case)) * SIZES[case["arch"]][0])


def work(case):
    """Bytes and operations of a pass.

    A trial: each cell's state in and out once, the counts out, and per synaptic event its table
    entry (word and weight); a dense projection reads every entry once a step by definition.
    About 20 operations per cell and substep and one addition per event."""
    w = 2 if case["bf16"] else 4
    if case["kind"] == "deliver":
        events = case["cells"] * case["active"] * case["fan"]
        return {"bytes": case["cells"] + events * (4 + w + 8), "flops": events}
    scale, steps = sum(_scales(case)), case["steps"]
    cells, inputs, synapses = (x * scale for x in SIZES[case["arch"]])
    events = synapses * MEAN_RATE_HZ * DT_MS * 1e-3 * case["substeps"] * steps
    moved = 24.0 * (cells - inputs) + 28.0 * steps * case["instances"] + events * (4 + w)
    if case["prop"] == "pull":
        moved += 4.0 * synapses * steps
    if case["plastic"]:
        moved += (4.0 + 8.0) * 0.64 * synapses + 4.0 * 0.64 * synapses * steps
    return {"bytes": moved, "flops": 20.0 * cells * case["substeps"] * steps + events}


def exact(case, seed):
    """The first trial of a small event-driven net in 64 bits.  None for the others: a scaffold is
    chaotic, so after some thousand steps, or with rounded tables, a trajectory in other
    arithmetic is another trajectory."""
    if (case["kind"] != "sim" or case["bf16"] or case["substeps"] != 1 or case["plastic"] or case["rates"]
            or case["instances"] > 1 or not case["state"] or case["steps"] > 1000
            or SIZES[case["arch"]][2] * case["scale"] > 500_000):
        return None
    net, steps = _networks(case)[0], case["steps"]
    pops = net.populations
    base = np.cumsum([0] + [p.num for p in pops])
    n = int(base[-1])
    source = np.concatenate([np.full(p.num, p.dev_type == sg.INPUT) for p in pops])

    def per_cell(value):
        return np.concatenate([np.full(p.num, float(value(p))) for p in pops])

    def channel(p, c, k, other=0.0):
        return p.channels[c][k] if c < len(p.channels) else other

    cm, el, vr, vth, ie, gl = (per_cell(lambda p, a=a: getattr(p, a)) for a in
                               ("Cm", "El", "Vr", "Vth", "Ie", "gL"))
    cm[source] = 1.0
    ref_steps = per_cell(lambda p: int(p.dt_ref / DT_MS)).astype(np.int64)
    rev = [per_cell(lambda p, c=c: channel(p, c, 1)) for c in (0, 1)]
    gain = [per_cell(lambda p, c=c: channel(p, c, 0) * channel(p, c, 2)) for c in (0, 1)]
    tau = [per_cell(lambda p, c=c: channel(p, c, 3, 1.0)) for c in (0, 1)]
    # Every synapse, by its source cell.
    pre, post, wgt, dly, inh = [], [], [], [], []
    for p in net.projections:
        a, b, w, d = net.synapses(p.index)
        pre.append(base[p.pre] + a.astype(np.int64))
        post.append(base[p.post] + b.astype(np.int64))
        wgt.append(w.astype(np.float64))
        dly.append(d.astype(np.int64))
        inh.append(np.full(a.size, p.channel, np.int64))
    pre, post, wgt, dly, inh = (np.concatenate(x) for x in (pre, post, wgt, dly, inh))
    order = np.argsort(pre, kind="stable")
    post, wgt, dly, inh = post[order], wgt[order], dly[order], inh[order]
    row = np.concatenate([[0], np.cumsum(np.bincount(pre, minlength=n))])
    # Stimulus: a cell of source population q fires when its draw is under any of its sources' thresholds.
    threshold = np.zeros((len(net.inputs()), n), np.float64)
    windows = []
    for j, (pop, p, ids) in enumerate(net.inputs()):
        threshold[j, base[pop] + (np.arange(pops[pop].num) if len(ids) == 0 else ids.astype(np.int64))] = math.floor(
            min(1.0, p["rate_hz"] * DT_MS / 1000.0) * 2.0**32)
        windows.append([round(p[k] / DT_MS) for k in ("win_period_ms", "win_start_ms", "win_end_ms")])
    key = seed * 64 + 1
    cells = np.arange(n)
    u = np.where(source, 0.0, vr + (vth - vr) * ((_draws(key, cells, 0, 2) >> np.uint64(8)) + np.uint64(1)) / 2.0**24)
    g = np.zeros((2, n))
    ref = np.zeros(n, np.int64)
    slots = 16
    ring = np.zeros((slots, n, 2))
    counts = np.zeros((steps, len(pops)), np.int64)
    for t in range(steps):
        x = _draws(key, cells[source], t, 1).astype(np.float64)
        fired = np.zeros(n, bool)
        for th, (period, lo, hi) in zip(threshold, windows):
            at = t % period if period > 0 else t
            if hi <= lo or lo <= at < hi:
                fired[source] |= x < th[source]
        inc = ring[t % slots].copy()
        ring[t % slots] = 0.0
        cur = gl * (el - u) + ie - g[0] * (u - rev[0]) - g[1] * (u - rev[1])
        du = DT_MS / cm * cur
        for c in (0, 1):
            own = np.where(rev[c] > el, inc[:, 0], inc[:, 1])
            g[c] = np.where(source, 0.0, g[c] * (1.0 - DT_MS / tau[c]) + gain[c] * own)
        above = ~source & (u > vth)
        fired |= above
        ref = np.where(above, ref_steps, np.maximum(ref - 1, 0))
        u = np.where(source, 0.0, np.where(ref > 0, vr, u + du))
        ref[source] = 0
        counts[t] = np.add.reduceat(fired.astype(np.int64), base[:-1])
        q = np.concatenate([np.arange(row[c], row[c + 1]) for c in np.flatnonzero(fired)] or [np.zeros(0, np.int64)])
        np.add.at(ring, ((t + dly[q]) % slots, post[q], inh[q]), wgt[q])
    return {"counts": None, "u": u, "g": np.ascontiguousarray(g.T), "ref": None}


def _draws(key, cells, step, tag):
    """First word of Philox4x32-10 (Salmon et al., SC'11) on the counter (cell, step, 0, tag)."""
    mask = np.uint64(0xFFFFFFFF)
    c = [cells.astype(np.uint64), np.full(cells.size, step, np.uint64), np.zeros(cells.size, np.uint64),
         np.full(cells.size, tag, np.uint64)]
    k0, k1 = key & 0xFFFFFFFF, key >> 32
    for _ in range(10):
        a, b = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(b >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), b & mask, (a >> np.uint64(32)) ^ c[3] ^ np.uint64(k1),
             a & mask]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c[0]
