"""Performance cases: the work a program on this framework has it do, through its public calls.

A case is a dict of plain values; prepare() builds the networks it runs on (the synthetic networks
of braingrid_gb300.netgen, with the sizes and distributions of the benchmark workloads and the test
configurations) and run() makes one pass: the simulation steps of an epoch or of a call, the
results a program reads back, and the epoch end.

Kinds of case
  lif        one LIF network; radius is the connection radius it was grown to (0.4, the growth
             rule's start radius, leaves it without synapses)
  growth     one ConnGrowth pass over a grown network
  izh        one Izhikevich network: static wiring, dynamic STDP, Poisson drive
  lif_batch  the growth parameter sweep: LIF networks of uneven size advanced together
  izh_batch  many Izhikevich + STDP networks advanced together
  served     a mixed stream of jobs through the job server
  state      save a network, load it back, read its whole state
"""
import math

import numpy as np

from braingrid_gb300 import lib as bg
from braingrid_gb300 import netgen
from braingrid_gb300 import serve
from braingrid_gb300 import workloads

DT = 1e-4
SYN = {"spiking": bg.BG3_SYN_SPIKING, "ds": bg.BG3_SYN_DS, "stdp": bg.BG3_SYN_STDP,
       "dstdp": bg.BG3_SYN_DYNSTDP}
SPREAD = 0.05   # grown radii are spread by this much about the case's radius


def lif_case(**kw):
    """drive: "none", or the inputs "poisson" (10 Hz on every neuron) and "regular" (pulses on
    one neuron in five); scale: factor on the grown weights; noise: "device", or "reference" for
    the reference's own stream drawn on the host; end: how the epoch ends."""
    return dict(dict(kind="lif", side=10, radius=0.4, steps=1000, syn="ds", drive="none",
                     scale=1.0, noise="device", end="record"), **kw)


def listed():
    return [
        # a program that watches the 10x10 benchmark network step by step: one step, one readback
        lif_case(name="lockstep_10x10", side=10, radius=2.5, steps=1, scale=0.003),
        # the 10x10 network run from its parameter file: the reference's noise, growth at the end
        lif_case(name="epoch_10x10_reference_noise", side=10, radius=1.5, steps=5000,
                 noise="reference", end="growth"),
        # a 30x30 network of STDP synapses with the regular stimulus, as the STDP test networks
        lif_case(name="stdp_30x30", side=30, radius=2.0, steps=500, syn="stdp", drive="regular",
                 scale=0.003),
        # how every growth run begins: 100x100 at the start radius, no synapse yet
        lif_case(name="start_100x100", side=100, steps=1000, end="growth"),
        # the headline network: 100x100, 7.6 M synapses, driven at the growth rule's target rate
        lif_case(name="driven_100x100", side=100, radius=8.4, steps=500, drive="poisson",
                 scale=0.0003),
        # a large served network after its first growth pass: it fires at about 300 Hz
        lif_case(name="bursting_180x180", side=180, radius=8.4, steps=100),
        # the epoch end of the headline network: the weights of 7.6 M synapses
        dict(name="growth_100x100", kind="growth", side=100, radius=8.4),
        # one Izhikevich network of the largest size of the 512-network batch
        dict(name="izh_90x90", kind="izh", width=90, height=90, steps=500),
        # the growth parameter sweep: 36 networks of 30x30 to 100x100
        dict(name="lif36_batch", kind="lif_batch", count=36, steps=100),
        # a share of the 512-network Izhikevich batch: 500 to 8,000 neurons each
        dict(name="izh64_batch", kind="izh_batch", count=64, steps=300),
        # a mixed stream of short jobs through the server
        dict(name="served_6_jobs", kind="served", jobs=6, side=60, neurons=3000, epoch=0.05),
        # stop and resume: the lossless checkpoint both ways and the state a run ends with
        dict(name="state_33x33", kind="state", side=33, radius=3.0),
    ]


def _between(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["lif", "lif", "lif", "lif", "growth", "izh", "izh", "lif_batch",
                       "izh_batch", "izh_batch", "served", "state"])
    if kind == "lif":
        side = _between(rng, 8, 160)
        grown = rng.random() < 0.7
        c = lif_case(side=side, radius=round(rng.uniform(1.0, min(8.4, 0.4 * side)), 2) if grown
                     else 0.4)
        # scaled weights: a driven network near its target rate; full weights: bursts
        c["scale"], c["drive"] = rng.choice([(0.0003, "poisson"), (0.003, "none"), (1.0, "none"),
                                             (0.003, "regular")])
        c["syn"] = rng.choice(["ds", "ds", "ds", "spiking", "stdp", "dstdp"]) if side <= 60 else "ds"
        c["noise"] = rng.choice(["device", "device", "reference"]) if side <= 50 else "device"
        c["end"] = rng.choice(["record", "growth"])
        most = min(1500.0, 2e9 / max(1, synapses(side, c["radius"])),
                   1e7 / side ** 2 if c["noise"] == "reference" else 1e9)
        c["steps"] = _between(rng, 1, most)
        return c
    if kind == "growth":
        side = _between(rng, 10, 110)
        return dict(kind=kind, side=side, radius=round(rng.uniform(0.4, min(8.4, 0.4 * side)), 2))
    if kind == "izh":
        w = _between(rng, 8, 160)
        return dict(kind=kind, width=w, height=max(5, int(w * rng.uniform(0.7, 1.3))),
                    steps=_between(rng, 5, 600))
    if kind == "lif_batch":
        return dict(kind=kind, count=_between(rng, 2, 30), steps=_between(rng, 3, 100))
    if kind == "izh_batch":
        return dict(kind=kind, count=_between(rng, 2, 56), steps=_between(rng, 5, 300))
    if kind == "served":
        return dict(kind=kind, jobs=rng.randint(2, 6), side=_between(rng, 10, 60),
                    neurons=_between(rng, 500, 3000), epoch=rng.choice([0.02, 0.03, 0.05]))
    return dict(kind=kind, side=_between(rng, 8, 34), radius=round(rng.uniform(1.0, 3.0), 2))


# ---- shapes -----------------------------------------------------------------------------------
def _offsets(side, reach):
    """Grid offsets (dx, dy) != (0, 0) within reach that fit on a side x side grid."""
    k = min(side - 1, int(math.floor(reach)))
    return [(dx, dy) for dx in range(-k, k + 1) for dy in range(-k, k + 1)
            if (dx or dy) and dx * dx + dy * dy < reach * reach]


def synapses(side, radius):
    """Synapses of a side x side grid whose radii are all radius (pairs closer than 2 radius)."""
    return sum((side - abs(dx)) * (side - abs(dy)) for dx, dy in _offsets(side, 2 * radius))


def max_synapses(side, radius):
    """Slots per neuron: what the largest radii reach plus room for an epoch's growth."""
    return max(8, len(_offsets(side, 2 * (radius + SPREAD) + 0.2)))


def _epoch(steps):
    """Epoch length (s) of a network whose pass is one epoch of that many steps (0.01 s at least)."""
    return max(steps, 100) * DT


# ---- networks ---------------------------------------------------------------------------------
def _lif(c, seed, radii_seed=None):
    side, grown = c["side"], c["radius"] > 0.5
    spec = netgen.lif_network(side, side, seed=seed % (1 << 31))
    inject = c["noise"] == "reference"
    stdp = c["syn"] in ("stdp", "dstdp")
    net = bg.Network(spec["N"], max_synapses(side, c["radius"]), side, side,
                     0.2 if stdp else _epoch(c["steps"]), DT, 1000, 10, SYN[c["syn"]],
                     bg.BG3_NOISE_INJECT if inject else bg.BG3_NOISE_DEVICE, seed & 0xFFFFFFFF)
    netgen.configure_lif(net, spec)
    if stdp:
        net.set_stdp_constants(**netgen.STDP_ADDITIVE)
    if grown:
        netgen.pregrow(net, spec, c["radius"], spread=SPREAD, weight_scale=c["scale"],
                       seed=(radii_seed if radii_seed is not None else seed + 11) % (1 << 31))
    rs = np.random.RandomState((seed + 23) % (1 << 31))
    if c["drive"] == "poisson":
        arr, lam = netgen.poisson_arrays(spec, 10.0, 9.5)
        net.input_poisson(lam, seed=seed & 0xFFFFFFFF, step=0, **arr)
    elif c["drive"] == "regular":
        values = np.where(rs.uniform(size=spec["N"]) < 0.2, np.float32(5e-9), np.float32(0))
        net.input_regular(values, rs.randint(0, 500, spec["N"]), 200, 1000)
    s = dict(kind="lif", net=net, steps=c["steps"], end=c["end"], N=spec["N"], epoch=0, gen=None,
             history=not stdp)
    if inject:
        s["gen"] = bg.NormStream(seed & 0xFFFFFFFF)
    if grown and not inject:
        net.step(300)            # past the common start: arrivals under way
        net.record()
    net.sync()
    return s


def _izh(width, height, seed):
    spec, syn, counts, M = netgen.izh_static_spec(width, height, seed % (1 << 30))
    net = bg.Network(spec["N"], M, width, height, 1.0, DT, 1000, 10, bg.BG3_SYN_DYNSTDP,
                     bg.BG3_NOISE_DEVICE, seed & 0xFFFFFFFF, neuron_kind=bg.BG3_NEURON_IZH)
    netgen.configure_izh_static(net, spec, syn, counts, input_seed=seed & 0xFFFFFFFF)
    return net


def prepare(case, seed):
    kind = case["kind"]
    if kind == "lif":
        return _lif(case, seed)
    if kind == "growth":
        s = _lif(lif_case(side=case["side"], radius=case["radius"]), seed)
        rs = np.random.RandomState((seed + 5) % (1 << 31))
        s["radii"] = rs.uniform(case["radius"] - SPREAD, case["radius"] + SPREAD,
                                s["N"]).astype(np.float32)
        return dict(s, kind=kind)
    if kind == "izh":
        net = _izh(case["width"], case["height"], seed)
        net.step(1200)           # STDP brings the network to its steady rate
        net.record()
        net.sync()
        return dict(kind=kind, nets=[net], steps=case["steps"])
    if kind == "lif_batch":
        members = workloads.sweep36_members()[:case["count"]]
        nets = [workloads.build_member(dict(w, seed=w["seed"] + 64 * (seed % (1 << 20))))[1]
                for w in members]
        batch = bg.Batch(nets)
        batch.step(64)
        batch.sync()
        return dict(kind=kind, nets=nets, batch=batch, steps=case["steps"])
    if kind == "izh_batch":
        nets = [_izh(w, h, 1000 * (seed % (1 << 18)) + k) for k, (w, h) in
                enumerate(workloads.izh512_shapes(case["count"]))]
        batch = bg.Batch(nets)
        batch.step(1200)
        for net in nets:
            net.record()
        batch.sync()
        return dict(kind=kind, nets=nets, batch=batch, steps=case["steps"])
    if kind == "served":
        return _stream(case, seed)
    # radii of their own seed: the index maps' length is part of the case
    s = _lif(lif_case(side=case["side"], radius=case["radius"], steps=200), seed, radii_seed=5)
    return dict(s, kind=kind)


def _stream(case, seed):
    """Job descriptions: LIF growth networks and Izhikevich networks of falling sizes, 1 to 3
    epochs each, their setup arrays in hand."""
    jobs = []
    for k in range(case["jobs"]):
        js, epochs = (seed + 101 * k) % (1 << 30), 1 + k % 3
        if k % 3 == 2:
            w = max(5, int(round(math.sqrt(case["neurons"] / (1 + k // 3)))))
            spec, syn, counts, M = netgen.izh_static_spec(w, w, js)
            desc = bg.NetDesc(spec["N"], M, w, w, case["epoch"], DT, 1000, epochs,
                              bg.BG3_NEURON_IZH, bg.BG3_SYN_DYNSTDP, bg.BG3_NOISE_DEVICE, js)

            def setup(net, spec=spec, syn=syn, counts=counts, js=js):
                netgen.configure_izh_static(net, spec, syn, counts, input_seed=js)
            jobs.append((desc, epochs, False, setup))
        else:
            side = max(8, case["side"] - 7 * k)
            radius = min(8.4, 0.45 * side)
            spec = netgen.lif_network(side, side, seed=js)
            desc = bg.NetDesc(spec["N"], max_synapses(side, radius), side, side, case["epoch"], DT,
                              1000, epochs, bg.BG3_NEURON_LIF, bg.BG3_SYN_DS, bg.BG3_NOISE_DEVICE, js)

            def setup(net, spec=spec, radius=radius, js=js):
                netgen.configure_lif(net, spec)
                netgen.pregrow(net, spec, radius, spread=SPREAD, weight_scale=0.003, seed=js)
            jobs.append((desc, epochs, True, setup))
    return dict(kind="served", jobs=jobs)


# ---- one pass ---------------------------------------------------------------------------------
NEURONS = ("Vm", "summation", "nStepsInRefr", "spikeCount", "spikeCountOffset")


def _neurons(net, history=False):
    out = net.download_lif(fields=NEURONS + (("history",) if history else ()))
    if history:
        out["history"] = out["history"].view(np.int64)
    return out


def run(state):
    kind = state["kind"]
    if kind == "lif":
        net = state["net"]
        if state["gen"] is not None:
            # one value per neuron and step has to be held before the steps are queued
            short = state["N"] * state["steps"] - net.noise_pending()
            if short > 0:
                net.push_noise(state["gen"].take(short))
        net.step(state["steps"])
        out = _neurons(net, state["history"])
        state["epoch"] += 1
        if state["end"] == "growth":
            net.growth(state["epoch"])
            out["radii"], out["rates"] = net.download_growth()
        else:
            net.record()
        return out
    if kind == "growth":
        net = state["net"]
        net.upload_growth(radii=state["radii"], **netgen.GROWTH)
        net.growth(1)
        radii, rates = net.download_growth()
        return dict(radii=radii, rates=rates, synapses=net.total_synapses())
    if kind == "served":
        srv = serve.Server(chunk_steps=2000)
        jobs = [serve.Job(*j) for j in state["jobs"]]
        for j in jobs:
            srv.submit(j)
        srv.run_all()
        srv.close()
        return [dict(j.outputs(), status=j.result.status) for j in jobs]
    if kind == "state":
        net = state["net"]
        net.load_checkpoint(net.checkpoint())
        out = net.download_state()
        for part, name in (("neurons", "history"), ("synapses", "lastSpike")):
            out[part][name] = out[part][name].view(np.int64)
        return out
    nets = state["nets"]
    (state["batch"] if kind != "izh" else nets[0]).step(state["steps"])
    fields = {k: [] for k in NEURONS + (("u",) if kind != "lif_batch" else ())}
    for net in nets:
        for k, v in _neurons(net).items():
            fields[k].append(v)
        if "u" in fields:
            fields["u"].append(net.download_izh()["u"])
        net.record()
    return {k: np.concatenate(v) for k, v in fields.items()}


# ---- what a pass cannot do without ------------------------------------------------------------
def _cost(n, syn, steps, izh, slots=0, epoch_end=0):
    """A network's hot state read and written once (8.5 bytes a synapse, 48 or 94 a neuron), its
    results, and per step 2 operations a synapse and about 20 (LIF) or 50 (Izhikevich) a neuron."""
    return dict(bytes=8.5 * syn + (94 if izh else 48) * n + 20 * n + epoch_end,
                flops=steps * (2.0 * syn + (50 if izh else 20) * n))


def work(case):
    kind = case["kind"]
    if kind == "lif":
        n, syn = case["side"] ** 2, synapses(case["side"], case["radius"])
        # epoch end with growth: every weight rewritten from its pair's radii and positions
        w = _cost(n, syn, case["steps"], False, epoch_end=(8 * syn if case["end"] == "growth" else 0))
        if case["syn"] in ("ds", "spiking"):
            w["bytes"] += 8 * n * int(np.float32(_epoch(case["steps"])) * np.float32(1000))
        if case["noise"] == "reference":
            w["bytes"] += 8 * n * case["steps"]
        return w
    if kind in ("growth", "state"):
        n, syn = case["side"] ** 2, synapses(case["side"], case["radius"])
        if kind == "growth":
            # per overlapping pair: the source read, the weight written; two arc cosines, two sines
            return dict(bytes=8 * syn + 24 * n, flops=100.0 * max(syn, n))
        slots = n * max_synapses(case["side"], case["radius"])
        return dict(bytes=3 * 46.5 * slots + 100 * n, flops=0)
    if kind == "izh":
        n = case["width"] * case["height"]
        return _cost(n, 10 * n, case["steps"], True)
    total = dict(bytes=0.0, flops=0.0)
    if kind == "served":
        parts = []
        for k in range(case["jobs"]):
            steps = int(round((1 + k % 3) * case["epoch"] / DT))
            if k % 3 == 2:
                n = max(5, int(round(math.sqrt(case["neurons"] / (1 + k // 3))))) ** 2
                parts.append(_cost(n, 10 * n, steps, True))
            else:
                side = max(8, case["side"] - 7 * k)
                parts.append(_cost(side ** 2, synapses(side, min(8.4, 0.45 * side)), steps, False))
    elif kind == "lif_batch":
        parts = [_cost(w["width"] ** 2, synapses(w["width"], w["radius"]), case["steps"], False)
                 for w in workloads.sweep36_members()[:case["count"]]]
    else:
        parts = [_cost(4250, 42500, case["steps"], True)] * case["count"]
    for p in parts:
        total = {k: total[k] + p[k] for k in total}
    return total


# ---- results in 64 bits -----------------------------------------------------------------------
def _normal(seed, step, n):
    """The device generator's N(0, 1) draws of neurons 0 .. n - 1 at a step: Box-Muller of two
    24-bit uniforms from Philox4x32-10 (Salmon et al., SC'11), key (seed, seed ^ 0x5bd1e995)."""
    lo32 = np.uint64(0xFFFFFFFF)
    c = [np.arange(n, dtype=np.uint64), np.full(n, step & 0xFFFFFFFF, np.uint64),
         np.full(n, step >> 32, np.uint64), np.zeros(n, np.uint64)]
    k0, k1 = seed, seed ^ 0x5BD1E995
    for _ in range(10):
        a, b = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(b >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), b & lo32,
             (a >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), a & lo32]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    u1 = ((c[0] >> np.uint64(8)).astype(np.float64) + 0.5) / 16777216.0
    u2 = (c[1] >> np.uint64(8)).astype(np.float64) / 16777216.0
    return np.sqrt(-2.0 * np.log(u1)) * np.cos(2.0 * np.pi * u2)


def _grown(radii, rates, seconds):
    """ConnGrowth's radius update in 64 bits."""
    g = netgen.GROWTH
    top = g["target_rate"] / g["epsilon"]
    e = np.exp((g["epsilon"] - rates / top) / g["beta"])
    return np.maximum(radii + seconds * g["rho"] * (1.0 - 2.0 / (e + 1.0)), g["min_radius"])


def exact(case, seed):
    """Networks with synapses feed rounding back through their spikes, so that a trajectory has no
    64-bit value to compare with; what has one: the independent neurons of a network at the
    start radius on device noise, and the growth rule's radii."""
    if case["kind"] == "growth":
        n = case["side"] ** 2
        rs = np.random.RandomState((seed + 5) % (1 << 31))
        radii = rs.uniform(case["radius"] - SPREAD, case["radius"] + SPREAD, n).astype(np.float32)
        # no step since the last epoch end when the network was grown and settled: rates are 0
        return dict(radii=_grown(radii.astype(np.float64), np.zeros(n), _epoch(1000)),
                    rates=np.zeros(n), synapses=None)
    if case["kind"] != "lif" or case["radius"] > 0.5 or case["drive"] != "none" or \
            case["noise"] != "device":
        return None
    spec = netgen.lif_network(case["side"], case["side"], seed=seed % (1 << 31))
    f = {k: spec[k].astype(np.float64) for k in ("Vm", "Vthresh", "Vreset", "I0", "Inoise", "C1",
                                                 "C2", "Trefract")}
    V, refr = f["Vm"], np.zeros(spec["N"], np.int64)
    count = np.zeros(spec["N"])
    for t in range(case["steps"]):
        waits = refr > 0
        fires = ~waits & (V >= f["Vthresh"])
        sp = f["I0"] + _normal(seed & 0xFFFFFFFF, t, spec["N"]) * f["Inoise"]
        V = np.where(waits, V, np.where(fires, f["Vreset"], f["C1"] * V + f["C2"] * sp))
        refr = np.where(waits, refr - 1, np.where(fires, (f["Trefract"] / DT + 0.5).astype(int), 0))
        count += fires
    out = dict(Vm=V, summation=np.zeros(spec["N"]), nStepsInRefr=None, spikeCount=None,
               spikeCountOffset=None)
    if case["syn"] in ("ds", "spiking"):
        out["history"] = None
    if case["end"] == "growth":
        T = 0.2 if case["syn"] in ("stdp", "dstdp") else _epoch(case["steps"])
        out["radii"] = _grown(np.full(spec["N"], 0.4), count / T, T)
        out["rates"] = None      # whole spikes over the epoch
    return out
