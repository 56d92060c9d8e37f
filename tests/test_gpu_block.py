"""Blocks of steps (bg3_block.cu) against the per-step kernels, bit for bit: the same network
advanced by both (small_max_slots 0 keeps a network on the per-step kernels, 1 keeps it off the
one-launch path of small networks, 65,536 takes that path where it is small enough), at sizes around the 32-neuron tiles, the row quads and the
eight steps of a block, with downloads, epoch ends and single steps in between."""
import threading

import numpy as np
import pytest

from braingrid_gb300 import lib as bg
from braingrid_gb300 import netgen

pytestmark = pytest.mark.gpu

STEPS = (1, 8, 7, 9, 131, 3)   # remainders of a block, a graph's worth of blocks


def lif(w, h, syn, radius, drive, max_syn, seed=5):
    spec = netgen.lif_network(w, h, seed=seed)
    # membranes near threshold: the network fires, and its spikes arrive, from the first steps
    spec["Vm"] = np.random.RandomState(seed).uniform(13.2e-3, 15.2e-3, spec["N"]).astype(np.float32)
    net = bg.Network(spec["N"], max_syn, w, h, 0.1, 1e-4, 1000, 4, syn, bg.BG3_NOISE_DEVICE, seed)
    netgen.configure_lif(net, spec)
    if syn >= bg.BG3_SYN_STDP:
        net.set_stdp_constants(**netgen.STDP_ADDITIVE)
    if radius:
        netgen.pregrow(net, spec, radius, weight_scale=0.3)
    rs = np.random.RandomState(seed + 1)
    if drive == "poisson":
        arr, lam = netgen.poisson_arrays(spec, 40.0, 9.5)
        net.input_poisson(lam, seed=seed, step=0, **arr)
    elif drive == "regular":
        net.input_regular(np.full(spec["N"], 4e-9, np.float32), rs.randint(0, 40, spec["N"]), 20, 60)
    return net


def izh(w, h, seed=5):
    net = netgen.make_izh_static(w, h, seed, epoch_duration=0.1)[1]
    net.set_launch(small_max_slots=0)
    net.step(900)      # per-step kernels, until STDP and the drive have the network firing
    net.record()
    return net


def state(net):
    out = dict(net.download_lif())
    out.update({"syn_" + k: v for k, v in net.download_synapses().items()})
    if net.desc.neuron_kind == bg.BG3_NEURON_IZH:
        out.update({"izh_" + k: v for k, v in net.download_izh().items()})
    out["step"], out["err"] = net.sim_step, net.error_word
    return out


def same(a, b, what):
    x, y = state(a), state(b)
    for k in x:
        u, v = np.asarray(x[k]), np.asarray(y[k])
        if u.dtype == np.float32:
            u, v = u.view(np.uint32), v.view(np.uint32)
        assert np.array_equal(u, v), "%s: %s differs at %s" % (what, k, np.nonzero(u != v)[0][:5])


def advance(make, end="record", small=1):
    blocks, plain = make(), make()
    blocks.set_launch(small_max_slots=small)
    plain.set_launch(small_max_slots=0)
    spikes = 0
    for i, n in enumerate(STEPS):
        b0 = blocks.launches
        blocks.step(n)
        plain.step(n)
        assert blocks.launches - b0 <= 2 * ((n + 7) // 8)     # it did run in blocks
        if i % 2:
            same(blocks, plain, "after call %d (%d steps)" % (i, n))
            spikes = max(spikes, int(blocks.download_lif(fields=("spikeCount",))["spikeCount"].sum()))
    if end == "growth":
        blocks.growth(1)
        plain.growth(1)
    else:
        blocks.record()
        plain.record()
    # masks -> ring -> masks: per-step kernels for a while, then blocks again
    blocks.set_launch(small_max_slots=0)
    blocks.step(5)
    plain.step(5)
    blocks.set_launch(small_max_slots=small)
    blocks.step(40)
    plain.step(40)
    same(blocks, plain, "after the epoch end")
    assert spikes > 0
    assert blocks.error_word == 0
    for net in (blocks, plain):
        net.close()


@pytest.mark.parametrize("small", [1, 65536])
@pytest.mark.parametrize("syn", [bg.BG3_SYN_SPIKING, bg.BG3_SYN_DS, bg.BG3_SYN_STDP, bg.BG3_SYN_DYNSTDP])
@pytest.mark.parametrize("w,h,radius,drive,max_syn", [
    (9, 7, 1.2, "none", 30),        # 63 neurons, a partial last quad
    (13, 5, 1.5, "poisson", 33),    # 65 neurons: one past a tile
    (8, 4, 0.0, "regular", 4),      # one tile, no synapse
    (40, 33, 1.9, "poisson", 64),   # the widest rows of a thin tile
])
def test_thin_blocks_equal_steps(small, syn, w, h, radius, drive, max_syn):
    advance(lambda: lif(w, h, syn, radius, drive, max_syn), end="growth", small=small)


@pytest.mark.parametrize("syn", [bg.BG3_SYN_SPIKING, bg.BG3_SYN_DS])
@pytest.mark.parametrize("w,h,radius,drive,max_syn", [
    (9, 7, 6.0, "poisson", 65),     # every pair connected, 62 rows: one chunk and a row
    (13, 5, 4.0, "none", 130),      # 64 rows at most in use, three chunks allocated
    (40, 33, 3.4, "none", 190),     # a partial third chunk; bursts: the chunk-by-chunk arrivals
    (40, 33, 3.4, "poisson", 191),
    (30, 30, 13.5, "regular", 900), # fifteen chunks, most of the network in every row
])
def test_dense_blocks_equal_steps(syn, w, h, radius, drive, max_syn):
    advance(lambda: lif(w, h, syn, radius, drive, max_syn), end="growth")


@pytest.mark.parametrize("w,h,small", [(9, 7, 1), (13, 5, 65536), (33, 32, 65536), (60, 41, 1)])
def test_izhikevich_stdp_blocks_equal_steps(w, h, small):
    advance(lambda: izh(w, h), small=small)


@pytest.mark.parametrize("syn", [bg.BG3_SYN_DS, bg.BG3_SYN_DYNSTDP])
@pytest.mark.parametrize("w,h,radius,max_syn", [(9, 7, 6.0, 65), (13, 5, 4.0, 301), (5, 4, 3.0, 19), (40, 40, 1.2, 37)])
def test_small_network_blocks_equal_steps(syn, w, h, radius, max_syn):
    """Rows beyond a thin tile's, one block and eight."""
    advance(lambda: lif(w, h, syn, radius, "poisson", max_syn), small=65536)


def test_batched_blocks_equal_steps():
    shapes = [(9, 7), (13, 5), (32, 20), (25, 41)]
    a, b = [izh(w, h, 20 + w) for w, h in shapes], [izh(w, h, 20 + w) for w, h in shapes]
    batch = bg.Batch(a)
    for n in STEPS:
        batch.step(n)
        for net in b:
            net.step(n)
    batch.sync()
    for x, y in zip(a, b):
        same(x, y, "batched")
    batch.set_launch(small_max_slots=0)     # the batch's per-step kernels, and back
    batch.step(3)
    batch.set_launch(small_max_slots=65536)
    batch.step(21)
    for x, y in zip(a, b):
        y.step(24)
        same(x, y, "batched, after per-step kernels")
    batch.close()


def test_batched_dense_and_thin_blocks_equal_steps():
    shapes = [(9, 7, 6.0, 65), (40, 33, 3.4, 190), (13, 5, 1.5, 33), (33, 31, 1.9, 64)]
    a, b = ([lif(w, h, bg.BG3_SYN_DS, r, "none", m) for w, h, r, m in shapes] for _ in range(2))
    batch = bg.Batch(a)
    for net in b:
        net.set_launch(small_max_slots=0)
    for n in STEPS:
        batch.step(n)
        for net in b:
            net.step(n)
    batch.sync()
    for x, y in zip(a, b):
        same(x, y, "batched")
    batch.close()


def test_two_spikes_at_one_synapse_in_a_block():
    """Neurons without a refractory period whose reset lies above the threshold fire on every
    step, so that each synapse receives several spikes within a block."""
    for radius, max_syn in ((1.5, 33), (4.0, 130)):
        nets = []
        for small in (1, 65536, 0):
            net = lif(13, 5, bg.BG3_SYN_DS, radius, "none", max_syn)
            v = net.download_lif(fields=("Vthresh", "Vreset", "Trefract"))
            v["Trefract"][::3] = 0.0
            v["Vreset"][::3] = v["Vthresh"][::3] + np.float32(1e-3)
            v["Vthresh"][1::3] -= np.float32(1.0e-3)
            net.upload_lif(**v)
            net.set_launch(small_max_slots=small)
            nets.append(net)
        for n in (8, 8, 3, 40):
            for net in nets:
                net.step(n)
            same(nets[0], nets[2], "radius %g after %d steps" % (radius, n))
            same(nets[1], nets[2], "small, radius %g after %d steps" % (radius, n))
        assert int(nets[0].download_lif(fields=("spikeCount",))["spikeCount"].max()) > 8


@pytest.mark.parametrize("seed", [5, 6])
def test_overlap_area_matches_fp64(seed):
    """The overlap area in float-float arithmetic gives the FP64 pipe's bits on equal, close,
    just touching, nearly contained and independent radii, and hands only the uncertain few back."""
    n = 1 << 25
    bad, handed, without = bg.selftest_overlap(samples=n, seed=seed)
    assert bad == 0
    assert without < n // 2 and handed < n // 50, (handed, without)


@pytest.mark.parametrize("syn", [bg.BG3_SYN_DS, bg.BG3_SYN_DYNSTDP])
@pytest.mark.parametrize("w,h,radius,max_syn,steps", [
    (10, 10, 1.5, 30, 300),         # four tiles, one block
    (9, 7, 6.0, 65, 300),
    (33, 31, 1.2, 37, 300),         # 32 tiles in eight blocks
    (45, 45, 0.7, 9, 300),          # 64 tiles, the most
    (10, 10, 1.5, 30, 40),          # the stream runs out: zeros and the error flag
])
def test_small_network_blocks_draw_injected_noise(syn, w, h, radius, max_syn, steps):
    values = np.random.RandomState(3).standard_normal(w * h * steps).astype(np.float32)
    nets = []
    for small in (65536, 0):
        net = lif(w, h, syn, radius, "poisson", max_syn)
        net.set_noise_mode(bg.BG3_NOISE_INJECT, 1)
        net.push_noise(values)
        net.set_launch(small_max_slots=small)
        nets.append(net)
    for n in STEPS:
        b0 = nets[0].launches
        for net in nets:
            net.step(n)
        assert nets[0].launches - b0 == 1
        same(nets[0], nets[1], "after %d steps" % n)
        assert nets[0].noise_pending() == nets[1].noise_pending()
    assert int(nets[0].download_lif(fields=("spikeCount",))["spikeCount"].sum()) > 0
    assert (nets[0].error_word != 0) == (steps < sum(STEPS))
    for net in nets:
        net.close()


def test_narrow_network_below_the_thin_option():
    """thin_max_quads below the width of a network that could run thin blocks (10 row quads): the
    per-step kernels, set by the caller, in a batch, from a checkpoint and by the tuner."""
    def make():
        return lif(50, 42, bg.BG3_SYN_DS, 1.55, "poisson", 40)
    want, a, b, c = make(), make(), make(), make()
    want.set_launch(small_max_slots=0)
    a.set_launch(thin_max_quads=1)
    batch = bg.Batch([b])
    batch.set_launch(thin_max_quads=9)
    for n in STEPS:
        want.step(n)
        a.step(n)
        batch.step(n)
    batch.sync()
    same(a, want, "set by the caller")
    same(b, want, "in a batch")
    batch.close()
    c.load_checkpoint(a.checkpoint())
    assert c.launch["thin_max_quads"] == 1
    for net in (c, want):
        net.step(41)
    same(c, want, "from a checkpoint")
    cfg, ms = c.autotune(steps_per_trial=40)
    assert ms > 0
    same(c, want, "after tuning")
    for net in (c, want):
        net.step(30)
    same(c, want, "with the tuned launch")
    assert int(want.download_lif(fields=("spikeCount",))["spikeCount"].sum()) > 0


def test_batch_graphs_of_the_two_forms_are_told_apart():
    """Blocks, a refresh, a run of single steps long enough for a graph of them (a member that
    draws injected noise keeps its batch off the blocks), and blocks again without a refresh."""
    shapes = [(40, 33, 3.4, 190), (33, 31, 1.9, 64)]
    a, b = ([lif(w, h, bg.BG3_SYN_DS, r, "none", m) for w, h, r, m in shapes] for _ in range(2))
    for net in b:
        net.set_launch(small_max_slots=0)
    batch = bg.Batch(a)
    batch.step(130)
    batch.refresh()
    a[0].set_noise_mode(bg.BG3_NOISE_INJECT, 5)
    b0 = batch.launches
    batch.step(40)
    assert batch.launches - b0 > 40
    a[0].set_noise_mode(bg.BG3_NOISE_DEVICE, 5)
    batch.step(300)
    batch.sync()
    for net, other in zip(a, b):
        other.step(470)
        same(net, other, "batched")
    batch.close()


def test_small_networks_of_several_threads():
    """A narrow and a wide small network stepped at the same time by two threads: every launch is
    accepted, and each network ends as it does alone."""
    shapes = [(10, 10, 1.5, 30), (13, 5, 4.0, 301)]    # 8 and 76 row quads
    nets, alone = ([lif(w, h, bg.BG3_SYN_DS, r, "poisson", m) for w, h, r, m in shapes] for _ in range(2))
    errors, start = [], threading.Barrier(len(nets))

    def run(net):
        try:
            start.wait()
            for _ in range(3000):
                net.step(1)
            net.sync()
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=run, args=(net,)) for net in nets]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for net, other in zip(nets, alone):
        other.step(3000)
        same(net, other, "stepped beside another")


def firing_at_intervals(steps, max_spikes, seed=7):
    """65 neurons that fire every `steps` steps, in random phases, on STDP synapses."""
    spec = netgen.lif_network(13, 5, seed=seed)
    net = bg.Network(spec["N"], 33, 13, 5, (max_spikes + 0.5) * 1e-3, 1e-4, 1000, 9, bg.BG3_SYN_DYNSTDP,
                     bg.BG3_NOISE_DEVICE, seed)
    netgen.configure_lif(net, spec)
    net.set_stdp_constants(**netgen.STDP_ADDITIVE)
    netgen.pregrow(net, spec, 1.5, weight_scale=0.3)
    v = net.download_lif(fields=("Vthresh", "Vreset", "Trefract", "Vm"))
    v["Vreset"] = v["Vthresh"] + np.float32(1e-3)
    v["Vm"] = v["Vreset"].copy()
    v["Trefract"][:] = (steps - 1) * 1e-4
    v["nStepsInRefr"] = np.random.RandomState(seed).randint(0, steps, spec["N"]).astype(np.int32)
    net.upload_lif(**v)
    return net


@pytest.mark.parametrize("small", [1, 65536])
def test_longer_refractory_periods_beside_a_dense_history(small):
    """Spikes seven steps apart, then a pause longer than the delays (a walk ends at a spike that is
    still under way): the walks of the next spikes read the 3 tau+ before, to the ring's last entry."""
    nets = [firing_at_intervals(7, 85) for _ in range(2)]
    nets[0].set_launch(small_max_slots=small)
    nets[1].set_launch(small_max_slots=0)
    for net in nets:
        for _ in range(4):
            net.step(190)
            net.record()
        net.upload_lif(Trefract=np.full(65, 31e-4, np.float32))
        net.step(40)
    same(nets[0], nets[1], "longer periods")
    assert nets[0].max_spikes == 85


@pytest.mark.parametrize("form", [1, 65536, "batch"])
def test_spikes_put_in_the_delay_queues(form):
    """Spikes on their way that no history holds: an upload adds them to the delay queues.  A post
    spike before such an arrival learns from the source's older spikes, and the arrival has the new
    weight."""
    nets = [firing_at_intervals(41, 85) for _ in range(2)]
    nets[0].set_launch(small_max_slots=1 if form == "batch" else form)
    nets[1].set_launch(small_max_slots=0)
    batch = bg.Batch(nets[:1]) if form == "batch" else None
    added = 0
    for net in nets:
        run = batch if batch and net is nets[0] else net
        run.step(200)
        for _ in range(6):
            syn = net.download_synapses()
            used = syn["in_use"].astype(bool)
            # the sources without a spike under way: one at the last step, of every second of them
            busy = np.unique(syn["src"][used & (syn["delayQueue"] != 0)])
            put = used & ~np.isin(syn["src"], busy) & (syn["src"] % 2 == 0)
            bit = (syn["delayIdx"] + syn["total_delay"] - 1) & 31
            syn["delayQueue"][put] |= (np.uint32(1) << bit[put].astype(np.uint32))
            added += int(put.sum())
            net.upload_synapses(net.sim_step, **syn)
            if batch and net is nets[0]:
                batch.refresh()
            run.step(23)
    assert added > 0
    same(nets[0], nets[1], "spikes added")
    if batch:
        batch.close()


def few_firing(w, h, syn, period, count, max_syn=260, radius=4.2, seed=9):
    """`count` neurons fire every `period` steps, the others never (0: all of them, in turn)."""
    spec = netgen.lif_network(w, h, seed=seed)
    net = bg.Network(spec["N"], max_syn, w, h, 0.1, 1e-4, 1000, 4, syn, bg.BG3_NOISE_DEVICE, seed)
    netgen.configure_lif(net, spec)
    netgen.pregrow(net, spec, radius, weight_scale=0.3)
    rs = np.random.RandomState(seed)
    on = np.zeros(spec["N"], bool)
    on[rs.permutation(spec["N"])[:count or spec["N"]]] = True
    v = net.download_lif(fields=("Vthresh", "Vreset", "Trefract", "Vm"))
    v["Vthresh"][~on] = 1.0
    v["Vreset"][on] = v["Vthresh"][on] + np.float32(1e-3)
    v["Vm"][on] = v["Vreset"][on]
    v["Trefract"][:] = np.float32((period - 1) * 1e-4)
    v["nStepsInRefr"] = rs.randint(0, period, spec["N"]).astype(np.int32)
    net.upload_lif(**v)
    return net, on


@pytest.mark.parametrize("syn", [bg.BG3_SYN_SPIKING, bg.BG3_SYN_DS])
@pytest.mark.parametrize("w,h", [(50, 42), (80, 70), (110, 100)])    # 66, 175 and 344 tiles
@pytest.mark.parametrize("period,share", [(29, 130), (1, 130), (7, 130), (29, 0)])
def test_dense_blocks_by_tiles_and_arrivals(syn, w, h, period, share):
    """Networks of one tile an SM and of more.  A few neurons (fewer than N / 128: pushed arrivals)
    reach most of a tile's rows with one spike a block, one at every step, or two; or all of
    them do (arrivals looked up)."""
    count = w * h // share if share else 0
    nets = [few_firing(w, h, syn, period, count) for _ in range(2)]
    nets[1][0].set_launch(small_max_slots=0)
    for calls in ((8, 8, 3), (16, 5, 8)):
        for net, _ in nets:
            for n in calls:
                net.step(n)
        same(nets[0][0], nets[1][0], "after calls of %s steps" % (calls,))
    fired = nets[0][0].download_lif(fields=("spikeCount",))["spikeCount"] > 0
    on = nets[0][1]
    assert fired[~on].sum() == 0 and fired[on].all()
    assert count == 0 or 0 < on.sum() * 128 <= w * h
    syn_ = nets[0][0].download_synapses()
    used = syn_["in_use"].astype(bool)
    if syn == bg.BG3_SYN_DS:
        # rows that received a spike in more than eight groups of 16 of some neuron's
        rows = (used & (syn_["lastSpike"] != np.uint64(2**64 - 1))).reshape(w * h, -1)
        groups = np.add.reduceat(rows, np.arange(0, rows.shape[1], 16), axis=1) > 0
        tiles = np.array([groups[d:d + 32].any(axis=0).sum() for d in range(0, w * h, 32)])
        assert tiles.max() > 8
    for net, _ in nets:
        net.close()


def test_batched_dense_blocks_by_tiles():
    """Batches of up to 152, up to 304 and more tiles."""
    for shapes in ([(50, 42)], [(50, 42), (70, 68)], [(50, 42), (70, 68), (80, 70)]):
        pairs = [[few_firing(w, h, bg.BG3_SYN_DS, 7, c)[0] for w, h in shapes for c in (0,)] for _ in range(2)]
        batch = bg.Batch(pairs[0])
        for net in pairs[1]:
            net.set_launch(small_max_slots=0)
        for n in (8, 5, 19):
            batch.step(n)
            for net in pairs[1]:
                net.step(n)
        batch.sync()
        for x, y in zip(*pairs):
            same(x, y, "batched")
        batch.close()
        for net in pairs[0] + pairs[1]:
            net.close()


@pytest.mark.parametrize("w,h,max_syn,radius", [(33, 33, 64, 1.9), (33, 33, 190, 3.4), (60, 60, 600, 6.0)])
def test_calls_of_few_steps(w, h, max_syn, radius):
    """Calls that run in blocks and calls too short for them in turn, a graph of blocks kept between
    them; wide networks take one step as step by step."""
    nets = [few_firing(w, h, bg.BG3_SYN_DS, 29, 0, max_syn, radius)[0] for _ in range(3)]
    nets[1].set_launch(small_max_slots=0)
    batch = bg.Batch(nets[2:])
    for n in (1, 1, 130, 1, 2, 3, 160, 1, 9, 1, 10, 40, 1, 33, 130):
        counts = [net.launches for net in nets[:2]]
        for run in (nets[0], nets[1], batch):
            run.step(n)
        if n == 1 and max_syn == 600:
            assert nets[0].launches - counts[0] == nets[1].launches - counts[1]
        if n >= 8:
            assert nets[0].launches - counts[0] < nets[1].launches - counts[1]
    batch.sync()
    same(nets[0], nets[1], "plain")
    same(nets[2], nets[1], "batched")
    batch.close()


@pytest.mark.parametrize("dt", [1.5e-4, 2e-4, 3e-4, 5e-4, 8e-4])
@pytest.mark.parametrize("w,h,max_syn,radius", [(33, 33, 64, 1.9), (33, 33, 190, 3.4), (60, 60, 600, 6.0)])
def test_longer_steps_take_shorter_blocks(w, h, max_syn, radius, dt):
    """Delays of fewer than eight steps: blocks of two to six."""
    nets = []
    for small in (1, 0):
        spec = netgen.lif_network(w, h, seed=5, delta_t=dt)
        spec["Vm"] = np.random.RandomState(5).uniform(13.2e-3, 15.2e-3, spec["N"]).astype(np.float32)
        net = bg.Network(spec["N"], max_syn, w, h, 0.1, dt, 1000, 4, bg.BG3_SYN_DS, bg.BG3_NOISE_DEVICE, 5)
        netgen.configure_lif(net, spec)
        netgen.pregrow(net, spec, radius, weight_scale=0.3)
        net.set_launch(small_max_slots=small)
        nets.append(net)
    for n in (1, 3, 40, 7, 130):
        for net in nets:
            net.step(n)
    same(nets[0], nets[1], "dt %g" % dt)
    if max_syn < 600 or dt < 4e-4:      # two steps at a time do not pay on wide rows
        assert nets[0].launches < nets[1].launches
    assert int(nets[0].download_lif(fields=("spikeCount",))["spikeCount"].sum()) > 0


@pytest.mark.parametrize("noise", [bg.BG3_NOISE_DEVICE, bg.BG3_NOISE_INJECT])
@pytest.mark.parametrize("syn", [bg.BG3_SYN_DS, bg.BG3_SYN_DYNSTDP])
@pytest.mark.parametrize("w,h,radius,max_syn", [(8, 4, 1.5, 30), (16, 16, 1.5, 30), (32, 16, 1.2, 20), (33, 16, 1.2, 20)])
def test_small_networks_in_calls_of_one_and_two_steps(noise, syn, w, h, radius, max_syn):
    """1, 8, 16 and 17 tiles: one CTA and the cluster in turn."""
    nets = []
    for small in (65536, 0):
        net = lif(w, h, syn, radius, "poisson", max_syn)
        if noise == bg.BG3_NOISE_INJECT:
            net.set_noise_mode(noise, 1)
            net.push_noise(np.random.RandomState(3).standard_normal(w * h * 120).astype(np.float32))
        net.set_launch(small_max_slots=small)
        nets.append(net)
    for n in (1, 2, 1, 40, 2, 2, 1, 1, 9, 1, 20):
        b0 = nets[0].launches
        for net in nets:
            net.step(n)
        assert nets[0].launches - b0 == 1
    same(nets[0], nets[1], "short calls")
    if noise == bg.BG3_NOISE_INJECT:
        assert nets[0].noise_pending() == nets[1].noise_pending()
    assert int(nets[0].download_lif(fields=("spikeCount",))["spikeCount"].sum()) > 0


def test_tuning_times_the_kernels_that_read_an_option():
    """A network that runs in blocks: the per-step kernels' options are timed on those (delivery
    grid and start, thin sweep), the batch's too."""
    net, twin = (lif(50, 42, bg.BG3_SYN_DS, 1.55, "poisson", 40) for _ in range(2))
    l0 = net.launches
    net.autotune(steps_per_trial=50)
    assert net.launches - l0 > 5 * 2 * 50      # five options off the default, two launches a step
    batch = bg.Batch([net])
    l0 = batch.launches
    batch.autotune(steps_per_trial=50)
    assert batch.launches - l0 > 3 * 2 * 50
    assert batch.launch["small_max_slots"] == net.launch["small_max_slots"] == 65536
    batch.step(40)
    batch.sync()
    twin.step(40)
    same(net, twin, "tuned")
    batch.close()


def test_growth_pass_counts_its_launches():
    net = lif(9, 7, bg.BG3_SYN_DS, 1.2, "none", 30)
    l0 = net.launches
    net.growth(1)
    assert net.launches - l0 == 7


@pytest.mark.parametrize("seed", [5, 6])
def test_stdp_sum_matches_fp64(seed):
    """The STDP weight sum in float-float arithmetic gives the FP64 pipe's bits; what is uncertain, or far
    in size from the weight, is handed back."""
    n = 1 << 25
    bad, handed = bg.selftest_stdp_sum(samples=n, seed=seed)
    assert bad == 0
    assert handed < 3 * n // 4, handed      # about a third of the changes are below 2^-60


@pytest.mark.parametrize("syn", [bg.BG3_SYN_SPIKING, bg.BG3_SYN_DS, bg.BG3_SYN_STDP, bg.BG3_SYN_DYNSTDP])
def test_thin_blocks_of_one_warp_a_tile(syn):
    """657 tiles: more than four warps a tile are used for."""
    nets = [lif(150, 140, syn, 1.5, "poisson", 33) for _ in range(2)]
    nets[1].set_launch(small_max_slots=0)
    for n in (8, 3, 130):
        for net in nets:
            net.step(n)
    same(nets[0], nets[1], "one warp a tile")
    assert nets[0].launches < nets[1].launches
    assert int(nets[0].download_lif(fields=("spikeCount",))["spikeCount"].sum()) > 0
    for net in nets:
        net.close()


@pytest.mark.parametrize("w,h", [(197, 196), (200, 197)])   # 1,207 and 1,232 tiles
def test_dense_blocks_past_the_bitmap_in_shared_memory(w, h):
    nets = [few_firing(w, h, bg.BG3_SYN_DS, 29, 0, 84, 2.3)[0] for _ in range(2)]
    nets[1].set_launch(small_max_slots=0)
    for n in (8, 8, 21):
        for net in nets:
            net.step(n)
    same(nets[0], nets[1], "%dx%d" % (w, h))
    assert nets[0].launches < nets[1].launches
    for net in nets:
        net.close()


@pytest.mark.parametrize("syn", [bg.BG3_SYN_SPIKING, bg.BG3_SYN_DYNSTDP])
def test_networks_do_not_wait_for_the_default_stream(syn):
    """A network made, grown, saved and loaded while the program's default stream is busy: nothing
    of it comes after later calls, or has to wait."""
    torch = pytest.importorskip("torch")
    twin = lif(13, 5, syn, 1.5, "none", 40)          # and the process's shared tables
    torch.cuda.synchronize()
    busy = torch.cuda.Event()
    torch.cuda._sleep(1 << 30)                        # half a second on the default stream
    busy.record()
    net = lif(13, 5, syn, 1.5, "none", 40)
    net.step(100)
    net.record()
    net.sync()
    early = not busy.query()
    buf = twin.checkpoint()                           # through the default stream: waits
    torch.cuda.synchronize()
    assert early
    twin.step(100)
    twin.record()
    net.growth(2)
    twin.growth(2)
    for n in (net, twin):
        n.step(30)
    same(net, twin, "made beside a busy default stream")
    loaded = lif(13, 5, syn, 1.5, "none", 40)
    torch.cuda._sleep(1 << 28)
    loaded.load_checkpoint(buf)
    loaded.step(100)
    loaded.record()
    loaded.growth(2)
    loaded.step(30)
    loaded.sync()
    torch.cuda.synchronize()
    same(loaded, twin, "loaded beside a busy default stream")


@pytest.mark.parametrize("small", [1, 65536])
def test_histories_out_of_order(small):
    """Offsets that put the next entries two places before the ring's end, unused, with the valid
    ones after them: the ring's fullness, which an arrival flags, comes with the third spike, where a ring
    in order would be almost empty."""
    nets = [firing_at_intervals(41, 700) for _ in range(2)]
    nets[0].set_launch(small_max_slots=small)
    nets[1].set_launch(small_max_slots=0)
    for net in nets:
        net.step(200)
        count = net.download_lif(fields=("spikeCount",))["spikeCount"]
        assert count.min() > 2 and count.max() < 8
        net.upload_lif(spikeCountOffset=(698 - count).astype(np.int32))
        for n in (40, 5, 100):
            net.step(n)
    same(nets[0], nets[1], "out of order")
    assert nets[0].error_word != 0


@pytest.mark.parametrize("form", ["upload", "checkpoint"])
def test_a_resumed_stdp_network_runs_in_blocks(form):
    """Histories in order, uploaded or loaded, have the spacing that is found in them."""
    nets = [firing_at_intervals(41, 60) for _ in range(3)]
    for net in nets:
        net.set_launch(small_max_slots=1)
    nets[1].set_launch(small_max_slots=0)
    for net in nets[:2]:
        net.step(300)
        net.record()
        net.step(100)
    if form == "upload":
        nets[2].upload_lif(**nets[0].download_lif())
        nets[2].upload_synapses(nets[0].sim_step, **nets[0].download_synapses())
    else:
        nets[2].load_checkpoint(nets[0].checkpoint())
    l0 = nets[2].launches
    for net in nets:
        net.step(331)
    assert nets[2].launches - l0 < 31 * 4 + 2 * 40     # step by step while spikes are under way, then blocks
    same(nets[0], nets[1], "went on")
    same(nets[2], nets[1], "resumed")
