"""The tiled step group (state and input rings on the chip, synapses cut by
tile), which runs by default where the network has its layout, gives the
rasters, state and event count of the graphs of single-step kernels, bit for
bit: at tile edges (sizes that are no multiple of 4, fewer neuron groups than
SMs), for every record form (one delay with one sign per source, both signs,
several delays, fixed point), delays of one step, dense rows (segments shared
by lanes), more spikes in a window than shared memory holds, group lengths that
are no multiple of the window, and mixed with the other forms."""
import numpy as np
import pytest

import mgbrain_b200 as mgb

LIFC = np.zeros(30, np.float32)
LIFC[0], LIFC[3], LIFC[4], LIFC[8] = 1e-4, 0.0, 0.02, 0.0005


def lif_exp():
    c = LIFC.copy()
    c[4], c[12], c[13], c[15], c[16], c[17] = 0.01, 0.004, 0.004, 0.98, 0.97, 0.995
    return c


def network(n, nx, k, delays, seed, kind="lifb", signs="source", weights="one", rate=0.02):
    """n neurons (the last fifth inhibitory), nx POISSON inputs first, k synapses per neuron."""
    rng = np.random.default_rng(seed)
    tot = n + nx
    types = np.full(tot, mgb.POISSON, np.int8)
    types[nx:] = {"lifb": mgb.LIFB, "lif": mgb.LIF}[kind]
    if kind == "lif":
        types[nx::3] = mgb.LIFE
    if tot > 20:
        types[nx + 1], types[nx + 2] = mgb.RAW, mgb.POISSON   # inside a group of LIF neurons
    src = rng.integers(0, tot, (n, k)).reshape(-1).astype(np.int32)
    tar = np.repeat(np.arange(nx, tot, dtype=np.int32), k)
    inh = src >= nx + int(0.8 * n) if signs == "source" else rng.random(len(src)) < 0.2
    j = 0.04 / k if kind == "lifb" else 0.1 / k
    w = np.where(inh, -4 * j, 3 * j).astype(np.float32)
    if weights == "ranged":
        w *= rng.integers(1, 9, len(w)).astype(np.float32) * np.float32(0.25)
    d = rng.choice(np.asarray(delays), len(src)).astype(np.int32)
    d[:len(delays)] = delays
    r = np.zeros(tot, np.float32)
    r[types == mgb.POISSON] = rate
    v0 = rng.uniform(0, 0.02 if kind == "lifb" else 0.01, tot).astype(np.float32)
    return (tot, types, src, tar, w, d, LIFC if kind == "lifb" else lif_exp()), dict(rate=r, v_init=v0)


CASES = {
    "one_delay": (dict(n=1000, nx=101, k=60, delays=[15]), {}),
    "one_delay_both_signs": (dict(n=700, nx=70, k=40, delays=[9], signs="any"), {}),
    "delays": (dict(n=1202, nx=99, k=50, delays=[3, 5, 21]), {}),
    "long_delay": (dict(n=300, nx=40, k=30, delays=[2, 200]), {}),
    "one_step": (dict(n=900, nx=50, k=40, delays=[1]), {}),
    "from_one_step": (dict(n=403, nx=50, k=40, delays=[1, 2, 7]), {}),
    "ranged": (dict(n=801, nx=60, k=40, delays=[4, 11], weights="ranged"), {}),
    "currents": (dict(n=702, nx=60, k=40, delays=[10, 13], kind="lif"), {}),
    "currents_ranged": (dict(n=401, nx=60, k=40, delays=[1, 6], kind="lif", weights="ranged"), {}),
    "tiny": (dict(n=5, nx=2, k=3, delays=[2], rate=0.3), {}),
    "dense": (dict(n=44, nx=12, k=1500, delays=[16], rate=0.1), {}),
    "dense_delays": (dict(n=44, nx=12, k=1500, delays=[8, 9], rate=0.1), {}),
    "many_spikes": (dict(n=600, nx=900, k=50, delays=[16], rate=0.9), {}),
    "many_spikes_ranged": (dict(n=300, nx=900, k=50, delays=[8, 12], rate=0.9, weights="ranged"), {}),
    "big_counts": (dict(n=16, nx=700, k=2000, delays=[8], rate=0.9), {}),
}


def run(spec, chunks, forms, steps_kw):
    args, kw = network(seed=7, **spec)
    sim = mgb.Simulator.from_arrays(*args, **kw, seed=5, raster_ids=1 << 21, **steps_kw)
    for c, f in zip(chunks, forms):
        if f is not None:
            sim.set_persistent(f)
        sim.run(c)
    sim.sync()
    out = sim.read_raster(), sim.state(), sim.info()
    sim.close()
    return out


def same(a, b):
    (fa, ca, ia), sa, na = a
    (fb, cb, ib), sb, nb = b
    assert np.array_equal(ca, cb) and np.array_equal(ia, ib)
    for key in sa:
        assert np.array_equal(sa[key].view(np.int32), sb[key].view(np.int32)), key
    assert na["events"] == nb["events"] and na["step"] == nb["step"]
    assert ca.sum() > 0


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(CASES))
def test_tiles_equal_graphs(name):
    spec, _ = CASES[name]
    chunks = [1, 2, 3, 17, 500, 77, 16, 384]
    ref = run(spec, chunks, [0] + [None] * 7, {})
    got = run(spec, chunks, [None] * 8, {})
    assert got[2]["device_bytes"] > 0
    same(ref, got)
    # another form from the middle of a run on: the tiles' end state is the single-step kernels'
    mixed = run(spec, [333, 5, 662], [None, 0, None], {})
    same(ref, mixed)


@pytest.mark.gpu
def test_tiles_continue_a_checkpoint_and_after_other_forms():
    args, kw = network(900, 80, 50, [7, 18], 3)

    def make():
        return mgb.Simulator.from_arrays(*args, **kw, seed=9)
    ref = make()
    ref.set_persistent(0)
    ref.run(900)
    a = make()
    a.set_persistent(0)
    a.run(301)
    ck = a.checkpoint()
    b = make()                       # never told a form: tiles, from a graph handle's checkpoint
    b.restore(ck)
    b.run(212)
    ck2 = b.checkpoint()
    c = make()
    c.set_persistent(3)              # and back
    c.restore(ck2)
    c.run(900 - 513)
    for s in (ref, c):
        s.sync()
    sr, sc = ref.state(), c.state()
    for key in sr:
        assert np.array_equal(sr[key].view(np.int32), sc[key].view(np.int32)), key
    assert ref.info()["events"] == c.info()["events"]


@pytest.mark.gpu
def test_tiles_poisson_ids_offset():
    """POISSON draws keyed by ids that start inside a group of four."""
    pops = [(0, 300, mgb.LIFB), (300, 60, mgb.LIFB), (360, 41, mgb.POISSON)]
    projs = [(0, 0, 20, 0.002, 5, 9), (0, 1, 20, 0.002, 5, 9), (1, 0, 5, -0.004, 5, 9), (2, 0, 9, 0.004, 5, 9),
             (2, 1, 9, 0.004, 5, 9)]
    rate = np.zeros(401, np.float32)
    rate[360:] = 0.05
    outs = []
    for form in (0, None):
        sim = mgb.Simulator.fixed_indegree(pops, projs, LIFC, rate=rate, seed=3, conn_seed=2, id_offset=6)
        if form is not None:
            sim.set_persistent(form)
        sim.run(701)
        sim.sync()
        outs.append((sim.read_raster(), sim.state(), sim.info()))
        sim.close()
    same(*outs)


@pytest.mark.gpu
def test_tiles_raster_overflow_is_reported():
    args, kw = network(400, 200, 40, [10], 1, rate=0.2)
    sim = mgb.Simulator.from_arrays(*args, **kw, seed=5, raster_ids=5000, raster_steps=4096)
    sim.run(1000)
    with pytest.raises(mgb.MgcError) as e:
        sim.read_raster()
    assert e.value.status == mgb.capi.MGC_ERR_OVERFLOW
    ref = mgb.Simulator.from_arrays(*args, **kw, seed=5)
    ref.set_persistent(0)
    ref.run(1000)
    ref.sync()
    assert np.array_equal(ref.state()["V"], sim.state()["V"])   # the simulation itself is unaffected


@pytest.mark.gpu
def test_tiles_in_fixed_point_on_request():
    args, kw = network(700, 70, 40, [6, 12], 2)
    outs = []
    for form in (0, None):
        sim = mgb.Simulator.from_arrays(*args, **kw, seed=5)
        sim.set_accumulation(mgb.capi.ACC_FIXED)
        if form is not None:
            sim.set_persistent(form)
        sim.run(600)
        sim.sync()
        outs.append((sim.read_raster(), sim.state(), sim.info()))
        sim.close()
    same(*outs)


@pytest.mark.gpu
@pytest.mark.parametrize("nx,delays", [(2, [1]), (3, [1]), (5, [3, 4]), (148 * 44 + 3, [1]), (148 * 44 + 4, [1]),
                                       (148 * 12, [4, 6]), (148 * 12 - 4, [4, 6])])
def test_tiles_mailbox_edges(nx, delays):
    """Inputs that fire in every step fill a tile's mailbox place to a chunk's edge
    (2 and 3 spikes, 5 and 6), to its last spike and one beyond (47 and 48)."""
    spec = dict(n=61, nx=nx, k=40, delays=delays, rate=1.0)
    ref = run(spec, [100, 57], [0, None], {})
    same(ref, run(spec, [100, 57], [None, None], {}))
