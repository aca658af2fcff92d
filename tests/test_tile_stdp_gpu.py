"""The tiled step group of plastic networks (ring method with STDP, fixed-point
sums), which runs by default, gives the rasters, state, weights and event count
of the graphs of single-step kernels bit for bit: several delays, exponential
currents, every synapse plastic, both sides of a synapse firing in one step,
more spikes in a step than shared memory holds, sizes that are no multiple of 4,
mixed with the other form and across checkpoints."""
import numpy as np
import pytest

import mgbrain_b200 as mgb

import stdp_net

STDP = np.array([0.01, -0.0105, 40.0, 40.0, 1.0, 0.0], np.float32)


def network(n, nx, k, delays, seed, kind=mgb.LIFB, plastic="some", rate=0.05, into_inputs=False):
    rng = np.random.default_rng(seed)
    tot = n + nx
    types = np.full(tot, kind, np.int8)
    types[:nx] = mgb.POISSON
    if tot > 20:
        types[nx + 1], types[nx + 2] = mgb.RAW, mgb.POISSON
    S = n * k
    src = rng.integers(0, tot, S).astype(np.int32)
    tar = rng.integers(0 if into_inputs else nx, tot, S).astype(np.int32)
    w = rng.uniform(0.0, 6.0 / k, S).astype(np.float32)
    w[rng.random(S) < 0.1] = -0.5
    d = rng.choice(np.asarray(delays), S).astype(np.int32)
    d[:len(delays)] = delays
    pl = None if plastic == "all" else (rng.random(S) < 0.5).astype(np.uint8)
    lif = np.zeros(30, np.float32)
    lif[0], lif[4], lif[8], lif[9] = 5e-4, 1.0, 0.002, 0.02
    if kind == mgb.LIF:
        lif[4], lif[12], lif[13], lif[15], lif[16], lif[17] = 0.2, 0.2, 0.2, 0.9, 0.9, 0.98
    r = np.zeros(tot, np.float32)
    r[types == mgb.POISSON] = rate
    v0 = rng.uniform(0, 0.5, tot).astype(np.float32)
    return (tot, types, src, tar, w, d, lif, STDP), dict(rate=r, v_init=v0, stdp=True, plastic=pl, seed=3)


CASES = {
    "one_step": dict(n=300, nx=61, k=30, delays=[1]),
    "delays": dict(n=403, nx=50, k=30, delays=[1, 3, 17]),
    "later": dict(n=202, nx=50, k=40, delays=[4, 9]),
    "all_plastic": dict(n=150, nx=30, k=50, delays=[1, 2], plastic="all"),
    "currents": dict(n=300, nx=60, k=30, delays=[2, 5], kind=mgb.LIF),
    "tiny": dict(n=3, nx=2, k=4, delays=[1], rate=0.4),
    "into_inputs": dict(n=200, nx=100, k=30, delays=[1], rate=0.5, into_inputs=True),
    "many_spikes": dict(n=300, nx=6000, k=40, delays=[1], rate=0.95, into_inputs=True),
}


def outcome(sim):
    sim.sync()
    out = sim.read_raster(max_ids=1 << 22), sim.state(), sim.weights(), sim.info()
    sim.close()
    return out


def same(a, b):
    (_, ca, ia), sa, wa, na = a
    (_, cb, ib), sb, wb, nb = b
    assert np.array_equal(ca, cb) and np.array_equal(ia, ib) and ca.sum() > 0
    for key in sa:
        assert np.array_equal(sa[key].view(np.int32), sb[key].view(np.int32)), key
    assert np.array_equal(wa.view(np.int32), wb.view(np.int32))
    assert na["events"] == nb["events"] and na["step"] == nb["step"] and na["mode"] == mgb.capi.MODE_PUSH


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(CASES))
def test_plastic_tiles_equal_graphs(name):
    args, kw = network(seed=5, **CASES[name])
    kw["raster_ids"] = 1 << 22
    outs = []
    for forms in ([0, None, None, None], [None, None, None, None], [None, 0, None, None]):
        sim = mgb.Simulator.from_arrays(*args, **kw)
        for steps, form in zip((1, 2, 150, 147), forms):
            if form is not None:
                sim.set_persistent(form)
            sim.run(steps)
        outs.append(outcome(sim))
    w0 = args[4]
    assert not np.array_equal(outs[0][2], w0) or name == "tiny"   # something was learned
    same(outs[0], outs[1])
    same(outs[0], outs[2])


@pytest.mark.gpu
def test_plastic_tiles_across_checkpoints_and_rates():
    net = stdp_net.build(n_in=196, n_exc=101)

    def make(form):
        s = mgb.Simulator.from_arrays(net["n"], net["type"], net["src"], net["tar"], net["weight"], net["delay"],
                                      net["lifconst"], net["stdpconst"], stdp=True, plastic=net["plastic"], seed=11)
        if form is not None:
            s.set_persistent(form)
        return s

    ref, a, b = make(0), make(None), make(None)
    b.run(50)                                   # its own weights, then the checkpoint's
    for s in (ref, a):
        s.set_rates(stdp_net.rates(net, 0))
        s.run(301)
    blob = a.checkpoint()
    a.profile(3)                                # steps in another form behind the tiles' back
    b.restore(blob)
    ref.read_raster()
    for s in (ref, b):
        s.set_rates(stdp_net.rates(net, 1))
        s.run(400)
    ref.profile(5)
    b.run(5)
    ref.run(100)
    b.profile(1)
    b.run(99)
    same(outcome(ref), outcome(b))
    a.close()
