"""The work this library is used for, as measurable cases: networks simulated
through the Python binding (mgbrain_b200.Simulator) over the C ABI.

A case is a dict of plain values.  `prepare` builds what a user's program has
in hand (the handle of a network, its input rates), `run` is one pass through
the public entry points, `work` its unavoidable traffic and operations, and
`exact` the same pass in 64-bit floats by plain numpy for the small networks
given as synapse lists.  Everything follows from (case, seed).

Kinds of network, with the sizes and constants of this repository's
configurations, tests and benchmark:

vogels   Vogels-Abbott-style recurrent network, 80/20 LIFB, p = 0.02, one-step
         delays, 5 % of the neurons kicked one to one by POISSON inputs
         (a synapse list).
brunel   Brunel network by NetGen's fixed-probability rule, generated on the
         device: 80/20 LIFB, p = 0.1, J 0.1 mV, g 5, one 1.5 ms delay.
maker    the model maker's Brunel network (50 % POISSON, 40 % exc, 10 % inh,
         p = 0.1, 1.6 ms), the network the published run times are quoted on.
indeg    fixed in-degree Brunel network generated on the device, uniform
         delays (the large benchmark network), or one delay and g = 2 (volleys).
ranged   exponential-current LIF, weights and delays drawn from ranges (a
         synapse list): unequal weights of one sign.
stdp     all-to-all plastic inputs onto a layer with lateral inhibition, the
         input rates redrawn every 350 ms.
sweep    many small independent Brunel networks in one handle.
build    a fixed in-degree network built, run for 10 ms and dropped.
"""
import math

import numpy as np

import mgbrain_b200 as mgb
from mgbrain_b200 import brunel

DT = 1e-4
J = 1e-4


def listed():
    return [
        # a closed loop: 1 ms of a small network per call, new input rates each
        # time, spikes and state read back (the smallest call: latency counts)
        dict(name="loop_1ms_4k", kind="vogels", n=4000, steps=10, hz=100.0, loop=1),
        # the same network simulated for 1 s: one-step delays, nothing to batch
        dict(name="vogels_4k_1s", kind="vogels", n=4000, steps=10000, hz=100.0, loop=0),
        # an ordinary balanced network, 1.1e7 synapses, 1 s at 20 Hz inputs
        dict(name="brunel_11k_1s", kind="brunel", n=10000, steps=9990, hz=20.0),
        # the published benchmark network at 1e8 synapses, inputs 20 Hz, 0.5 s
        dict(name="maker_1e8", kind="maker", syn=100000000, steps=4992, hz=20.0),
        # the same driven hard (inputs 1 kHz), an odd size
        dict(name="maker_3e7_hot", kind="maker", syn=30011000, steps=1001, hz=1000.0),
        # the large benchmark network, 1.1e9 synapses, autotuned, 0.5 s
        dict(name="indeg_1m", kind="indeg", n=1000000, k=1000, g=5.0, dmin=10, dmax=50, steps=5000, hz=20.0, tune=1),
        # the same network driven (inputs 200 Hz) as a handle runs by default, 0.1 s
        dict(name="indeg_1m_driven", kind="indeg", n=1000000, k=1000, g=5.0, dmin=10, dmax=50, steps=1000, hz=200.0,
             tune=0),
        # synchronous volleys: excitation dominates, one delay
        dict(name="volleys_11k", kind="indeg", n=10000, k=1000, g=2.0, dmin=15, dmax=15, steps=3000, hz=100.0, tune=0),
        # unequal weights and ragged delays, exponential currents, a ragged size
        dict(name="ranged_9k", kind="ranged", n=9013, k=210, dmin=10, dmax=30, steps=600, hz=100.0),
        # learning: seven 350 ms input epochs, the weights read at the end
        dict(name="stdp_784_1600", kind="stdp", n_in=784, n_out=1600, epochs=7, steps=700),
        # a parameter sweep in one handle, 0.2 s
        dict(name="sweep_24", kind="sweep", count=24, n_min=1000, n_max=20000, steps=2000),
        # building a network: 1.1e8 synapses, then 10 ms
        dict(name="build_1e8", kind="build", n=100000, k=1000, g=5.0, dmin=10, dmax=50, steps=100, hz=20.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["vogels", "loop", "brunel", "maker", "indeg", "indeg", "ranged", "stdp", "sweep", "build"])
    if kind == "loop":
        return dict(kind="vogels", n=_log(rng, 500, 8000), steps=_log(rng, 1, 100), hz=rng.choice([50.0, 100.0, 400.0]),
                    loop=1)
    if kind == "vogels":
        return dict(kind=kind, n=_log(rng, 500, 8000), steps=_log(rng, 1000, 10000),
                    hz=rng.choice([50.0, 100.0, 400.0]), loop=0)
    if kind == "brunel":
        return dict(kind=kind, n=_log(rng, 2000, 20000), steps=15 * _log(rng, 40, 600),
                    hz=rng.choice([20.0, 100.0, 200.0]))
    if kind == "maker":
        return dict(kind=kind, syn=_log(rng, 10 ** 6, 10 ** 8), steps=_log(rng, 300, 2000),
                    hz=rng.choice([20.0, 100.0, 500.0]))
    if kind == "indeg":
        one = rng.random() < 0.3
        n = _log(rng, 5000, 30000 if one else 500000)
        dmin = rng.randint(2, 20)
        return dict(kind=kind, n=n, k=min(1000, _log(rng, 100, 1000)), g=rng.choice([2.0, 5.0]) if one else 5.0,
                    dmin=dmin, dmax=dmin if one else dmin + rng.randint(1, 40), steps=_log(rng, 300, 2000),
                    hz=rng.choice([20.0, 100.0, 200.0]), tune=0)
    if kind == "ranged":
        dmin = rng.randint(1, 12)
        return dict(kind=kind, n=_log(rng, 1000, 10000), k=_log(rng, 30, 250), dmin=dmin,
                    dmax=dmin + rng.randint(1, 30), steps=_log(rng, 100, 600), hz=rng.choice([50.0, 100.0]))
    if kind == "stdp":
        return dict(kind=kind, n_in=_log(rng, 100, 800), n_out=_log(rng, 100, 1600), epochs=rng.randint(1, 7),
                    steps=700)
    if kind == "sweep":
        return dict(kind=kind, count=rng.randint(2, 24), n_min=1000, n_max=_log(rng, 4000, 20000),
                    steps=_log(rng, 300, 2000))
    return dict(kind=kind, n=_log(rng, 2000, 100000), k=_log(rng, 100, 1000), g=5.0, dmin=10, dmax=50, steps=100,
                hz=20.0)


# ---- the networks ---------------------------------------------------------------

def _lif_exp():
    """Exponential-current LIF: tau_m 20 ms, tau_syn 5 ms, t_ref 1 ms, V_th 10 mV,
    unit membrane resistance, in the layout of lifconst."""
    c = np.zeros(30, np.float32)
    f = np.float32
    tm, ts = f(0.02), f(0.005)
    cm, cs = np.exp(f(-DT) / tm, dtype=f), np.exp(f(-DT) / ts, dtype=f)
    c[0], c[4], c[6], c[8], c[10], c[11] = DT, 0.01, tm, 0.001, ts, ts
    c[12] = c[13] = ts / (ts - tm) * (cs - cm)
    c[15] = c[16] = cs
    c[17] = cm
    return c


def _vogels(case, seed):
    """Synapse list of the recurrent network; weights shrink with the size's
    in-degree so that every size stays in the same regime."""
    rng = np.random.default_rng((seed, 1))
    n = case["n"]
    ne, nk = int(0.8 * n), max(1, n // 20)
    total = n + nk
    k = max(1, int(0.02 * n))
    src = rng.integers(0, n, (n, k)).astype(np.int32)
    tar = np.repeat(np.arange(n, dtype=np.int32), k)
    src = src.reshape(-1)
    scale = 80.0 / k
    w = np.where(src < ne, 0.00027 * scale, -0.0045 * scale).astype(np.float32)
    src = np.concatenate([np.arange(n, n + nk, dtype=np.int32), src])       # the kick, one to one
    tar = np.concatenate([np.arange(nk, dtype=np.int32), tar])
    w = np.concatenate([np.full(nk, 0.02, np.float32), w])
    types = np.full(total, mgb.LIFB, np.int8)
    types[n:] = mgb.POISSON
    lif = np.zeros(30, np.float32)
    lif[0], lif[3], lif[4], lif[8] = DT, 0.0, 0.01, 0.005
    v0 = np.zeros(total, np.float32)
    v0[:n] = rng.uniform(0.0, 0.01, n)
    rate = np.zeros(total, np.float32)
    rate[n:] = case["hz"] * DT
    return dict(n=total, type=types, src=src, tar=tar, weight=w, delay=np.ones(len(src), np.int32), lif=lif, v0=v0,
                rate=rate, pois=(n, total))


def _ranged(case, seed):
    rng = np.random.default_rng((seed, 2))
    n, k = case["n"], case["k"]
    ne, nx = int(0.8 * n), max(1, n // 10)
    total = n + nx
    kx = max(1, k // 10)
    src = rng.integers(0, n, (n, k)).astype(np.int32)
    ext = rng.integers(n, total, (n, kx)).astype(np.int32)
    src = np.concatenate([src, ext], axis=1)
    tar = np.repeat(np.arange(n, dtype=np.int32), k + kx)
    src = src.reshape(-1)
    # in steps, as NetGen draws ranged weights; the inputs dominate
    we = rng.integers(4, 13, len(src)) * (1e-5 * 200.0 / k)
    wi = rng.integers(-60, -39, len(src)) * (5e-6 * 200.0 / k)
    wx = rng.integers(20, 61, len(src)) * (0.6e-4 * 20.0 / kx)
    w = np.where(src >= n, wx, np.where(src < ne, we, wi)).astype(np.float32)
    types = np.full(total, mgb.LIF, np.int8)
    types[n:] = mgb.POISSON
    v0 = np.zeros(total, np.float32)
    v0[:n] = rng.uniform(0.0, 0.01, n)
    rate = np.zeros(total, np.float32)
    rate[n:] = case["hz"] * DT
    delay = rng.integers(case["dmin"], case["dmax"] + 1, len(src)).astype(np.int32)
    return dict(n=total, type=types, src=src, tar=tar, weight=w, delay=delay, lif=_lif_exp(), v0=v0, rate=rate,
                pois=(n, total))


def _stdp(case, seed):
    rng = np.random.default_rng((seed, 3))
    ni, no = case["n_in"], case["n_out"]
    n, E, I = ni + 2 * no, ni, ni + no
    types = np.full(n, mgb.LIFB, np.int8)
    types[:ni] = mgb.POISSON
    s1 = np.repeat(np.arange(ni), no)
    t1 = np.tile(np.arange(E, E + no), ni)
    w1 = rng.uniform(0.0, 0.3 * 784.0 / ni, len(s1)).clip(0.0, 1.0)
    s2, t2 = np.arange(E, E + no), np.arange(I, I + no)
    ii, ee = np.meshgrid(np.arange(no), np.arange(no), indexing="ij")
    keep = ii != ee
    s3, t3 = I + ii[keep], ee[keep] + E
    lif = np.zeros(30, np.float32)
    lif[0], lif[3], lif[4], lif[8], lif[9] = 5e-4, 0.0, 20.0, 0.005, 0.025
    m = len(s1) + len(s2) + len(s3)
    return dict(n=n, type=types, src=np.concatenate([s1, s2, s3]).astype(np.int32),
                tar=np.concatenate([t1, t2, t3]).astype(np.int32),
                weight=np.concatenate([w1, np.full(len(s2), 25.0), np.full(len(s3), -17.0)]).astype(np.float32),
                delay=np.ones(m, np.int32), plastic=(np.arange(m) < len(s1)).astype(np.uint8), lif=lif,
                v0=np.zeros(n, np.float32), rate=np.zeros(n, np.float32), pois=(0, ni),
                stdp=np.array([0.01, -0.0105, 40.0, 40.0, 1.0, 0.0], np.float32))


def _rates(net, seed, epoch, case):
    """New input rates, as a caller hands them over: the whole network's array."""
    r = np.zeros(net["n"], np.float32)
    a, b = net["pois"]
    u = np.random.default_rng((seed, 4, epoch)).uniform(0.0, 1.0, b - a)
    r[a:b] = u * (63.75 * 5e-4 if case["kind"] == "stdp" else 2.0 * case["hz"] * DT)
    return r


def _indeg(case, seed):
    n, k = case["n"], case["k"]
    ne, nx = int(0.8 * n), max(1, n // 10)
    ni = n - ne
    ke, kx = int(0.8 * k), max(1, k // 10)
    # weaker synapses for a larger in-degree keep the drive per neuron
    w = J * 1000.0 / k
    pops = [(0, ne, mgb.LIFB), (ne, ni, mgb.LIFB), (n, nx, mgb.POISSON)]
    projs = []
    for t in (0, 1):
        projs += [(0, t, ke, w, case["dmin"], case["dmax"]), (1, t, k - ke, -case["g"] * w, case["dmin"], case["dmax"]),
                  (2, t, kx, w, case["dmin"], case["dmax"])]
    rate = np.zeros(n + nx, np.float32)
    rate[n:] = case["hz"] * DT
    v0 = np.random.default_rng((seed, 5)).uniform(0.0, 0.02, n + nx).astype(np.float32)
    return mgb.Simulator.fixed_indegree(pops, projs, brunel.brunel_lifconst(), rate=rate, v_init=v0,
                                        conn_seed=seed + 1, seed=seed + 2, raster_ids=_cap(case))


def _generated(case, seed):
    if case["kind"] == "brunel":
        n = case["n"]
        ne, nx = int(0.8 * n), max(1, n // 10)
        pops = [(ne, mgb.LIFB), (n - ne, mgb.LIFB), (nx, mgb.POISSON)]
        w = J * 10000.0 / n
        conns = [(2, 0, w), (2, 1, w), (0, 0, w), (0, 1, w), (1, 0, -5 * w), (1, 1, -5 * w)]
        total, first, delay, lif = n + nx, n, 15, brunel.brunel_lifconst()
    else:
        size = int(math.sqrt(case["syn"] / 0.05))
        pops = [(size * 5 // 10, mgb.POISSON), (size * 4 // 10, mgb.LIFB), (size // 10, mgb.LIFB)]
        w1, w2 = 0.0001 * 20000 / size, -0.0005 * 20000 / size
        conns = [(0, 1, w1), (0, 2, w1), (1, 1, w1), (1, 2, w1), (2, 2, w2), (2, 1, w2)]
        total, first, delay = sum(p[0] for p in pops), 0, 16
        lif = np.zeros(30, np.float32)
        lif[0], lif[4], lif[8] = DT, 0.02, 0.002
    rate = np.zeros(total, np.float32)
    rate[first:first + (pops[2][0] if case["kind"] == "brunel" else pops[0][0])] = case["hz"] * DT
    projs = [dict(src=s, tar=t, rule=mgb.RULE_PROB, prob=0.1, weight=w, delay=delay) for s, t, w in conns]
    v0 = np.random.default_rng((seed, 6)).uniform(0.0, 0.02, total).astype(np.float32)
    return mgb.Simulator.generated(pops, projs, lif, mt_seed=seed + 1, rate=rate, v_init=v0, seed=seed + 2,
                                   raster_ids=_cap(case))


def _sweep_instances(case, seed):
    p = brunel.sweep_instances(case["count"], case["n_min"], case["n_max"])  # the case's sizes, whatever the seed
    for q in p:
        q["conn_seed"] += 1000 * seed
        q["v0_seed"] += 1000 * seed
    return p


def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case, seed=seed)
    if kind in ("vogels", "ranged", "stdp"):
        net = {"vogels": _vogels, "ranged": _ranged, "stdp": _stdp}[kind](case, seed)
        st["sim"] = mgb.Simulator.from_arrays(
            net["n"], net["type"], net["src"], net["tar"], net["weight"], net["delay"], net["lif"],
            stdpconst=net.get("stdp"), rate=net["rate"], v_init=net["v0"], stdp=kind == "stdp",
            plastic=net.get("plastic"), seed=seed + 2, raster_ids=_cap(case))
        epochs = case["epochs"] if kind == "stdp" else (1 if case.get("loop") else 0)
        st["rates"] = [_rates(net, seed, e, case) for e in range(epochs)]
    elif kind == "indeg":
        st["sim"] = _indeg(case, seed)
        if case["tune"]:
            st["sim"].autotune(rewind=True)
    elif kind in ("brunel", "maker"):
        st["sim"] = _generated(case, seed)
    elif kind == "sweep":
        st["sim"], _ = brunel.sweep_batch(_sweep_instances(case, seed), seed=seed + 2,
                                         raster_ids=_cap(case))
    return st  # build: the description alone


def _cap(case):
    """Spike ids a pass can record: the caller's raster capacity."""
    kind, hz = case["kind"], case.get("hz", 20.0)
    if kind == "stdp":
        n, nx, p, r = 2 * case["n_out"], case["n_in"], 63.75 * 5e-4, 0.05
    elif kind == "sweep":
        n = sum(q["N"] for q in _sweep_instances(case, 0))
        nx, p, r = n // 10, 0.003, 0.01
    elif kind == "maker":
        n = nx = int(math.sqrt(case["syn"] / 0.05)) // 2 + 1
        p, r = hz * DT, 0.05
    else:
        n, nx, p = case["n"], case["n"] // (20 if kind == "vogels" else 10) + 1, 2.0 * hz * DT
        r = 0.05 if kind != "indeg" or case["dmin"] == case["dmax"] else min(0.05, 3e-5 * hz)
        r = 0.001 if kind == "build" else r
    return int(case["steps"] * case.get("epochs", 1) * (n * r + nx * p)) + 65536


def _out(sim, case):
    first, counts, ids = sim.read_raster(max_ids=_cap(case))
    # the caller's buffer, of one size whatever the network did
    buf = np.zeros(_cap(case), np.int32)
    buf[:len(ids)] = ids
    return dict(raster=dict(first=first, counts=counts, ids=buf), state=sim.state())


def run(st):
    case, sim = st["case"], st.get("sim")
    if case["kind"] == "build":
        sim = _indeg(case, st["seed"])
        sim.run(case["steps"])
        out = _out(sim, case)
        sim.close()
        return out
    if case["kind"] == "stdp":
        for r in st["rates"]:
            sim.set_rates(r)
            sim.run(case["steps"])
        out = _out(sim, case)
        out["weights"] = sim.weights()
        return out
    if st.get("rates"):
        sim.set_rates(st["rates"][0])
    sim.run(case["steps"])
    return _out(sim, case)


# ---- the unavoidable work ----------------------------------------------------------

def work(case):
    """Each synapse word that some event of the pass needs read once, the neuron
    state read and written once, the spikes written once; an addition per
    event and five operations per neuron and step.  Only the inputs' spikes
    are known beforehand, so the recurrent events are left out (a lower bound)."""
    kind = case["kind"]
    steps = case["steps"] * case.get("epochs", 1)
    hz = case.get("hz", 20.0)
    p = hz * DT
    if kind == "vogels":
        n, nx = case["n"], max(1, case["n"] // 20)
        syn, out = nx + n * max(1, int(0.02 * n)), 1.0
    elif kind == "ranged":
        n, nx = case["n"], max(1, case["n"] // 10)
        kx = max(1, case["k"] // 10)
        syn, out = n * (case["k"] + kx), n * kx / nx
    elif kind in ("indeg", "build"):
        n, nx = case["n"], max(1, case["n"] // 10)
        kx = max(1, case["k"] // 10)
        syn, out = n * (case["k"] + kx), n * kx / nx
    elif kind == "brunel":
        n, nx = case["n"], max(1, case["n"] // 10)
        syn, out = 0.1 * n * (n + nx), 0.1 * n
    elif kind == "maker":
        size = int(math.sqrt(case["syn"] / 0.05))
        n, nx = size // 2, size // 2
        syn, out = case["syn"], 0.1 * n
    elif kind == "stdp":
        nx, n = case["n_in"], 2 * case["n_out"]
        syn, out, p = case["n_out"] * (nx + case["n_out"]), case["n_out"], 0.5 * 63.75 * 5e-4
    else:
        n = sum(q["N"] for q in _sweep_instances(case, 0))
        nx = n // 10
        syn, out = 110.0 * n, 100.0
    spikes = nx * p * steps
    events = spikes * out
    words = syn if kind == "build" else min(events, syn)
    state = 24.0 * (n + nx)
    return {"bytes": 8.0 * words + 2.0 * state + 4.0 * spikes, "flops": events + 5.0 * n * steps}


# ---- the same pass in 64 bits --------------------------------------------------------

def _philox_uniform(seed, first, last, step):
    """The POISSON draws of neurons [first, last) at a step: Philox4x32-10 with key
    (seed lo, hi) and counter (step lo, hi, neuron / 4, tag), word neuron mod 4."""
    m0, m1 = np.uint64(0xD2511F53), np.uint64(0xCD9E8D57)
    lo = np.uint64(0xFFFFFFFF)
    b0, b1 = first >> 2, (last + 3) >> 2
    c2 = np.arange(b0, b1, dtype=np.uint64)
    c0 = np.full_like(c2, step & 0xFFFFFFFF)
    c1 = np.full_like(c2, step >> 32)
    c3 = np.full_like(c2, 0x504F4953)
    k0, k1 = seed & 0xFFFFFFFF, (seed >> 32) & 0xFFFFFFFF
    for _ in range(10):
        p0, p1 = m0 * c0, m1 * c2
        c0, c1, c2, c3 = ((p1 >> np.uint64(32)) ^ c1 ^ np.uint64(k0), p1 & lo,
                          (p0 >> np.uint64(32)) ^ c3 ^ np.uint64(k1), p0 & lo)
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    u = np.stack([c0, c1, c2, c3], axis=1).reshape(-1)[first - 4 * b0:last - 4 * b0]
    return ((u >> np.uint64(8)) + np.uint64(1)).astype(np.float64) * 2.0 ** -24


def exact(case, seed):
    if case["kind"] not in ("vogels", "ranged", "stdp"):
        return None  # networks generated on the device: not restated here
    net = {"vogels": _vogels, "ranged": _ranged, "stdp": _stdp}[case["kind"]](case, seed)
    steps = case["steps"] * case.get("epochs", 1)
    if case["kind"] == "stdp" and case["n_out"] * case["n_in"] * steps > 7e9:
        return None  # over about 20 seconds
    n, C = net["n"], net["lif"].astype(np.float64)
    stdp = case["kind"] == "stdp"
    P = net["stdp"].astype(np.float64) if stdp else None
    order = np.argsort(net["src"], kind="stable")
    src, tar, delay = net["src"][order], net["tar"][order], net["delay"][order]
    w = net["weight"][order].astype(np.float64)
    plastic = net["plastic"][order] != 0 if stdp else None
    row = np.searchsorted(src, np.arange(n + 1))
    if stdp:
        by_tar = np.argsort(tar, kind="stable")
        col = np.searchsorted(tar[by_tar], np.arange(n + 1))
    M = int(delay.max()) + 1
    ring_e, ring_i = np.zeros((M, n)), np.zeros((M, n))
    V, ie, ii = net["v0"].astype(np.float64), np.zeros(n), np.zeros(n)
    v0 = V.copy()
    refrac, last, count = np.zeros(n, np.int64), np.zeros(n, np.int64), np.zeros(n, np.int64)
    ref_steps = int(round(float(net["lif"][8] / net["lif"][0]))) - 1
    leak = C[9] if C[9] != 0 else float(np.float32(0.005))
    a, b = net["pois"]
    lif = np.flatnonzero(net["type"] != mgb.POISSON)
    rate = net["rate"].astype(np.float64)
    counts, ids = [], []

    def gather(spikes, ptr):
        lens = ptr[spikes + 1] - ptr[spikes]
        return np.repeat(ptr[spikes] - np.concatenate([[0], np.cumsum(lens)[:-1]]), lens) + np.arange(lens.sum())

    def dw(dt, x):
        d = np.where(dt < 0, P[0] * np.exp(dt / P[2]), np.where(dt > 0, P[1] * np.exp(-dt / P[3]), 0.0))
        return np.clip(x + d, P[5], P[4])

    for s in range(steps):
        if s % case["steps"] == 0 and (stdp or case.get("loop")):
            rate = _rates(net, seed, s // case["steps"], case).astype(np.float64)
        re, ri = ring_e[s % M], ring_i[s % M]
        fired = np.zeros(n, bool)
        fired[a:b] = rate[a:b] > _philox_uniform(seed + 2, a, b, s)
        ref = refrac[lif] > 0
        go = lif[~ref]
        refrac[lif[ref]] -= 1
        if case["kind"] == "ranged":
            nv = C[17] * V[go] + C[14] + ie[go] * C[12] + ii[go] * C[13]
            ie[go] *= C[15]
            ii[go] *= C[16]
            f = nv >= C[4]
            nv[f] = C[3]
            ie[go[~f]] += re[go[~f]]
            ii[go[~f]] += ri[go[~f]]
            V[go] = nv
        else:
            f = V[go] >= C[4]
            q = go[~f]
            V[q] += re[q] + ri[q] - leak * V[q]
            V[go[f]] = C[3]
        refrac[go[f]] = ref_steps
        fired[go[f]] = True
        re[:] = 0
        ri[:] = 0
        spk = np.flatnonzero(fired)
        counts.append(len(spk))
        ids.append(spk)
        count[spk] += 1
        last[spk] = s
        if not len(spk):
            continue
        e = gather(spk, row)
        slot = (s + delay[e]) % M
        pos = w[e] > 0
        np.add.at(ring_e, (slot[pos], tar[e][pos]), w[e][pos])
        np.add.at(ring_i, (slot[~pos], tar[e][~pos]), w[e][~pos])
        if stdp:
            pl = e[plastic[e]]
            w[pl] = dw((last[src[pl]] - last[tar[pl]]).astype(np.float64), w[pl])
            back = by_tar[gather(spk, col)]
            back = back[plastic[back] & ~fired[src[back]]]
            w[back] = dw((last[src[back]] - last[tar[back]]).astype(np.float64), w[back])
    Vout = V.copy()
    Vout[a:b] = v0[a:b]
    ids = np.concatenate(ids)
    buf = np.zeros(_cap(case), np.int32)
    buf[:len(ids)] = ids
    out = dict(raster=dict(first=0, counts=np.array(counts, np.int64), ids=buf),
               state=dict(V=Vout, Iexc=ie, Iinh=ii, refrac=refrac.astype(np.int32), last_fired=last.astype(np.int32),
                          fire_cnt=count.astype(np.int32)))
    if stdp:
        full = np.empty_like(w)
        full[order] = w
        out["weights"] = full
    return out
