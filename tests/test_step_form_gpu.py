"""The step form that runs can be seen and chosen: mgc_get_step_form names it (and
the tiles), mgc_set_tiled brings the tiled group back after another form, and a
stored tune report gives the fastest of the other forms.  The tile suites'
networks do run on tiles, and the mailbox edges are met exactly."""
import numpy as np
import pytest

import mgbrain_b200 as mgb
import test_tile_group_gpu as group
import test_tile_stdp_gpu as plastic
from mgbrain_b200 import capi


def make(spec, build=group.network, seed=7):
    args, kw = build(seed=seed, **spec)
    return mgb.Simulator.from_arrays(*args, **dict(kw, seed=5, raster_ids=1 << 21))


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(group.CASES))
def test_networks_of_the_tile_suite_run_on_tiles(name):
    spec = group.CASES[name][0]
    sim = make(spec)
    f = sim.step_form()
    n = spec["n"] + spec["nx"]
    assert f["form"] == capi.FORM_TILED and f["window"] == min(16, min(spec["delays"]))
    assert f["tiles"] >= 1 and f["tiles"] * f["tile_neurons"] >= n and f["tile_neurons"] % 4 == 0
    sim.run(50)
    assert sim.step_form() == f          # the launch was not refused
    sim.close()


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(plastic.CASES))
def test_networks_of_the_plastic_suite_run_on_tiles(name):
    sim = make(plastic.CASES[name], plastic.network)
    f = sim.step_form()
    assert f["form"] == capi.FORM_TILED and f["window"] == 1
    sim.run(50)
    assert sim.step_form() == f
    sim.close()


@pytest.mark.gpu
def test_forms_chosen_and_taken_back():
    spec = group.CASES["one_delay"][0]
    ref = make(spec)
    ref.set_persistent(0)
    ref.run(60 * 7)
    ref.sync()
    sim = make(spec)
    tiled = sim.step_form()
    seen = []
    for choose in (lambda: None, lambda: sim.set_persistent(3), lambda: sim.set_tiled(), lambda: sim.set_tiled(False),
                   lambda: sim.set_persistent(2), lambda: sim.set_tiled(True), lambda: sim.set_persistent(0)):
        choose()
        sim.run(60)
        seen.append(sim.step_form()["form"])
    sim.sync()
    assert seen == [4, 3, 4, 3, 2, 4, 0]
    for x, y in zip(ref.read_raster(), sim.read_raster()):
        assert np.array_equal(x, y)
    assert np.array_equal(ref.state()["V"].view(np.int32), sim.state()["V"].view(np.int32))
    sim.set_tiled()
    assert sim.step_form() == tiled
    sim.close()
    ref.close()
    sim = make(spec)                      # never told a mode: the windowed group in the place of 2
    sim.set_tiled(False)
    assert sim.info()["persistent"] == 2 and sim.step_form() == dict(form=3, window=8, tiles=0, tile_neurons=0, min_steps=0)
    sim.close()


@pytest.mark.gpu
def test_a_network_without_tiles_refuses_them():
    spec = dict(n=300, nx=40, k=30, delays=[2, 900])     # a delay above the group's longest
    sim = make(spec)
    assert sim.step_form()["form"] != capi.FORM_TILED
    with pytest.raises(mgb.MgcError) as e:
        sim.set_tiled()
    assert e.value.status == capi.MGC_ERR_INVALID
    sim.close()


@pytest.mark.gpu
def test_tune_report_names_the_fastest_other_form():
    """A report stored and set on another handle by mgc_set_persistent gives a mode
    that was timed, not the builder's."""
    spec = dict(n=4000, nx=400, k=100, delays=[15], rate=0.002)
    sim = make(spec)
    rep = sim.autotune(steps_per_trial=640)
    assert sim.step_form()["form"] == capi.FORM_TILED     # several times the others' speed here
    assert sim.info()["persistent"] == rep["persistent"]
    sim.set_tiled(False)
    f = sim.step_form()
    assert f["form"] == rep["persistent"]
    assert rep["persistent"] == capi.FORM_WINDOWED      # half the time of mode 2, the builder's
    sim.close()


@pytest.mark.gpu
@pytest.mark.parametrize("extra,k", [(3, 8000), (4, 8000)])
def test_mailbox_holds_its_last_spike_and_one_beyond(extra, k):
    """148 tiles, 11 groups of four inputs each that fire in every step, and `extra`
    more in tile 0: 47 spikes of inputs, a mailbox's most, or 48, the first that goes
    through a list."""
    spec = dict(n=61, nx=148 * 44 + extra, k=k, delays=[1], rate=1.0)
    sim = make(spec)
    f = sim.step_form()
    if f["tiles"] != 148:
        pytest.skip("a device of another size")
    sim.run(8)
    _, counts, ids = sim.read_raster()
    step = ids[counts[0]:counts[0] + counts[1]]
    per_tile = np.bincount((step >> 2) % f["tiles"], minlength=f["tiles"])
    inputs = np.bincount((step[step < spec["nx"]] >> 2) % f["tiles"], minlength=f["tiles"])
    assert inputs[0] == 44 + extra and inputs.max() == 44 + extra and per_tile[0] >= 44 + extra
    sim.close()
    ref = group.run(spec, [100, 57], [0, None], {})
    group.same(ref, group.run(spec, [100, 57], [None, None], {}))


@pytest.mark.gpu
@pytest.mark.parametrize("groups", [11, 12])
def test_mailbox_edges_over_windows_of_four_steps(groups):
    spec = dict(n=61, nx=148 * groups, k=4000, delays=[4, 6], rate=1.0)
    sim = make(spec)
    f = sim.step_form()
    if f["tiles"] != 148:
        pytest.skip("a device of another size")
    assert f["form"] == capi.FORM_TILED and f["window"] == 4
    sim.close()
    ref = group.run(spec, [100, 57], [0, None], {})
    group.same(ref, group.run(spec, [100, 57], [None, None], {}))


@pytest.mark.gpu
@pytest.mark.parametrize("n,delays,form", [(200_000, (5, 8), capi.FORM_TILED), (300_000, (5, 8), capi.FORM_WINDOWED),
                                           (300_000, (8, 8), capi.FORM_TILED), (300_000, (1, 4), capi.FORM_TILED)])
def test_offsets_beyond_l2_keep_the_other_groups(n, delays, form):
    """Large networks with several delays: the tiles' offsets would miss L2."""
    lif = group.LIFC
    pops = [(0, n, mgb.LIFB), (n, n // 10, mgb.POISSON)]
    projs = [(0, 0, 600, 1e-4, *delays), (1, 0, 60, 1e-4, *delays)]
    rate = np.zeros(n + n // 10, np.float32)
    rate[n:] = 0.01
    sim = mgb.Simulator.fixed_indegree(pops, projs, lif, rate=rate, seed=3, conn_seed=2)
    assert sim.step_form()["form"] == form
    sim.run(30)
    sim.sync()
    assert sim.step_form()["form"] == form
    sim.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n,dmin,form", [(45_000, 5, capi.FORM_TILED), (60_000, 5, capi.FORM_WINDOWED),
                                         (60_000, 1, capi.FORM_TILED)])
def test_large_fixed_point_networks_keep_the_other_groups(n, dmin, form):
    pops = [(0, n, mgb.LIFB), (n, n // 10, mgb.POISSON)]
    projs = [(0, 0, 800, 1e-4, dmin, 8), (1, 0, 100, 3e-4, dmin, 8)]     # unequal weights of one sign
    rate = np.zeros(n + n // 10, np.float32)
    rate[n:] = 0.01
    sim = mgb.Simulator.fixed_indegree(pops, projs, group.LIFC, rate=rate, seed=3, conn_seed=2)
    assert sim.info()["accumulation"] == mgb.ACC_FIXED and sim.step_form()["form"] == form
    sim.close()


@pytest.mark.gpu
@pytest.mark.parametrize("inputs,form", [(3000, capi.FORM_TILED), (3200, capi.FORM_GRAPHS)])
def test_long_plastic_lists_keep_the_ring_kernels(inputs, form):
    n = 64
    types = np.full(inputs + n, mgb.LIFB, np.int8)
    types[:inputs] = mgb.POISSON
    src = np.tile(np.arange(inputs, dtype=np.int32), n)
    tar = np.repeat(np.arange(inputs, inputs + n, dtype=np.int32), inputs)
    rate = np.where(types == mgb.POISSON, 0.05, 0.0).astype(np.float32)
    lif = np.zeros(30, np.float32)
    lif[0], lif[4], lif[8], lif[9] = 5e-4, 20.0, 0.002, 0.02
    outs = []
    for choice in (0, None):
        sim = mgb.Simulator.from_arrays(inputs + n, types, src, tar, np.full(len(src), 0.2, np.float32),
                                        np.ones(len(src), np.int32), lif, plastic.STDP, rate=rate, stdp=True, seed=3)
        assert sim.step_form()["form"] == form
        if choice is not None:
            sim.set_persistent(choice)
        sim.run(60)
        sim.sync()
        outs.append((sim.read_raster(), sim.weights()))
        sim.close()
    for x, y in zip(outs[0][0], outs[1][0]):
        assert np.array_equal(x, y)
    assert np.array_equal(outs[0][1].view(np.int32), outs[1][1].view(np.int32))
