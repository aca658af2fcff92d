"""Device memory that only makes a handle faster (the tiled group's copy of the
synapses, the kept buffer of plastic weights) is done without where the device has
none: the network is built and runs in another form, with the same results."""
import gc

import numpy as np
import pytest
import torch

import mgbrain_b200 as mgb
import test_tile_group_gpu as group
import test_tile_stdp_gpu as plastic
from mgbrain_b200 import capi

NETS = {"one_delay": (group.network, group.CASES["one_delay"][0]),
        "ranged": (group.network, group.CASES["ranged"][0]),
        "plastic": (plastic.network, plastic.CASES["delays"])}


def outcome(sim):
    sim.run(300)
    sim.sync()
    return sim.read_raster(), sim.state(), sim.weights()


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(NETS))
def test_networks_are_built_without_the_tiles_memory(name):
    build, spec = NETS[name]
    args, kw = build(seed=7, **spec)
    make = lambda: mgb.Simulator.from_arrays(*args, **dict(kw, seed=5))  # noqa: E731
    ref = make()
    ref.set_persistent(0)
    want = outcome(ref)
    ref.close()
    gc.collect()
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    without = k = 0
    while True:
        k += 1
        assert k < 500
        mgb.fault_inject_alloc(k)
        try:
            sim = make()
        except mgb.MgcError as e:
            assert e.status == capi.MGC_ERR_NOMEM and without == 0, (k, str(e))
            continue                          # memory that the handle cannot do without
        finally:
            mgb.fault_inject_alloc(0)
        tiled = sim.step_form()["form"] == capi.FORM_TILED
        if not tiled or without == 0:
            got = outcome(sim)
            for x, y in zip(want[0], got[0]):
                assert np.array_equal(x, y)
            for key in want[1]:
                assert np.array_equal(want[1][key].view(np.int32), got[1][key].view(np.int32)), key
            assert np.array_equal(want[2].view(np.int32), got[2].view(np.int32))
        sim.close()
        without += not tiled
        if tiled and without > 0:
            break
    assert without >= 6                       # several of its allocations, each given up cleanly
    gc.collect()
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] > free0 - (64 << 20)


def tiled_net():
    args, kw = group.network(seed=7, n=4000, nx=400, k=100, delays=[15], rate=0.002)
    return mgb.Simulator.from_arrays(*args, **dict(kw, seed=5))


@pytest.mark.gpu
def test_another_form_gives_the_tiles_memory_back():
    sim = tiled_net()
    held = sim.info()["device_bytes"]
    copy = 2 * 4000 * 100                       # 16-bit records at least
    sim.set_persistent(3)
    assert sim.info()["device_bytes"] < held - copy
    sim.set_tiled()
    assert sim.info()["device_bytes"] == held
    sim.set_tiled(False)
    assert sim.info()["device_bytes"] < held - copy
    sim.autotune(steps_per_trial=64)            # times the tiles all the same
    assert sim.step_form()["form"] == capi.FORM_TILED and sim.info()["device_bytes"] == held
    sim.close()


@pytest.mark.gpu
def test_memory_asked_for_comes_before_the_tiles():
    """Pull steps' rows that fit without the tiles take their place."""
    sim = tiled_net()
    ref = tiled_net()
    ref.set_persistent(0)
    for s in (sim, ref):
        s.run(100)
        s.sync()
    for k in range(1, 9):                       # every allocation of the rows
        s = tiled_net()
        mgb.fault_inject_alloc(k)
        try:
            s.set_pull(500)
        finally:
            mgb.fault_inject_alloc(0)
        assert s.step_form()["form"] != capi.FORM_TILED
        s.close()
    mgb.fault_inject_alloc(1)
    try:
        sim.stage_raster()
    finally:
        mgb.fault_inject_alloc(0)
    assert sim.step_form()["form"] != capi.FORM_TILED
    for x, y in zip(sim.collect_raster(), ref.read_raster()):
        assert np.array_equal(x, y)
    for s in (sim, ref):
        s.run(100)
        s.sync()
    for x, y in zip(sim.read_raster(), ref.read_raster()):
        assert np.array_equal(x, y)
    sim.close()
    ref.close()


@pytest.mark.gpu
def test_rows_that_do_not_fit_leave_nothing_behind():
    sim = tiled_net()
    sim.set_persistent(3)
    held = sim.info()["device_bytes"]
    for k in range(1, 9):
        mgb.fault_inject_alloc(k)
        with pytest.raises(mgb.MgcError) as e:
            sim.set_pull(500)
        mgb.fault_inject_alloc(0)
        assert e.value.status == capi.MGC_ERR_NOMEM
        assert sim.info()["device_bytes"] == held
    sim.set_pull(500)
    sim.run(200)
    sim.sync()
    sim.close()


@pytest.mark.gpu
@pytest.mark.parametrize("big", [False, True])
def test_weights_are_read_on_a_full_device(big):
    n, k = (20_000, 250) if big else (300, 20)       # (5e6 synapses: two stretches)
    args, kw = group.network(seed=7, n=n, nx=40, k=k, delays=[3, 9], weights="ranged")
    sim = mgb.Simulator.from_arrays(*args, **kw)
    mgb.fault_inject_alloc(1)
    try:
        w = sim.weights()
    finally:
        mgb.fault_inject_alloc(0)
    assert np.array_equal(w.view(np.int32), args[4].view(np.int32))
    assert np.array_equal(w, sim.weights())
    sim.close()
