"""Calls of a few steps: the tiled step group keeps the inputs in flight on the
device between its launches, and other forms, checkpoints and new rates in between
leave nothing stale: rasters, state and event counts equal the graphs' after every
call."""
import numpy as np
import pytest

import mgbrain_b200 as mgb
import test_tile_group_gpu as group
from mgbrain_b200 import capi

CALLS = [1, 2, 1, 7, 30, 3, 3, 64, 5, 130, 1, 1, 40]


def pair(spec, **more):
    args, kw = group.network(seed=11, **spec)
    ref = mgb.Simulator.from_arrays(*args, **dict(kw, seed=5, raster_ids=1 << 21))
    ref.set_persistent(0)
    return ref, mgb.Simulator.from_arrays(*args, **dict(kw, seed=5, raster_ids=1 << 21)), args, kw


def check(ref, sim):
    for s in (ref, sim):
        s.sync()
    for x, y in zip(ref.read_raster(), sim.read_raster()):
        assert np.array_equal(x, y)
    a, b = ref.state(), sim.state()
    for key in a:
        assert np.array_equal(a[key].view(np.int32), b[key].view(np.int32)), key
    assert ref.info()["events"] == sim.info()["events"]


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(group.CASES))
def test_calls_of_a_few_steps(name):
    ref, sim, _, _ = pair(group.CASES[name][0])
    for c in CALLS:
        ref.run(c)
        sim.run(c)
        check(ref, sim)
    assert sim.step_form()["form"] == capi.FORM_TILED


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["one_delay", "delays", "from_one_step", "ranged", "currents_ranged"])
def test_other_steps_between_them(name):
    """Steps in another form, a checkpoint of another past at the same step, new
    rates: nothing of the inputs that the group had kept comes back."""
    ref, sim, args, kw = pair(group.CASES[name][0])
    for s in (ref, sim):
        s.run(50)
    check(ref, sim)
    saved = sim.checkpoint()
    rate2 = np.where(kw["rate"] > 0, 0.3, 0.0).astype(np.float32)
    for s in (ref, sim):
        s.set_rates(rate2)
        s.run(20)
    check(ref, sim)
    sim.profile(3)                       # steps in another form
    ref.run(3)
    ref.read_raster(), sim.read_raster()
    for s in (ref, sim):
        s.run(21)
    check(ref, sim)
    other = mgb.Simulator.from_arrays(*args, **dict(kw, seed=77, raster_ids=1 << 21))
    other.run(50)
    other.read_raster()
    other.run(20)                        # the same step, another past
    blob = other.checkpoint()
    sim.restore(saved)
    sim.run(20)
    sim.sync()
    sim.restore(blob)
    ref.restore(blob)
    sim.set_rates(kw["rate"])
    ref.set_rates(kw["rate"])
    for c in (1, 33):
        for s in (ref, sim):
            s.run(c)
        check(ref, sim)
    for s in (ref, sim, other):
        s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("build", ["static", "plastic"])
def test_calls_below_the_shortest_take_the_other_form(build):
    """A call of fewer than min_steps steps is not worth the group's launch."""
    import test_tile_stdp_gpu as plastic
    if build == "static":
        args, kw = group.network(seed=3, **group.CASES["one_delay"][0])
    else:
        args, kw = plastic.network(seed=3, **plastic.CASES["delays"])
    sim = mgb.Simulator.from_arrays(*args, **dict(kw, seed=5))
    shortest = sim.step_form()["min_steps"]
    assert shortest >= 2
    sim.run(100)
    sim.sync()
    with pytest.raises(mgb.MgcError):        # (a wait that runs out shows which form runs)
        sim.selftest_tile_timeout()
        sim.sync()
    step = sim.info()["step"]
    sim.run(shortest)                        # the tiled group's launch, refused since
    assert sim.info()["step"] == step
    sim.run(shortest - 1)                    # another form's
    assert sim.info()["step"] == step + shortest - 1
    sim.close()


@pytest.mark.gpu
@pytest.mark.parametrize("delays", [[12, 30], [5, 8]])
def test_windowed_and_pipelined_calls_mixed(delays):
    """A handle without tiles, never told a mode: calls of one or two steps run
    pipelined, longer ones windowed, with the accumulators' cycle moved between."""
    ref, sim, _, _ = pair(dict(n=1202, nx=99, k=50, delays=delays))
    sim.set_tiled(False)
    assert sim.step_form()["form"] == capi.FORM_WINDOWED
    for c in [2, 1] + CALLS:
        ref.run(c)
        sim.run(c)
        check(ref, sim)
