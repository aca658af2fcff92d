"""Handles of different sizes that run the same kernels alive together: the
limit on a kernel's dynamic shared memory belongs to the kernel in the context,
not to the handle that was built last.  A launch above the limit is refused, and
the handle would fall back to a slower step form for good: it must take as many
launches as it takes alone, with the same results."""
import numpy as np
import pytest

import mgbrain_b200 as mgb
from test_tile_group_gpu import network
from test_tile_stdp_gpu import network as plastic_network


def make(spec, form, build):
    args, kw = build(seed=7, **spec)
    sim = mgb.Simulator.from_arrays(*args, **dict(kw, seed=5))
    if form is not None:
        sim.set_persistent(form)
    return sim


def outcome(sim, steps=400):
    before = sim.kernel_launches
    sim.run(steps)
    sim.sync()
    launches = sim.kernel_launches - before
    out = launches, sim.read_raster(), sim.state()
    sim.close()
    return out


def check_pair(large, small, form, build=network):
    alone, raster, state = outcome(make(large, form, build))
    a = make(large, form, build)
    b = make(small, form, build)              # built after it, with less shared memory
    outcome(b)
    launches, raster2, state2 = outcome(a)
    assert launches == alone
    for x, y in zip(raster, raster2):
        assert np.array_equal(x, y)
    for key in state:
        assert np.array_equal(state[key].view(np.int32), state2[key].view(np.int32)), key


@pytest.mark.gpu
@pytest.mark.parametrize("delays,weights", [([60], "one"), ([7, 60], "one"), ([7, 60], "ranged")])
def test_a_smaller_tiled_network_built_later(delays, weights):
    check_pair(dict(n=20_000, nx=2000, k=60, delays=delays, weights=weights),
               dict(n=300, nx=30, k=40, delays=[min(d, 9) for d in delays], weights=weights), None)


@pytest.mark.gpu
def test_a_smaller_plastic_network_built_later():
    check_pair(dict(n=3000, nx=300, k=60, delays=[1, 40]), dict(n=300, nx=30, k=40, delays=[1, 2]), None,
               plastic_network)


@pytest.mark.gpu
def test_windowed_group_of_fewer_delays_built_later():
    check_pair(dict(n=800, nx=80, k=60, delays=[8, 900]), dict(n=300, nx=30, k=40, delays=[8, 9]), 3)
