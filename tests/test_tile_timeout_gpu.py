"""A wait of the tiled step group that runs out: sync reports it, the handle
takes no further step in that group (the counters that the launch left would give
raster places outside their arrays), and a checkpoint loaded afterwards brings it
back whole, with the rasters, state and event count of the graphs."""
import numpy as np
import pytest

import mgbrain_b200 as mgb
from test_tile_group_gpu import network
from test_tile_stdp_gpu import network as plastic_network

NETS = {
    "one_delay": (network, dict(n=1000, nx=101, k=60, delays=[15])),
    "ranged": (network, dict(n=801, nx=60, k=40, delays=[4, 11], weights="ranged")),
    "plastic": (plastic_network, dict(n=403, nx=50, k=30, delays=[1, 3, 17])),
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(NETS))
def test_timed_out_wait_is_reported_and_a_checkpoint_recovers(name):
    build, spec = NETS[name]
    args, kw = build(seed=4, **spec)

    def make():
        return mgb.Simulator.from_arrays(*args, **dict(kw, seed=5))
    ref = make()
    ref.set_persistent(0)
    ref.run(200)
    ref.read_raster()
    ref.run(400)
    ref.sync()
    sim = make()
    sim.run(200)
    sim.sync()
    sim.read_raster()
    saved = sim.checkpoint()
    sim.selftest_tile_timeout()
    for _ in range(2):
        with pytest.raises(mgb.MgcError) as e:
            sim.sync()
        assert e.value.status == mgb.capi.MGC_ERR_CUDA
        sim.run(50)                       # does nothing
    assert sim.info()["step"] == 200
    sim.restore(saved)
    sim.run(400)
    sim.sync()
    for x, y in zip(ref.read_raster(), sim.read_raster()):
        assert np.array_equal(x, y)
    a, b = ref.state(), sim.state()
    for key in a:
        assert np.array_equal(a[key].view(np.int32), b[key].view(np.int32)), key
    assert ref.info()["events"] == sim.info()["events"]
    if name == "plastic":
        assert np.array_equal(ref.weights().view(np.int32), sim.weights().view(np.int32))
    ref.close()
    sim.close()


@pytest.mark.gpu
def test_other_forms_have_no_tile_wait_to_run_out():
    args, kw = network(seed=4, **NETS["one_delay"][1])
    sim = mgb.Simulator.from_arrays(*args, **kw, seed=5)
    sim.set_persistent(0)
    with pytest.raises(mgb.MgcError) as e:
        sim.selftest_tile_timeout()
    assert e.value.status == mgb.capi.MGC_ERR_INVALID
    sim.close()
