"""The tiled step group's windows are counted in 32 bits; a run that passes the
end of the count gives the rasters and state of the graphs."""
import numpy as np
import pytest

import mgbrain_b200 as mgb
from test_tile_group_gpu import network
from test_tile_stdp_gpu import network as plastic_network


@pytest.mark.gpu
@pytest.mark.parametrize("build,spec", [
    (network, dict(n=900, nx=300, k=40, delays=[1], rate=0.2)),
    (network, dict(n=1000, nx=101, k=60, delays=[15])),
    (plastic_network, dict(n=403, nx=150, k=30, delays=[1, 3, 17])),
], ids=["one_step", "windows_of_15", "plastic"])
def test_count_of_windows_wraps(build, spec):
    args, kw = build(seed=4, **spec)
    ref = mgb.Simulator.from_arrays(*args, **dict(kw, seed=5))
    ref.set_persistent(0)
    sim = mgb.Simulator.from_arrays(*args, **dict(kw, seed=5))
    sim.selftest_tile_epoch(0xffffffff - 25)
    for steps in (40, 200, 1, 300):
        for s in (ref, sim):
            s.run(steps)
            s.sync()
        for x, y in zip(ref.read_raster(), sim.read_raster()):
            assert np.array_equal(x, y)
    a, b = ref.state(), sim.state()
    for key in a:
        assert np.array_equal(a[key].view(np.int32), b[key].view(np.int32)), key
    assert ref.info()["events"] == sim.info()["events"]
    ref.close()
    sim.close()
