"""The tiled step group where a tile has more spikes in a window than it has
threads (512): its lists are then written to the raster in several rounds while
other warps of the block may already be in the next window's update."""
import numpy as np
import pytest

import mgbrain_b200 as mgb
from test_tile_group_gpu import network


def rasters(spec, form):
    args, kw = network(seed=7, **spec)
    sim = mgb.Simulator.from_arrays(*args, **kw, seed=5, raster_ids=1 << 23)
    if form is not None:
        sim.set_persistent(form)
    out = []
    for steps in (1, 799, 640, 500):
        sim.run(steps)
        sim.sync()
        out.append(sim.read_raster(max_ids=1 << 23))
    state, events = sim.state(), sim.info()["events"]
    sim.close()
    return out, state, events


@pytest.mark.gpu
@pytest.mark.parametrize("delays,weights", [([16], "one"), ([16, 19], "ranged")])
@pytest.mark.parametrize("rate", [0.65, 0.8])
def test_more_spikes_a_tile_and_window_than_threads(delays, weights, rate):
    # 8,064 neurons on 148 tiles, 54 inputs each: 560 to 690 spikes a tile and window of 16 steps
    spec = dict(n=64, nx=8000, k=10_000, delays=delays, rate=rate, weights=weights)
    ref, sr, er = rasters(spec, 0)
    got, sg, eg = rasters(spec, None)
    assert len(ref[1][2]) / (799 / 16) / 148 > 512
    for (fa, ca, ia), (fb, cb, ib) in zip(ref, got):
        assert fa == fb and np.array_equal(ca, cb) and np.array_equal(ia, ib)
    for key in sr:
        assert np.array_equal(sr[key].view(np.int32), sg[key].view(np.int32)), key
    assert er == eg
