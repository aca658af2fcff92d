"""The raster read back in ascending order inside each step whatever its length
(one warp's sort, a block's, the bitmap in shared or device memory), and the
weights in synapse-list order: against numpy on networks whose spikes are known
(POISSON neurons that always fire)."""
import numpy as np
import pytest

import mgbrain_b200 as mgb


def firing(n, which):
    """n neurons of which `which` fire at every step."""
    c = np.zeros(30, np.float32)
    c[0], c[4] = 1e-4, 1.0
    types = np.full(n, mgb.RAW, np.int8)
    types[which] = mgb.POISSON
    rate = np.zeros(n, np.float32)
    rate[which] = 2.0
    one = np.zeros(1, np.int32)
    return (n, types, one, one, np.zeros(1, np.float32), np.full(1, 5, np.int32), c), dict(rate=rate)


@pytest.mark.gpu
@pytest.mark.parametrize("n,count", [(64, 1), (64, 2), (100, 31), (100, 32), (101, 33), (5000, 64), (5000, 65),
                                     (5000, 2047), (5000, 2048), (5001, 2049), (40000, 40000), (1_600_000, 2500),
                                     (1_600_001, 100_000)])
@pytest.mark.parametrize("form", [None, 0, 3])
def test_raster_is_sorted(n, count, form):
    rng = np.random.default_rng(n + count)
    which = np.sort(rng.choice(n, count, replace=False))
    args, kw = firing(n, which)
    sim = mgb.Simulator.from_arrays(*args, **kw, raster_ids=20 * count)
    if form is not None:
        sim.set_persistent(form)
    for steps in (3, 4):
        sim.run(steps)
        first, counts, ids = sim.read_raster()
        assert np.array_equal(counts, np.full(steps, count))
        assert np.array_equal(ids, np.tile(which, steps))
    sim.run(5)
    sim.stage_raster()
    sim.run(2)
    _, counts, ids = sim.collect_raster()
    assert np.array_equal(counts, np.full(5, count)) and np.array_equal(ids, np.tile(which, 5))
    # a reader with less room gets the first ids, in order
    sim.run(3)
    with pytest.raises(mgb.MgcError):
        sim.read_raster(max_ids=max(1, 3 * count))
    sim.close()


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [mgb.capi.MODE_AUTO, mgb.capi.MODE_PUSH, mgb.capi.MODE_PULL])
def test_weights_in_list_order(mode):
    rng = np.random.default_rng(4)
    n, S = 50, 1201
    c = np.zeros(30, np.float32)
    c[0], c[4] = 1e-4, 1.0
    w = rng.normal(size=S).astype(np.float32)
    sim = mgb.Simulator.from_arrays(n, np.full(n, mgb.LIFB, np.int8), rng.integers(0, n, S), rng.integers(0, n, S), w,
                                    rng.integers(1, 9, S), c, mode=mode)
    assert np.array_equal(sim.weights(), w)
