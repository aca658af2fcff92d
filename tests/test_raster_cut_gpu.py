"""Rasters come in arrays of their own, cut to size in place from the capacity
buffers: few ids (the allocator's small blocks) and many (mapped pages)."""
import numpy as np
import pytest

import mgbrain_b200 as mgb

LIFC = np.zeros(30, np.float32)
LIFC[0], LIFC[3], LIFC[4], LIFC[8] = 1e-4, 0.0, 0.02, 0.0005


@pytest.mark.gpu
@pytest.mark.parametrize("n", [37, 14561, 14563, 70001, 1048577])
def test_rasters_own_their_memory(n):
    """POISSON neurons at rate 1 fire in every step: the raster is known; staged and
    read rasters own their memory, cut to size (65,536 ids: the shortest cut in place)."""
    rate = np.zeros(n, np.float32)
    rate[::2] = 1.0
    sim = mgb.Simulator.from_arrays(n, np.full(n, mgb.POISSON, np.int8), np.zeros(1, np.int32), np.zeros(1, np.int32),
                                    np.full(1, 0.1, np.float32), np.full(1, 2, np.int32), LIFC, rate=rate,
                                    raster_ids=20 * n)
    sim.run(9)
    sim.stage_raster()
    sim.run(9)
    staged, read = sim.collect_raster(), sim.read_raster()
    st = sim.state()
    sim.close()
    for first, (f, c, ids) in zip((0, 9), (staged, read)):
        assert f == first and np.array_equal(c, np.full(9, (n + 1) // 2))
        assert np.array_equal(ids.reshape(9, -1), np.tile(np.arange(0, n, 2, dtype=np.int32), (9, 1)))
        assert ids.flags.owndata and ids.flags.c_contiguous and len(ids) == c.sum()
    assert np.array_equal(st["fire_cnt"][1::2], np.zeros(n // 2, np.int32))
