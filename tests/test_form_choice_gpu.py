"""The step form that a caller or the autotuner chose holds, whatever else is set
before the first step."""
import pytest

import mgbrain_b200 as mgb
from test_tile_group_gpu import network


def launches(sim, steps=512):
    sim.run(64)
    sim.sync()
    before = sim.kernel_launches
    sim.run(steps)
    sim.sync()
    return sim.kernel_launches - before


@pytest.mark.gpu
@pytest.mark.parametrize("form,want", [(0, 512), (2, 1), (3, 1)])
def test_set_accumulation_keeps_the_callers_form(form, want):
    args, kw = network(700, 70, 40, [6, 12], 2)
    plain = mgb.Simulator.from_arrays(*args, **kw, seed=5)
    plain.set_accumulation(mgb.ACC_FIXED)
    assert launches(plain) == 1
    plain.close()
    sim = mgb.Simulator.from_arrays(*args, **kw, seed=5)
    sim.set_persistent(form)
    sim.set_accumulation(mgb.ACC_FIXED)
    assert sim.info()["persistent"] == form
    assert launches(sim) == want
    sim.close()
