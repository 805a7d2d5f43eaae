"""One thread per particle in the default launch shapes (pbf_tuning.one_thread):
kept when the tuning is read and set again, and the same bits as the passes a
small scene takes by itself."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


@pytest.mark.parametrize("block", [(10, 9, 8), (16, 16, 16)])  # one launch a step, eight threads
def test_choice_is_kept(pbf, block):
    sc = pbf.scenes.dam_break(block, (1.6, 1.6, 1.6), seed=61)
    out = []
    for one_thread in (0, 1):
        with pbf.Simulation(sc.params, sc.particles) as sim:
            sim.init()
            t = sim.tuning()
            assert t.one_thread == 0
            t.one_thread = one_thread
            sim.set_tuning(t)
            launches = sim.launches_per_step()
            sim.step(2)
            sim.set_tuning(sim.tuning())
            assert sim.tuning().one_thread == one_thread
            assert sim.launches_per_step() == launches
            assert launches > 1 or (one_thread == 0 and sc.n <= 1024)
            sim.step(2)
            out.append(sim.dumpData())
            tuned = sim.autotune(1)
            launches = sim.launches_per_step()
            sim.set_tuning(tuned)
            assert sim.launches_per_step() == launches
    for x, y in zip(*out):
        assert np.array_equal(bits(x), bits(y))
