"""The one-launch step with sets that a group's own list does not hold: listed in
global memory, or past that capacity re-derived, beside sets that are held in the
same warp, and with groups past the last particle -- the bits of the one-thread
passes."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


@pytest.mark.parametrize("n", [70, 513, 961, 1024])
@pytest.mark.parametrize("max_neighbours,grow", [(64, 0), (96, 0), (128, 1), (1024, 0)])
def test_uneven_sets(pbf, n, max_neighbours, grow):
    p = pbf.scenes.base_params((1.0, 1.0, 1.0), (10, 10, 10))
    p.max_neighbours, p.grow_lists = max_neighbours, grow
    rng = np.random.default_rng(n)
    ps = np.zeros(n, pbf.PARTICLE_DTYPE)
    ps["m"] = 0.125
    # most within a cell or two of a corner, fewer and fewer away from it; the last
    # slot's cell among the crowded ones
    x = 0.9 - 0.85 * rng.uniform(0.0, 1.0, (n, 3)) ** 3
    ps["x"] = x.astype(np.float32)
    out = []
    for one_thread in (0, 1):
        with pbf.Simulation(p, ps) as sim:
            sim.init()
            t = sim.tuning()
            t.one_thread = one_thread
            sim.set_tuning(t)
            assert (sim.launches_per_step() == 1) == (one_thread == 0)
            sim.step(1)
            stats = sim.neighbour_stats()
            sim.step(3)
            out.append([*sim.dumpData(), sim.density(), np.array(stats, np.float32)])
    assert n < 100 or out[0][3][0] > 64
    for a, b in zip(*out):
        assert np.array_equal(bits(a), bits(b))
