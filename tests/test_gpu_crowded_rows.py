"""List builds over crowded rows: more masks than a thread's queue holds, so that a
warp hands its members on together several times, with lanes whose sets are far
smaller, particles in the outermost cells and a last warp that is not full -- the
bits and counts of the build that stores members as it finds them."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


@pytest.mark.parametrize("n", [16385, 16415, 20000])
@pytest.mark.parametrize("fuse", [0, 1])
def test_masks_and_members_as_found(pbf, n, fuse):
    p = pbf.scenes.base_params((2.0, 0.6, 0.7), (20, 6, 7))
    p.max_neighbours = 512
    rng = np.random.default_rng(n)
    ps = np.zeros(n, pbf.PARTICLE_DTYPE)
    ps["m"] = 0.125
    # every density from a few to some 250 per cell, along x and across the walls
    x = rng.uniform(0.0, 1.0, (n, 3)) ** (2.5, 1.0, 1.0)
    ps["x"] = (x * (1.95, 0.55, 0.65) + 0.025).astype(np.float32)
    out = []
    for masked in (0, 1):
        with pbf.Simulation(p, ps) as sim:
            sim.init()
            t = sim.tuning()
            t.masked_build, t.fuse_first = masked, fuse
            sim.set_tuning(t)
            sim.step(1)
            stats = sim.neighbour_stats()
            sim.step(2)
            out.append([*sim.dumpData(), sim.density(), np.array(stats, np.float32)])
    assert out[0][3][0] > 300  # members: over 14 masks in every row
    for a, b in zip(*out):
        assert np.array_equal(bits(a), bits(b))
