"""The order of the particles in a cell, which a step's gather of the state
restores for cells of up to 64 particles and a kernel of its own for larger
ones: the stable order of the particles by cell, at every boundary between the
two, in both equation modes (integers: exact)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# particles in the one crowded cell: around one warp, around the 64-particle
# line, around the 256 threads and 2048 counts of a CTA, and over 8192
@pytest.mark.parametrize("crowd", [1, 2, 31, 33, 63, 64, 65, 66, 255, 257, 2049, 8193])
@pytest.mark.parametrize("mode", ["paper", "ref"])
def test_stable_order_in_every_cell(pbf, mode, crowd):
    cells = (7, 6, 5) if crowd < 2049 else (70, 60, 50)  # one or several scan tiles
    box = tuple(0.1 * c for c in cells)
    p = pbf.scenes.base_params(box, cells, mode=pbf.MODE_PAPER if mode == "paper" else pbf.MODE_REF_COMPAT)
    p.gravity_y = 0.0
    p.time_step_length = 1e-9  # nothing moves: the step's cells are the ones placed here
    rng = np.random.default_rng(crowd)
    spread = rng.uniform(0.02, np.array(box) - 0.02, (777, 3))
    packed = rng.uniform(0.21, 0.29, (crowd, 3))
    xyz = rng.permutation(np.concatenate([spread, packed]))
    ps = np.zeros(len(xyz), pbf.PARTICLE_DTYPE)
    ps["x"] = xyz.astype(np.float32)
    ps["m"] = 0.125
    with pbf.Simulation(p, ps) as sim:
        sim.init()
        for _ in range(2):  # the second step starts from the first one's order
            sim.step(1)
            hsh, perm, ranges = sim.cells()
            assert np.array_equal(perm, np.argsort(hsh, kind="stable"))
            count = np.bincount(hsh, minlength=p.ncells)
            assert count.max() >= crowd
            first = np.concatenate([[0], np.cumsum(count)[:-1]])
            assert np.array_equal(ranges[:, 0], np.where(count > 0, first, -1))
            sim.set_state(*pbf.state_from_particles(ps))


# on both sides of the particle count up to which the gather orders cells of
# any size; the crowded cells are one warp's, one CTA's and several CTAs'
@pytest.mark.parametrize("n", [65535, 65536, 65537])
@pytest.mark.parametrize("cells", [(32, 32, 16), (29, 113, 5), (1, 1, 1)])
@pytest.mark.parametrize("mode", ["paper", "ref"])
def test_stable_order_around_the_size_rules(pbf, mode, cells, n):
    if cells == (1, 1, 1):
        n -= 61440  # all in one cell: the passes visit n^2 pairs
    box = tuple(0.1 * c for c in cells)
    p = pbf.scenes.base_params(box, cells, mode=pbf.MODE_PAPER if mode == "paper" else pbf.MODE_REF_COMPAT)
    p.gravity_y = 0.0
    p.time_step_length = 1e-9
    p.solver_iterations = 1
    rng = np.random.default_rng(n)
    xyz = rng.uniform(0.02, np.array(box) - 0.02, (n, 3))
    at = 0
    for crowd in (65, 300, 2100):
        c = rng.integers(0, cells)
        xyz[at:at + crowd] = 0.1 * c + rng.uniform(0.021, 0.079, (crowd, 3))
        at += crowd
    ps = np.zeros(n, pbf.PARTICLE_DTYPE)
    ps["x"] = rng.permutation(xyz).astype(np.float32)
    ps["m"] = 0.125
    with pbf.Simulation(p, ps) as sim:
        sim.init()
        for _ in range(2):
            sim.step(1)
            hsh, perm, ranges = sim.cells()
            assert np.array_equal(perm, np.argsort(hsh, kind="stable"))
            count = np.bincount(hsh, minlength=p.ncells)
            first = np.concatenate([[0], np.cumsum(count)[:-1]])
            assert np.array_equal(ranges[:, 0], np.where(count > 0, first, -1))
            assert np.array_equal(ranges[:, 1][count > 0], (first + count - 1)[count > 0])
            sim.set_state(*pbf.state_from_particles(ps))
