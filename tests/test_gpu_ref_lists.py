"""REF_COMPAT neighbour lists on the GPU: the pairs of a solver iteration are
found once and kept as lists in the reference's visiting order.  Whatever the
lists hold -- every set, some sets, sets that end in the middle of a word --
and whichever sort laid the cells out, positions, velocities and densities are
the ones of the binary32 restatement of the reference's kernels, bit for bit
(both evaluate the same operations in the same order, so no tolerance)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


def check(pbf, oracle_mod, p, ps, steps, wave=0.0):
    pos0, vel0 = pbf.state_from_particles(ps)
    cfg = oracle_mod.Config(p.x_min, p.x_max, p.y_min, p.y_max, p.z_min, p.z_max, p.x_n, p.y_n, p.z_n,
                            p.time_step_length, p.rest_density)
    with pbf.Simulation(p, ps) as sim:
        sim.init()
        sim.setWaveGenerator(wave)
        sim.step(steps)
        pos, vel = sim.dumpData()
        hsh, perm, ranges = sim.cells()
    want = oracle_mod.refcompat_steps_f32(cfg, pos0, vel0, steps, wave=wave)
    assert np.array_equal(bits(pos), bits(want[0]))
    assert np.array_equal(bits(vel), bits(want[1]))
    assert np.array_equal(perm, np.argsort(hsh, kind="stable"))
    first = np.searchsorted(np.sort(hsh), np.arange(p.ncells))
    count = np.bincount(hsh, minlength=p.ncells)
    assert np.array_equal(ranges[:, 0], np.where(count > 0, first, -1))
    assert np.array_equal(ranges[:, 1], np.where(count > 0, first + count - 1, -1))


# a compressed block (about 60 members inside it): lists that hold nothing
# much, that cut sets off at and off a word's end, and that hold every set
@pytest.mark.parametrize("max_neighbours", [1, 8, 24, 45, 64, 128, 1024])
def test_list_capacities(pbf, oracle_mod, max_neighbours):
    p = pbf.scenes.base_params((1.2, 1.0, 0.9), (12, 10, 9), mode=pbf.MODE_REF_COMPAT)
    p.max_neighbours = max_neighbours
    ps = pbf.generate_block((0.15, 0.15, 0.15), 13, 11, 9, 0.041, 0.004, 0.125, 5)
    check(pbf, oracle_mod, p, ps, 3)


# one long row of candidates (over 32 and over 64 in three cells), particles in
# the outermost cells, an empty half, and a moved wave wall
@pytest.mark.parametrize("count", [1, 33, 200, 513])
def test_crowded_rows_and_edges(pbf, oracle_mod, count):
    p = pbf.scenes.base_params((0.6, 0.5, 1.4), (6, 5, 14), mode=pbf.MODE_REF_COMPAT)
    rng = np.random.default_rng(count)
    ps = np.zeros(count, pbf.PARTICLE_DTYPE)
    ps["x"] = rng.uniform((0.11, 0.11, 0.11), (0.49, 0.39, 0.55), (count, 3)).astype(np.float32)
    ps["v"] = rng.normal(0, 1.0, (count, 3)).astype(np.float32)
    ps["m"] = 0.125
    check(pbf, oracle_mod, p, ps, 2, wave=0.01)


# a grid of mostly empty cells sorts by radix, a fuller one by counting
@pytest.mark.parametrize("cells", [(8, 8, 8), (64, 48, 80)])
def test_both_sorts(pbf, oracle_mod, cells):
    p = pbf.scenes.base_params(tuple(0.1 * c for c in cells), cells, mode=pbf.MODE_REF_COMPAT)
    ps = pbf.generate_block((0.12, 0.14, 0.13), 11, 9, 10, 0.05, 0.002, 0.125, 9)
    check(pbf, oracle_mod, p, ps, 2)


# eight threads per particle up to 16,384 particles, one beyond: both with lists
# that hold every set, some, and almost none
@pytest.mark.parametrize("nz,max_neighbours", [(16, 128), (16, 32), (17, 128), (17, 32), (17, 8)])
def test_threads_per_particle(pbf, oracle_mod, nz, max_neighbours):
    p = pbf.scenes.base_params((1.9, 1.9, 1.2), (19, 19, 12), mode=pbf.MODE_REF_COMPAT)
    p.max_neighbours = max_neighbours
    ps = pbf.generate_block((0.15, 0.15, 0.15), 32, 32, nz, 0.048, 0.008, 0.125, 31)
    check(pbf, oracle_mod, p, ps, 2, wave=0.004)


# rows of hundreds of candidates and sets of hundreds of members, in either form
@pytest.mark.parametrize("count", [700, 17000])
def test_crushed(pbf, oracle_mod, count):
    p = pbf.scenes.base_params((1.0, 1.0, 1.0), (10, 10, 10), mode=pbf.MODE_REF_COMPAT)
    rng = np.random.default_rng(count)
    ps = np.zeros(count, pbf.PARTICLE_DTYPE)
    side = 0.05 * (count / 6.0) ** (1 / 3)
    ps["x"] = (0.15 + rng.uniform(0, side, (count, 3))).astype(np.float32)
    ps["m"] = 0.125
    check(pbf, oracle_mod, p, ps, 1)
