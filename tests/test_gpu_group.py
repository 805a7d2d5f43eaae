"""Gather passes with eight threads per particle (scenes of up to 16,384
particles), and the step as one launch (up to 1,024), against the one-thread passes, which any launch shape but the
default selects: the same operations in the same order, so the same bits."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


def run(pbf, params, ps, steps, single):
    with pbf.Simulation(params, ps) as sim:
        sim.init()
        if single:
            t = sim.tuning()
            t.threads[0] = 256
            sim.set_tuning(t)
        sim.setWaveGenerator(0.004)
        sim.step(steps)
        return [*sim.dumpData(), sim.density()], sim.neighbour_stats()


def same(pbf, params, ps, steps=3):
    a, sa = run(pbf, params, ps, steps, False)
    b, sb = run(pbf, params, ps, steps, True)
    for x, y in zip(a, b):
        assert np.array_equal(bits(x), bits(y))
    assert sa == sb  # the lists hold the same members
    return sa


def cloud(pbf, n, size, seed):
    rng = np.random.default_rng(seed)
    ps = np.zeros(n, pbf.PARTICLE_DTYPE)
    ps["x"] = (0.3 + rng.uniform(0.0, size, (n, 3))).astype(np.float32)
    ps["v"] = rng.normal(0, 0.5, (n, 3)).astype(np.float32)
    ps["m"] = 0.125
    return ps


# a group, a warp's four particles, a CTA's 16, and both sides of the line
@pytest.mark.parametrize("n", [1, 2, 4, 5, 15, 16, 17, 33, 1000, 16383, 16384, 16385])
def test_particle_counts(pbf, n):
    p = pbf.scenes.base_params((2.0, 2.0, 2.0), (20, 20, 20))
    same(pbf, p, cloud(pbf, n, 0.05 * n ** (1 / 3), n))


# sets of about 48 (a round), 64 (the shared list), more than 16 masks of 32
# candidates, and lists that hold only some of the sets
@pytest.mark.parametrize("crowding,max_neighbours", [(1.2, 128), (1.5, 128), (2.0, 128), (4.0, 512), (2.0, 16), (9.0, 64)])
def test_crowded_sets(pbf, crowding, max_neighbours):
    p = pbf.scenes.base_params((1.0, 1.0, 1.0), (10, 10, 10))
    p.max_neighbours = max_neighbours
    p.grow_lists = 0
    n = 1500
    ps = cloud(pbf, n, 0.05 * (n / crowding) ** (1 / 3), int(10 * crowding))
    same(pbf, p, ps, 2)
    most, over = same(pbf, p, ps, 1)  # (the second step starts from a cloud flying apart)
    assert most > 32
    assert (over > 0) == (most > max_neighbours)


@pytest.mark.parametrize("scorr_n,iterations", [(0, 1), (3, 2), (4, 7), (10, 4)])
def test_solver_settings(pbf, scorr_n, iterations):
    p = pbf.scenes.base_params((1.0, 0.1, 1.0), (10, 1, 10))
    p.scorr_n, p.solver_iterations = scorr_n, iterations
    ps = cloud(pbf, 300, 0.3, 5)
    ps["x"][:, 1] = 0.03 + 0.04 * (ps["x"][:, 1] - 0.3) / 0.3
    same(pbf, p, ps, 4)


# the one-launch step: one to sixteen CTAs, both sides of its lines in particles
# and cells
@pytest.mark.parametrize("n,cells", [(63, 10), (64, 10), (65, 18), (513, 10), (1023, 18), (1024, 18), (1025, 18), (1000, 19)])
def test_one_launch(pbf, n, cells):
    p = pbf.scenes.base_params((0.1 * cells,) * 3, (cells,) * 3)
    with pbf.Simulation(p, cloud(pbf, n, 0.05 * n ** (1 / 3), 3 * n)) as sim:
        sim.init()
        assert (sim.launches_per_step() == 1) == (n <= 1024 and cells <= 18)  # 18^3 = 5,832 of 6,144 cells
    same(pbf, p, cloud(pbf, n, 0.05 * n ** (1 / 3), 3 * n), 5)


@pytest.mark.parametrize("crowding,max_neighbours", [(2.0, 128), (4.0, 512), (9.0, 64), (200.0, 1024)])
def test_one_launch_crowded(pbf, crowding, max_neighbours):
    p = pbf.scenes.base_params((1.0, 1.0, 1.0), (10, 10, 10))
    p.max_neighbours = max_neighbours
    p.grow_lists = 0
    same(pbf, p, cloud(pbf, 900, 0.05 * (900 / crowding) ** (1 / 3), int(crowding)), 2)


def test_paths_in_turn(pbf):
    """One simulation through every form of the step in turn: what one leaves
    behind is what the next expects."""
    p = pbf.scenes.base_params((1.0, 1.0, 1.0), (10, 10, 10))
    ps = cloud(pbf, 700, 0.42, 8)

    def tuned(sim, **kw):
        t = pbf.Tuning()
        t.threads[:] = [128, 128, 256, 128, 256, 128]
        t.batch[:] = [4] * 6
        t.fuse_first = t.masked_build = 1
        for k, v in kw.items():
            setattr(t, k, v)
        sim.set_tuning(t)

    with pbf.Simulation(p, ps) as sim:
        sim.init()
        for turn in range(2):
            sim.step(1)
            sim.set_stage_timing(True)
            sim.step(1)
            sim.set_stage_timing(False)
            sim.step(1)
            tuned(sim, radix_sort=1)
            sim.step(1)
            tuned(sim)
            sim.step(1)
            tuned(sim, staged=1)
            sim.step(1)
            tuned(sim, masked_build=0)
            sim.step(1)
            tuned(sim)
            sim.set_graph(False)
            sim.step(1)
            sim.set_graph(True)
            sim.autotune(1)
        got = sim.dumpData()
    with pbf.Simulation(p, ps) as sim:
        sim.init()
        t = sim.tuning()
        t.threads[0] = 256
        sim.set_tuning(t)
        sim.step(16)
        want = sim.dumpData()
    for x, y in zip(got, want):
        assert np.array_equal(bits(x), bits(y))
