"""A batch that holds fewer cells than it has room for: the scan over its cells
takes other tiles than the full batch's would, on control words that were zeroed
for them as well.  Bit for bit the scenes stepped alone."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


def alone(pbf, scene, steps):
    with pbf.Simulation(scene.params, scene.particles) as sim:
        sim.init()
        sim.step(steps)
        return sim.dumpData()


@pytest.mark.parametrize("max_cells", [114689, 131072, 458752, 500000])
def test_fewer_cells_than_room(pbf, max_cells):
    torch = pytest.importorskip("torch")
    dam = pbf.scenes.dam_break
    scenes = [dam((12, 10, 14), (6.4, 3.2, 3.2), seed=21, name="65,536 cells"),
              dam((16, 9, 11), (3.2, 3.2, 3.2), seed=22, name="32,768 cells"),
              dam((7, 8, 9), (1.6, 1.6, 1.6), seed=23, name="4,096 cells")]
    # memory that was in use before, with every bit set
    used = [torch.full((1 << 20,), -1, dtype=torch.int32, device="cuda") for _ in range(64)]
    torch.cuda.synchronize()
    del used
    torch.cuda.empty_cache()
    with pbf.Batch(scenes[0].params, 3, sum(s.n for s in scenes), max_cells) as b:
        ids = [b.add_scene(s.params, s.particles) for s in scenes]
        b.step(3)
        for i, s in zip(ids, scenes):
            for got, want in zip(b.dump_scene(i), alone(pbf, s, 3)):
                assert np.array_equal(bits(got), bits(want)), s.name
        b.remove_scene(ids[1])  # a layout of fewer tiles, then of more again
        b.step(2)
        ids[1] = b.add_scene(scenes[1].params, scenes[1].particles)
        b.step(1)
        for i, s, steps in zip(ids, scenes, (6, 1, 6)):
            for got, want in zip(b.dump_scene(i), alone(pbf, s, steps)):
                assert np.array_equal(bits(got), bits(want)), s.name
