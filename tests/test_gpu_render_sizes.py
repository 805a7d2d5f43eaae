"""Rendering at sizes where a sprite's eight threads and the kept scratch can go
wrong: sprites of less than a pixel to the size cap, cut off at every edge,
images of odd and growing and shrinking size, one particle, and counts that
share factors with the order's step -- pixel for pixel the restatement."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import render as oracle_render

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 8, 89])
def test_sizes(pbf, n):
    p = pbf.scenes.base_params((1.0, 1.0, 1.0), (10, 10, 10))
    rng = np.random.default_rng(n)
    ps = np.zeros(n, pbf.PARTICLE_DTYPE)
    ps["x"] = rng.uniform(0.0, 1.0, (n, 3)).astype(np.float32)
    ps["m"] = 0.125
    with pbf.Simulation(p, ps) as sim:
        sim.init()
        pos, vel = sim.dumpData()
        pos[:, 3] = rng.uniform(0, 2, n)
        sim.set_state(pos, vel)
        pos, _ = sim.dumpData()
        for width, height, near, cap in ((64, 48, 1.0, 64.0), (133, 81, 0.35, 64.0),
                                         (31, 17, 2.0, 5.0), (80, 80, 40.0, 64.0), (1, 1, 1.0, 3.0)):
            cam = pbf.default_camera(p)
            cam.distance *= near
            cam.max_point_size = cap
            img = sim.render(cam, width, height)
            want = oracle_render.render(pos, p, cam, width, height)
            assert np.array_equal(img, want), (width, height, near, cap)


def picture(pbf, p, pos, width, height, near, cap):
    ps = np.zeros(len(pos), pbf.PARTICLE_DTYPE)
    ps["x"] = 0.5
    ps["m"] = 0.125
    with pbf.Simulation(p, ps) as sim:
        sim.init()
        sim.set_state(pos, np.zeros_like(pos))
        cam = pbf.default_camera(p)
        cam.distance *= near
        cam.max_point_size = cap
        return sim.render(cam, width, height)


# 81,919 sprites are drawn in one part; with particles outside the view added,
# which draw nothing, in two, the second taking the image in blocks of eight by
# eight pixels, of which these images hold whole ones, cut ones and less than one
@pytest.mark.parametrize("width, height, near, cap", [(133, 81, 1.0, 12.0), (640, 512, 0.35, 64.0),
                                                      (96, 64, 40.0, 12.0), (5, 3, 1.0, 200.0)])
def test_two_parts_draw_what_one_does(pbf, width, height, near, cap):
    p = pbf.scenes.base_params((1.0, 1.0, 1.0), (10, 10, 10))
    n = 81919
    rng = np.random.default_rng(width)
    pos = rng.uniform(0.0, 1.0, (n, 4)).astype(np.float32)
    pos[1::2, 2] = 0.5  # depths that many share
    want = picture(pbf, p, pos, width, height, near, cap)
    assert len(np.unique(want)) > 2
    for more in (1, 33, 5000):
        outside = np.full((more, 4), 1e6, np.float32)
        for both in (np.concatenate([pos, outside]), np.insert(pos, n // 3, outside, axis=0)):
            assert np.array_equal(picture(pbf, p, both, width, height, near, cap), want)
