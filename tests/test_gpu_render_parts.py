"""Images drawn in two parts, the second without the sprites that the first hides
(k_render_far, k_render_splat_rest), against the numpy restatement pixel for pixel:
small sprites on an image of whole blocks of eight by eight pixels, large ones and
an image of cut blocks, and an image of less than one block.  Most particles lie
outside the view, which brings their number over the line and leaves the
restatement few to draw."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import render as oracle_render
from test_host_rules import evaluate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width, height, near, cap, visible",
                         [(96, 64, 1.0, 11.5, 4000), (133, 81, 0.5, 48.0, 400), (5, 3, 1.0, 200.0, 2000)])
def test_hidden_sprites_left_out(pbf, tmp_path, width, height, near, cap, visible):
    p = pbf.scenes.base_params((1.0, 1.0, 1.0), (10, 10, 10))
    n = 81920
    rng = np.random.default_rng(width)
    pos = np.full((n, 4), 1e6, np.float32)
    seen = rng.permutation(n)[:visible]
    pos[seen] = rng.uniform(0.0, 1.0, (visible, 4)).astype(np.float32)
    pos[seen[::3], 2] = 0.5  # depths that many share
    cam = pbf.default_camera(p)
    cam.distance *= near
    cam.max_point_size = cap
    size = min(200.0 / abs(cam.distance), cap)
    rule = f"""std::printf("%d %d\\n", draws_in_two_parts({n}u, {width * height}u, {size}f),
      draws_in_two_parts({n - 1}u, {width * height}u, {size}f));"""
    assert evaluate(pbf, tmp_path, rule) == ["1 0"]
    ps = np.zeros(n, pbf.PARTICLE_DTYPE)
    ps["x"] = 0.5
    ps["m"] = 0.125
    with pbf.Simulation(p, ps) as sim:
        sim.init()
        sim.set_state(pos, np.zeros_like(pos))
        img = sim.render(cam, width, height)
    want = oracle_render.render(pos, p, cam, width, height)
    assert len(np.unique(want)) > 2
    assert np.array_equal(img, want)
