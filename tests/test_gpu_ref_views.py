"""pbf_get_cells in REF_COMPAT mode: each view asked for alone, all of them, and
again, on grids that sort by counting and by radix; the views agree with the
positions they were taken from, and looking changes no later step."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


@pytest.mark.parametrize("cells", [(9, 7, 8), (60, 50, 70)])
@pytest.mark.parametrize("count", [1, 1000, 17000])
def test_views(pbf, cells, count):
    p = pbf.scenes.base_params(tuple(0.1 * c for c in cells), cells, mode=pbf.MODE_REF_COMPAT)
    rng = np.random.default_rng(count)
    ps = np.zeros(count, pbf.PARTICLE_DTYPE)
    ps["x"] = rng.uniform(0.15, 0.55, (count, 3)).astype(np.float32)
    ps["m"] = 0.125
    out = []
    for look in (False, True):
        with pbf.Simulation(p, ps) as sim:
            sim.init()
            sim.step(1)
            if look:
                hsh, perm, ranges = sim.cells()
                assert np.array_equal(perm, np.argsort(hsh, kind="stable"))
                first = np.searchsorted(np.sort(hsh), np.arange(p.ncells))
                many = np.bincount(hsh, minlength=p.ncells)
                assert np.array_equal(ranges[:, 0], np.where(many > 0, first, -1))
                assert np.array_equal(ranges[:, 1], np.where(many > 0, first + many - 1, -1))
                for which, whole in enumerate((hsh, perm, ranges)):
                    alone = np.zeros_like(whole)
                    args = [None, None, None]
                    args[which] = alone.ctypes.data_as(C.c_void_p)
                    assert pbf.lib().pbf_get_cells(sim._h, *args) == 0
                    assert np.array_equal(alone, whole)
            sim.step(2)
            if look:
                sim.cells()
            sim.step(1)
            out.append(sim.dumpData())
    for x, y in zip(*out):
        assert np.array_equal(bits(x), bits(y))
