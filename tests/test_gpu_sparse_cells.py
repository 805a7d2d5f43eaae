"""Cells of a grid with fewer than two particles per cell (pbf_op_sort_cells):
around the size up to which a cell is sorted where it is found, in order, reversed
and mixed, against the stable order (integers: exact)."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_cell_counts import sorted_cells

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [2, 3, 4, 5, 16, 17])
@pytest.mark.parametrize("apart", [1, 5, 40000])
def test_small_cells(pbf, size, apart):
    # the particles of a cell `apart` indices from each other, so that their places
    # follow the order in which different threads, warps or CTAs counted them
    cells = 40000 if apart == 40000 else 20000
    i = np.arange(cells * size)
    k = i % cells if apart == 40000 else (i // (size * apart)) * apart + i % apart
    ncells = cells * size
    off, sk, perm = sorted_cells(pbf, k * 2 + 1, 2 * ncells)
    order = np.argsort(k, kind="stable")
    assert np.array_equal(perm, order)
    assert np.array_equal(sk, k[order] * 2 + 1)


@pytest.mark.parametrize("n,ncells", [(1000, 700), (300000, 300001), (1300000, 2600000)])
def test_random_cells(pbf, n, ncells):
    k = np.random.default_rng(n).integers(0, ncells, n)
    off, sk, perm = sorted_cells(pbf, k, ncells)
    assert np.array_equal(perm, np.argsort(k, kind="stable"))
    assert np.array_equal(off, np.searchsorted(np.sort(k), np.arange(ncells + 1)))
