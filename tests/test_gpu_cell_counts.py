"""Counting of cell keys in any order (pbf_op_sort_cells): warps that hold a key in
lanes apart, in two halves, in one run, once, or beside keys past the end, against
the stable order (integers: exact)."""
from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def sorted_cells(pbf, k, ncells):
    n = len(k)
    keys = torch.from_numpy(k.astype(np.uint32).view(np.int32)).cuda()
    size = pbf.op_sort_cells_scratch_bytes(n, ncells)
    scratch = torch.full((size,), 255, dtype=torch.uint8, device="cuda")
    off = torch.empty(ncells + 1, dtype=torch.int32, device="cuda")
    sk, perm = torch.zeros_like(keys), torch.zeros_like(keys)
    st = torch.cuda.current_stream().cuda_stream
    pbf.op_sort_cells(keys.data_ptr(), n, ncells, off.data_ptr(), sk.data_ptr(), perm.data_ptr(),
                      scratch.data_ptr(), size, st)
    pbf.op_sort_cells_status(scratch.data_ptr(), n, ncells, st)
    return [x.cpu().numpy().view(np.uint32) for x in (off, sk, perm)]


PATTERNS = {
    "random": lambda n, c, rng: rng.integers(0, c, n),
    "in turn": lambda n, c, rng: np.arange(n) % c,
    "halves": lambda n, c, rng: np.arange(n) // 16 % c,
    "pairs": lambda n, c, rng: (np.arange(n) // 2 * 7) % c,
    "one in most places": lambda n, c, rng: np.where(rng.random(n) < 0.5, c - 1, rng.integers(0, c, n)),
}


@pytest.mark.parametrize("pattern", PATTERNS)
@pytest.mark.parametrize("n", [31, 33, 1023, 1025, 40007, 1300001])
@pytest.mark.parametrize("ncells", [1, 2, 9, 70, 5003])
def test_keys_in_any_order(pbf, pattern, n, ncells):
    k = PATTERNS[pattern](n, ncells, np.random.default_rng(n + ncells))
    off, sk, perm = sorted_cells(pbf, k, ncells)
    order = np.argsort(k, kind="stable")
    assert np.array_equal(perm, order)
    assert np.array_equal(sk, k[order])
    assert np.array_equal(off, np.searchsorted(k[order], np.arange(ncells + 1)))
