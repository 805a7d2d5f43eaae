"""The sorts at the sizes and alignments where their kernels change: a key more
or less than a CTA, a tile and a wave takes, one and four keys per thread, keys
that do and do not start on a 16-byte boundary, and keys whose digits agree
across a warp, in runs, or not at all -- against the stable order (integers:
exact)."""
from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def keys_of(kind, n, top, rng):
    if kind == "random":
        k = rng.integers(0, top, n)
    elif kind == "equal":
        k = np.full(n, top - 1)
    elif kind == "runs":
        k = np.repeat(rng.integers(0, top, n // 5 + 1), 5)[:n]
    else:  # nearly in order
        k = np.clip(np.arange(n) * top // max(n, 1) + rng.integers(-40, 40, n), 0, top - 1)
    return k.astype(np.uint32)


def dev(a):
    return torch.from_numpy(a.view(np.int32)).cuda()


SIZES = [1, 3, 31, 257, 1025, 4095, 4097, 8193, 311297, 1245185]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("bits,kind", [(1, "random"), (9, "runs"), (13, "equal"), (18, "nearly"), (20, "nearly"), (32, "random")])
@pytest.mark.parametrize("shift", [0, 1, 3])
def test_sort_pairs(pbf, n, bits, kind, shift):
    rng = np.random.default_rng(n + bits)
    k = keys_of(kind, n, 1 << bits, rng)
    v = rng.permutation(n).astype(np.uint32)
    buf = torch.zeros(n + 4, dtype=torch.int32, device="cuda")
    buf[shift:shift + n] = dev(k)
    keys = buf[shift:shift + n]
    vals = dev(v)
    size = pbf.op_sort_scratch_bytes(n, bits)
    scratch = torch.empty(size, dtype=torch.uint8, device="cuda")
    ok, ov = torch.empty_like(vals), torch.empty_like(vals)
    order = np.argsort(k, kind="stable")
    st = torch.cuda.current_stream().cuda_stream
    for vp, want in ((None, order.astype(np.uint32)), (vals.data_ptr(), v[order])):
        pbf.op_sort_pairs(keys.data_ptr(), vp, n, bits, ok.data_ptr(), ov.data_ptr(), scratch.data_ptr(), size, st)
        pbf.op_sort_status(scratch.data_ptr(), n, bits, st)
        assert np.array_equal(ok.cpu().numpy().view(np.uint32), k[order])
        assert np.array_equal(ov.cpu().numpy().view(np.uint32), want)


# tiles of 4,096 keys in groups of 16: the last, the first and the only tile of a
# group, one group and several, a warp of one digit and a part of a warp at the end
@pytest.mark.parametrize("tiles", [2, 15, 16, 17, 31, 32, 33, 256, 257, 513])
@pytest.mark.parametrize("more", [-4095, -33, -1, 0])
@pytest.mark.parametrize("bits,kind", [(8, "random"), (18, "equal"), (18, "runs"), (24, "nearly")])
def test_tiles_and_groups(pbf, tiles, more, bits, kind):
    n = 4096 * tiles + more
    rng = np.random.default_rng(n + bits)
    k = keys_of(kind, n, 1 << bits, rng)
    keys = dev(k)
    size = pbf.op_sort_scratch_bytes(n, bits)
    scratch = torch.empty(size, dtype=torch.uint8, device="cuda")
    ok, ov = torch.empty_like(keys), torch.empty_like(keys)
    order = np.argsort(k, kind="stable")
    st = torch.cuda.current_stream().cuda_stream
    pbf.op_sort_pairs(keys.data_ptr(), None, n, bits, ok.data_ptr(), ov.data_ptr(), scratch.data_ptr(), size, st)
    pbf.op_sort_status(scratch.data_ptr(), n, bits, st)
    assert np.array_equal(ok.cpu().numpy().view(np.uint32), k[order])
    assert np.array_equal(ov.cpu().numpy().view(np.uint32), order)


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("ncells,kind", [(1, "equal"), (2048, "runs"), (114688, "nearly"), (114689, "random"), (600000, "nearly")])
def test_sort_cells(pbf, n, ncells, kind):
    rng = np.random.default_rng(n + ncells)
    k = keys_of(kind, n, ncells, rng)
    size = pbf.op_sort_cells_scratch_bytes(n, ncells)
    scratch = torch.empty(size, dtype=torch.uint8, device="cuda")
    off = torch.empty(ncells + 1, dtype=torch.int32, device="cuda")
    ok = torch.empty(n, dtype=torch.int32, device="cuda")
    op = torch.empty_like(ok)
    st = torch.cuda.current_stream().cuda_stream
    keys = dev(k)
    pbf.op_sort_cells(keys.data_ptr(), n, ncells, off.data_ptr(), ok.data_ptr(), op.data_ptr(), scratch.data_ptr(), size, st)
    pbf.op_sort_cells_status(scratch.data_ptr(), n, ncells, st)
    order = np.argsort(k, kind="stable")
    assert np.array_equal(op.cpu().numpy().view(np.uint32), order)
    assert np.array_equal(ok.cpu().numpy().view(np.uint32), k[order])
    want = np.concatenate([[0], np.cumsum(np.bincount(k, minlength=ncells))])
    assert np.array_equal(off.cpu().numpy(), want)


# cells of every size around the half and the whole of a small cell's network,
# their particles in any order
@pytest.mark.parametrize("largest", [2, 7, 8, 9, 15, 16, 17])
def test_small_cells_of_every_size(pbf, largest):
    rng = np.random.default_rng(largest)
    sizes = np.concatenate([np.arange(largest + 1), rng.integers(largest // 2, largest + 1, 9000)])
    k = rng.permutation(np.repeat(np.arange(len(sizes)), sizes)).astype(np.uint32)
    n, ncells = len(k), len(sizes)
    keys = dev(k)
    size = pbf.op_sort_cells_scratch_bytes(n, ncells)
    scratch = torch.empty(max(16, size), dtype=torch.uint8, device="cuda")
    off = torch.empty(ncells + 1, dtype=torch.int32, device="cuda")
    skeys, perm = torch.empty_like(keys), torch.empty_like(keys)
    st = torch.cuda.current_stream().cuda_stream
    pbf.op_sort_cells(keys.data_ptr(), n, ncells, off.data_ptr(), skeys.data_ptr(), perm.data_ptr(), scratch.data_ptr(),
                      size, st)
    order = np.argsort(k, kind="stable")
    assert np.array_equal(perm.cpu().numpy().view(np.uint32), order)
    assert np.array_equal(skeys.cpu().numpy().view(np.uint32), k[order])
    assert np.array_equal(off.cpu().numpy(), np.concatenate([[0], np.cumsum(sizes)]))
