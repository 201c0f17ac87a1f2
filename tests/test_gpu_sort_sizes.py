"""Cell sort at the sizes where its path changes: one CTA up to 8192 particles
(and 16384 tiles), then radix passes over blocks of 2048 or 3072 elements, with
digits of at most 8 or of 9 bits.  Keys, permutation, tile offsets and the
work-item prefix against a stable sort of the oracle's keys, all bit for bit,
from positions and from keys; packed row widths of the permutation."""

import numpy as np
import pytest
import torch

import oracle
from picasso_b200 import FieldLocation, UniformMesh, cell_sort, create_spline, permute

pytestmark = pytest.mark.gpu


def _check(cells, tile, count, chunk, ordered):
    h = 1.0 / max(cells)
    mesh = UniformMesh([0, 0, 0] + [h * n for n in cells], cell_size=h, periodic=(True, False, True),
                       halo_cell_width=1)
    rng = np.random.default_rng(count)
    x = rng.random((count, 3)) * np.array(cells) * h
    if ordered:
        q = np.floor(x / h).astype(int)
        x = x[np.lexsort((q[:, 2], q[:, 1], q[:, 0]))]
    x[::11, 1] -= 10.0  # outside the closed dimension: sorted last
    sdo = create_spline(FieldLocation.Node, 2, mesh, None).desc
    key_o, perm_o, off_o = oracle.cell_sort(sdo, x, tile)
    items = np.concatenate([[0], np.cumsum(-(-np.diff(off_o) // chunk))])
    sd = create_spline(FieldLocation.Node, 2, mesh, torch.as_tensor(x, device="cuda"))
    unsorted = np.empty(count, np.uint32)
    unsorted[perm_o] = key_o
    keys = torch.as_tensor(unsorted.view(np.int32), device="cuda")
    for source in (None, keys):
        key, perm, bins = cell_sort(sd, tile, chunk=chunk, keys=source)
        assert np.array_equal(key.cpu().numpy().view(np.uint32), key_o)
        assert np.array_equal(perm.cpu().numpy().view(np.uint32), perm_o)
        assert np.array_equal(bins.tile_offset.cpu().numpy(), off_o)
        assert np.array_equal(bins.tile_items.cpu().numpy().view(np.uint32), items)


@pytest.mark.parametrize("count", [1, 31, 1023, 1025, 8191, 8192, 8193, 10240, 10241])
def test_small(cuda, count):
    _check((20, 11, 13), (4, 4, 4), count, 64, False)


@pytest.mark.parametrize("count", [300, 9000])
def test_many_tiles(cuda, count):
    """More tiles than one CTA handles, and keys of 25 bits (9-bit digits)."""
    _check((40, 30, 20), (1, 1, 1), count, 32, False)
    _check((300, 290, 301), (8, 8, 8), count, 32, True)


@pytest.mark.parametrize("ordered", [False, True])
def test_block_sizes(cuda, ordered):
    edge = 148 * 256 * 12
    for count in (edge - 1, edge, edge + 3073):
        _check((64, 50, 40), (4, 8, 8), count, 1024, ordered)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("count", [1, 255, 1025])
def test_permute_row_widths(cuda, dtype, count):
    g = torch.Generator().manual_seed(count)
    perm = torch.randperm(count, generator=g).to(torch.int32).cuda()
    for comp in (1, 2, 3, 4, 6, 8, 12, 24, 81):
        src = torch.randn((count, comp), generator=g, dtype=dtype).cuda()
        assert torch.equal(permute(perm, src), src[perm.long()])
