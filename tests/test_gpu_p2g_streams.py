"""FP32-form tiled P2G where its streams and parts can go wrong: particle counts
around the table of a warp (30 or 32 particles), streams of unequal length, items
cut into parts (few items) with empty ones, particles of another tile in between
(skipped and counted), every order, collocated and staggered, from positions and
from records (bit for bit the same).

Tolerance 2e-6 of the largest value: a contribution is about 10 roundings of
6e-8, a node sums fewer than 300 of them in at most 4 partial sums."""

import numpy as np
import pytest
import torch

import oracle
from particles import periodic_mesh, rel_err
from picasso_b200 import (APIC, FieldLocation, FixedGrid, cell_sort, create_spline, permute_members,
                          spline_records)

pytestmark = pytest.mark.gpu
TOL = 2e-6


def _run(order, loc, count, tile, chunk, strays, seed):
    stag = loc not in (FieldLocation.Node, FieldLocation.Cell)
    mesh = periodic_mesh(12, halo=1)
    rng = np.random.default_rng(seed)
    x = rng.random((count, 3))
    m = rng.uniform(0.5, 1.5, count).astype(np.float32)
    c = rng.standard_normal((count, 4, 3)).astype(np.float32)
    c[:, 1:] *= 0.1
    sd0 = create_spline(loc, order, mesh, torch.as_tensor(x, device="cuda"))
    _, perm, bins = cell_sort(sd0, tile, chunk=chunk)
    xs, ms, cs = permute_members(perm, sd0.x, torch.as_tensor(m, device="cuda"),
                                 torch.as_tensor(c, device="cuda"))
    use = np.ones(count, bool)
    if strays:  # every fifth particle leaves its tile
        use[::5] = False
        xs[::5] = torch.remainder(xs[::5] + 0.5, 1.0)
    ext = mesh.extent(loc)
    sdo = create_spline(loc, order, mesh, None).desc
    gm_o = np.zeros(ext)
    gmu_o = np.zeros(ext) if stag else np.zeros(ext + (3,))
    xh, mh, ch = xs.cpu().numpy(), ms.double().cpu().numpy(), cs.double().cpu().numpy()
    oracle.apic_p2g(sdo, np.ascontiguousarray(xh[use]), mh[use], np.ascontiguousarray(ch[use]), gm_o,
                    gmu_o)
    sd = create_spline(loc, order, mesh, xs)
    outs = []
    for records in (False, True):
        if records:
            spline_records(sd, bins)
        acc = torch.zeros(ext + (2 if stag else 4,), dtype=torch.int64, device="cuda")
        gm = FixedGrid(acc[..., 0], 36)
        gmu = FixedGrid(acc[..., 1] if stag else acc[..., 1:], 36)
        err = torch.zeros(1, dtype=torch.int32, device="cuda")
        APIC.p2g(ms, cs, gm, gmu, sd, bins=bins, error_count=err)
        assert int(err) == count - use.sum()
        assert rel_err(gm.to_float().cpu().numpy(), gm_o) <= TOL
        assert rel_err(gmu.to_float().cpu().numpy(), gmu_o) <= TOL
        outs.append(acc)
    assert torch.equal(outs[0], outs[1])


@pytest.mark.parametrize("order", [1, 2, 3])
@pytest.mark.parametrize("loc", [FieldLocation.Node, FieldLocation.Cell, FieldLocation.Face(0),
                                 FieldLocation.Edge(2)])
def test_counts(cuda, order, loc):
    for count in (1, 2, 3, 29, 31, 32, 33, 61, 95, 641):
        _run(order, loc, count, (12, 12, 12) if order < 3 else (4, 12, 12), 4096, False, count)


@pytest.mark.parametrize("order", [1, 2, 3])
@pytest.mark.parametrize("strays", [False, True])
def test_parts_and_strays(cuda, order, strays):
    """12^3 cells in few tiles: the items are cut into 2 to 8 parts."""
    for count, tile, chunk in ((900, (4, 8, 8), 4096), (5000, (4, 4, 4), 256), (14000, (3, 5, 4), 97)):
        _run(order, FieldLocation.Node, count, tile, chunk, strays, count)
