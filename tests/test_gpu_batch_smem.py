"""FP32 batches whose padded P2G tile fits in shared memory alone but not beside the
arguments that the batch's kernels keep there: their tiles stay unpadded.  Against the
single calls, whose tiles have all of the shared memory."""

import pytest
import torch

from particles import rel_err
from picasso_b200 import (APIC, Batch, BatchInstance, FieldLocation, FixedGrid, UniformMesh, cell_sort,
                          create_spline, grid_velocity, permute_members)

pytestmark = pytest.mark.gpu
LOC = FieldLocation.Node


@pytest.mark.parametrize("mode", ["phased", "fused"])
@pytest.mark.parametrize("order,tile", [(1, (56, 24, 9)), (2, (34, 24, 12)), (3, (29, 23, 13))])
def test_padded_tile_beside_the_arguments(cuda, order, tile, mode):
    cells = (60, 25, 15)
    mesh = UniformMesh([0, 0, 0] + [c / 64 for c in cells], cell_size=1 / 64, periodic=(True,) * 3)
    g = torch.Generator(device="cuda").manual_seed(order)
    n = 60 * 25 * 15
    x = torch.rand((n, 3), generator=g, device="cuda", dtype=torch.float64)
    x *= torch.tensor(cells, dtype=torch.float64, device="cuda") / 64
    m = torch.rand(n, generator=g, device="cuda") + 0.5
    c = torch.randn((n, 4, 3), generator=g, device="cuda")
    c[:, 1:] *= 0.1
    _, perm, bins = cell_sort(create_spline(LOC, order, mesh, x), tile)
    x, m, c = permute_members(perm, x, m, c)
    sd = create_spline(LOC, order, mesh, x)

    def grids():
        acc = torch.zeros(mesh.extent(LOC) + (4,), dtype=torch.int64, device="cuda")
        u = torch.zeros(mesh.extent(LOC) + (3,), dtype=torch.float32, device="cuda")
        return acc, FixedGrid(acc[..., 0], 36), FixedGrid(acc[..., 1:], 36), u

    acc, gm, gmu, u = grids()
    APIC.p2g(m, c, gm, gmu, sd, bins=bins)
    grid_velocity(mesh.descriptor(LOC), gm, gmu, u, 1e-12)
    want = torch.zeros_like(c)
    APIC.g2p(u, want, sd, bins=bins)
    acc2, gm2, gmu2, u2 = grids()
    got = c.clone()
    Batch([BatchInstance(sd, m, got, gm2, gmu2, u2, bins, 1e-12)], mode=mode).step(graph=False)
    # FP32 sums of some tens of terms in another order
    for a, b in ((acc, acc2), (u, u2), (want, got)):
        assert rel_err(b.double().cpu().numpy(), a.double().cpu().numpy()) <= 1e-5
