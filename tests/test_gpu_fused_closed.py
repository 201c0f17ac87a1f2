"""P2G with the grid update in its flush on closed meshes: the node regions of the last
tiles end where the mesh ends.  Every grid lies between guard values, which must stay,
and grids and velocities are those of the separate passes bit for bit (walls, gravity
and a force field included)."""

import numpy as np
import pytest
import torch

from picasso_b200 import (APIC, FieldLocation, FixedGrid, UniformMesh, cell_sort, create_spline,
                          grid_update, permute_members)

pytestmark = pytest.mark.gpu
LOC = FieldLocation.Node


class Guarded:
    """A grid of `shape` between guards of four of its i-planes on either side."""

    def __init__(self, shape, dtype, value):
        n, guard = int(np.prod(shape)), 4 * int(np.prod(shape[1:]))
        self.all = torch.full((n + 2 * guard,), 77, dtype=dtype, device="cuda")
        self.grid = self.all[guard:guard + n].view(shape)
        self.grid.fill_(value)
        self.guards = self.all[:guard], self.all[guard + n:]

    def intact(self):
        return all(bool((g == 77).all()) for g in self.guards)


@pytest.mark.parametrize("order", [1, 2, 3])
@pytest.mark.parametrize("cells,tile,periodic", [((9, 12, 8), (4, 4, 8), (False,) * 3),
                                                 ((11, 7, 10), (4, 6, 5), (False, True, False)),
                                                 ((7, 7, 9), (12, 12, 14), (False,) * 3)])
def test_closed_mesh(cuda, order, cells, tile, periodic):
    mesh = UniformMesh([0, 0, 0] + [c / 16 for c in cells], cell_size=1 / 16, periodic=periodic,
                       halo_cell_width=2)
    bins_of = [mesh.owned_extent(LOC, d) if periodic[d] else mesh.extent(LOC)[d] for d in range(3)]
    # the fused form needs `order` bins in every tile
    tile = tuple(next(t for t in range(tile[d], 99) if not 0 < bins_of[d] % t < order)
                 for d in range(3))
    rng = np.random.default_rng(order)
    n = 3000
    x = torch.as_tensor(rng.random((n, 3)) * np.array(cells) / 16, device="cuda")
    m = torch.as_tensor(rng.uniform(0.5, 1.5, n), dtype=torch.float32, device="cuda")
    c = torch.as_tensor(rng.standard_normal((n, 4, 3)), dtype=torch.float32, device="cuda")
    _, perm, bins = cell_sort(create_spline(LOC, order, mesh, x), tile, chunk=512)
    x, m, c = permute_members(perm, x, m, c)
    sd = create_spline(LOC, order, mesh, x)
    ext = mesh.extent(LOC)
    f = Guarded(ext + (3,), torch.float64, 0.0)
    f.grid.copy_(torch.as_tensor(rng.standard_normal(ext + (3,))))
    wall = lambda d, kinds: ("none", "none") if periodic[d] else kinds
    upd = dict(dt=2e-3, gravity=(0.0, 1.0, -9.81), f_i=f.grid, wall_width=2,
               walls=[wall(0, ("no_slip", "free_slip")), wall(1, ("free_slip", "no_slip")),
                      wall(2, ("free_slip", "free_slip"))])
    got = []
    for fused in (False, True):
        acc = Guarded(ext + (4,), torch.int64, 0)
        u, u64 = Guarded(ext + (3,), torch.float32, 7.0), Guarded(ext + (3,), torch.float64, 7.0)
        gm, gmu = FixedGrid(acc.grid[..., 0], 36), FixedGrid(acc.grid[..., 1:], 36)
        if fused:
            APIC.p2g_update(m, c, gm, gmu, u.grid, sd, u64_i=u64.grid, bins=bins, **upd)
        else:
            APIC.p2g(m, c, gm, gmu, sd, bins=bins)
            grid_update(sd.desc.mesh, gm, gmu, u.grid, u64_i=u64.grid, **upd)
        assert acc.intact() and u.intact() and u64.intact()
        got.append((acc, u, u64))
    own = [slice(sd.desc.mesh.own_begin[d], sd.desc.mesh.own_begin[d] + sd.desc.mesh.own_extent[d])
           if periodic[d] else slice(None) for d in range(3)]
    for a, b in zip(*got):
        assert torch.equal(a.grid[tuple(own)], b.grid[tuple(own)])
