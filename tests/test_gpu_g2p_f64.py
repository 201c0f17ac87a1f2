"""FP64 APIC G2P: gathered from the node tile of cell-sorted particles or from
global memory (any order), with results staged per warp.  Against the oracle to
1e-12 of the largest value (some 100 roundings of 1.1e-16 per result, no
cancellation beyond the values' own size), and tile = global bit for bit, for
bins that match, bins the particles have left since the sort, particles outside
the mesh, tiles larger than the mesh and strided particle members."""

import numpy as np
import pytest
import torch

import oracle
from particles import rel_err
from picasso_b200 import APIC, FieldLocation, UniformMesh, cell_sort, create_spline, permute_members

pytestmark = pytest.mark.gpu
TOL = 1e-12


def _setup(cells, periodic, count, seed):
    h = 1.0 / max(cells)
    mesh = UniformMesh([0, 0, 0] + [h * n for n in cells], cell_size=h, periodic=(periodic,) * 3,
                       halo_cell_width=0 if periodic else 2)
    rng = np.random.default_rng(seed)
    x = rng.random((count, 3)) * np.array(cells) * h
    ext = mesh.extent(FieldLocation.Node)
    return mesh, rng, x, rng.standard_normal(ext + (3,))


@pytest.mark.parametrize("cells,periodic,tile", [((12, 9, 17), True, (4, 8, 8)),
                                                 ((3, 2, 5), True, (4, 4, 8)),
                                                 ((7, 10, 6), False, (2, 3, 4))])
@pytest.mark.parametrize("order", [1, 2, 3])
@pytest.mark.parametrize("moved", [False, True])
def test_tiled_equals_global_and_oracle(cuda, order, cells, periodic, tile, moved):
    loc = FieldLocation.Node
    for count in (1, 33, 129, 2500):
        mesh, rng, x, u = _setup(cells, periodic, count, 10 * order + count)
        if not periodic and count > 1:
            x[::9] -= 50.0 * mesh.cell_size
        xd = torch.as_tensor(x, device="cuda")
        ud = torch.as_tensor(u, device="cuda")
        _, perm, bins = cell_sort(create_spline(loc, order, mesh, xd), tile, chunk=64)
        (xs,) = permute_members(perm, xd)
        if moved:  # half of the particles have moved a cell and a half since the sort
            shift = 1.5 * mesh.cell_size
            xs[::2, 1] = torch.where(xs[::2, 1] > shift, xs[::2, 1] - shift, xs[::2, 1])
        xh = xs.cpu().numpy()
        sdo = create_spline(loc, order, mesh, None).desc
        c_o = np.full((count, 4, 3), 7.0)
        skipped = oracle.apic_g2p(sdo, xh, u, c_o)
        sd = create_spline(loc, order, mesh, xs)
        err = torch.zeros(2, dtype=torch.int32, device="cuda")
        c_t = torch.full((count, 4, 3), 7.0, dtype=torch.float64, device="cuda")
        c_g = c_t.clone()
        c_s = torch.full((count, 13), 7.0, dtype=torch.float64, device="cuda")[:, 1:].unflatten(1, (4, 3))
        APIC.g2p(ud, c_t, sd, bins=bins, error_count=err[:1])
        APIC.g2p(ud, c_g, sd, error_count=err[1:])
        APIC.g2p(ud, c_s, sd, bins=bins)
        assert err.tolist() == [skipped, skipped]
        assert rel_err(c_t.cpu().numpy(), c_o) <= TOL
        assert rel_err(c_g.cpu().numpy(), c_o) <= TOL
        assert torch.equal(c_s, c_t)
        if not moved:
            assert torch.equal(c_t, c_g)
        # with advection: same values, then the position update
        x2, c2 = xs.clone(), torch.full_like(c_t, 7.0)
        APIC.g2p_advect(ud, c2, create_spline(loc, order, mesh, x2), 0.01, bins=bins)
        assert torch.equal(c2, c_t)
        x3, c3 = xs.clone(), torch.full_like(c_t, 7.0)
        APIC.g2p_advect(ud, c3, create_spline(loc, order, mesh, x3), 0.01)
        assert torch.equal(c3, c_g)
        if not moved:
            assert torch.equal(x2, x3)


@pytest.mark.parametrize("order", [1, 2, 3])
@pytest.mark.parametrize("ncomp", [1, 2, 3])
def test_components_and_strides(cuda, order, ncomp):
    """Fewer components, and velocity components that are not adjacent."""
    loc = FieldLocation.Node
    mesh, rng, x, _ = _setup((9, 7, 11), True, 700, order)
    ext = mesh.extent(loc)
    u = rng.standard_normal(ext + (ncomp,))
    c_o = np.zeros((700, 4, ncomp))
    assert oracle.apic_g2p(create_spline(loc, order, mesh, None).desc, x, u, c_o) == 0
    sd = create_spline(loc, order, mesh, torch.as_tensor(x, device="cuda"))
    apart = torch.zeros((ncomp,) + ext, dtype=torch.float64, device="cuda").permute(1, 2, 3, 0)
    apart.copy_(torch.as_tensor(u, device="cuda"))
    for grid in (torch.as_tensor(u, device="cuda"), apart):
        c = torch.zeros((700, 4, ncomp), dtype=torch.float64, device="cuda")
        APIC.g2p(grid, c, sd)
        assert rel_err(c.cpu().numpy(), c_o) <= TOL
