"""The kernels of the fixed-point PolyPIC P2G -- one thread per particle without bins;
with them streams, or for sparse FP32 sets an integer tile -- fill the grid with the same
bits, and bins beyond the tile's limits (work items over 65536 particles, a tile that
does not fit in shared memory) only tell the particles' order: a particle that has left
its tile is added, not counted."""

import pytest
import torch

from picasso_b200 import (FieldLocation, FixedGrid, PolyPIC, UniformMesh, cell_sort, create_spline,
                          permute_members)

pytestmark = pytest.mark.gpu
LOC = FieldLocation.Node


def _sorted(order, dtype, cells, n, ncomp, tile, chunk, clustered=False):
    h = 1 / 32
    mesh = UniformMesh([0, 0, 0] + [c * h for c in cells], cell_size=h, periodic=(True,) * 3)
    g = torch.Generator(device="cuda").manual_seed(n)
    hi = torch.tensor([c * h for c in cells], device="cuda", dtype=torch.float64)
    x = torch.rand((n, 3), generator=g, device="cuda", dtype=torch.float64)
    if clustered:
        x[: n // 2] *= 0.2
    x *= hi
    modes = 8 if order == 1 else 27
    m = (torch.rand(n, generator=g, device="cuda") + 0.5).to(dtype)
    u = (0.1 * torch.randn((n, modes, 3), generator=g, device="cuda")).to(dtype)
    _, perm, bins = cell_sort(create_spline(LOC, order, mesh, x), tile, chunk=chunk)
    x, m, u = permute_members(perm, x, m, u)
    return mesh, x, m, u, u[..., :ncomp].contiguous(), bins


def _p2g(mesh, order, x, m, u, c, bins):
    ext = mesh.extent(LOC)
    acc = torch.zeros(ext + (1 + c.shape[2],), dtype=torch.int64, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    PolyPIC.p2g(m, u, c, FixedGrid(acc[..., 1:], 36), FixedGrid(acc[..., 0], 36), 0.01,
                create_spline(LOC, order, mesh, x), bins=bins, error_count=err)
    return acc, int(err)


# particles per cell below and above 1.5, and a quadratic FP32 set of over 500 000
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64], ids=["fp32", "fixed64"])
@pytest.mark.parametrize("order,cells,n,ncomp", [
    (1, (13, 9, 11), 1300, 3), (1, (13, 9, 11), 1931, 2), (1, (13, 9, 11), 2400, 1),
    (1, (40, 41, 39), 77001, 3), (2, (13, 9, 11), 1300, 3), (2, (13, 9, 11), 2400, 2),
    (2, (40, 41, 39), 77001, 1), (2, (80, 75, 70), 500001, 3)])
def test_kernels_agree_in_every_bit(cuda, order, cells, n, ncomp, dtype):
    for tile, clustered in (((4, 8, 8), False), ((3, 5, 4), True)):
        *set_, bins = _sorted(order, dtype, cells, n, ncomp, tile, 1024, clustered)
        mesh, x, m, u, c = set_
        sorted_, err = _p2g(mesh, order, x, m, u, c, bins)
        plain, err0 = _p2g(mesh, order, x, m, u, c, None)
        assert err == err0 == 0
        assert torch.equal(sorted_, plain)


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("density", [1, 4])
@pytest.mark.parametrize("tile,chunk,counts", [((4, 8, 8), 65536, True), ((4, 8, 8), 65537, False),
                                               ((16, 16, 16), 1024, False)])
def test_particles_out_of_their_tile(cuda, order, density, tile, chunk, counts):
    cells = (24, 20, 17)
    mesh, x, m, u, c, bins = _sorted(order, torch.float32, cells, density * 24 * 20 * 17, 3, tile, chunk)
    x[::5, 0] = torch.remainder(x[::5, 0] + 12.2 / 32, 24 / 32)  # half the box away
    got, err = _p2g(mesh, order, x, m, u, c, bins)
    if counts:
        stays = torch.ones(x.shape[0], dtype=torch.bool, device="cuda")
        stays[::5] = False
        want, _ = _p2g(mesh, order, x[stays], m[stays], u[stays], c[stays], None)
        assert err == int((~stays).sum())
    else:
        want, _ = _p2g(mesh, order, x, m, u, c, None)
        assert err == 0
    assert torch.equal(got, want)
