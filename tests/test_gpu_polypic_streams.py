"""PolyPIC P2G at the edges of its particle streams: particle counts around a
warp's tables and segments, runs of one stencil and none, the number of components,
staggered locations, strided records, stencils wider than a periodic mesh, particles
outside a closed one and particles that have left the tile of their sort (both
counted), against the oracle; the integer grid has to be the same in any order of
the particles."""

import numpy as np
import pytest
import torch

import oracle
from particles import rel_err
from picasso_b200 import (FieldLocation, FixedGrid, PolyPIC, UniformMesh, cell_sort, create_spline,
                          permute_members)

pytestmark = pytest.mark.gpu
DT = 0.01


def _mesh(kind):
    cells = {"periodic": (7, 5, 9), "thin": (2, 5, 1), "closed": (6, 8, 5)}[kind]
    hi = [c / 8 for c in cells]
    return UniformMesh([0, 0, 0] + hi, cell_size=1 / 8, periodic=(kind != "closed",) * 3,
                       halo_cell_width=2 if kind == "closed" else 0), np.array(hi)


def _p2g(mesh, loc, order, form, x, m, u, c, strided, bins=None):
    """Grid (mass, momentum) in FP64 and the count of skipped particles."""
    dtype = torch.float32 if form == "fp32" else torch.float64
    dev = lambda a, t: torch.as_tensor(np.ascontiguousarray(a), dtype=t, device="cuda")
    xd, md, ud, cd = dev(x, torch.float64), dev(m, dtype), dev(u, dtype), dev(c, dtype)
    if strided:
        wide = torch.zeros((c.shape[0], c.shape[1] + 1, c.shape[2]), dtype=dtype, device="cuda")
        wide[:, 1:] = cd
        cd = wide[:, 1:]
    ext = mesh.extent(loc)
    nc = c.shape[2]
    ncg = () if loc != FieldLocation.Node else (nc,)
    if form == "fp64":
        gm = torch.zeros(ext, dtype=torch.float64, device="cuda")
        gmu = torch.zeros(ext + ncg, dtype=torch.float64, device="cuda")
    else:
        gm = FixedGrid(torch.zeros(ext, dtype=torch.int64, device="cuda"), 36)
        gmu = FixedGrid(torch.zeros(ext + ncg, dtype=torch.int64, device="cuda"), 36)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    sd = create_spline(loc, order, mesh, xd)
    PolyPIC.p2g(md, ud, cd, gmu, gm, DT, sd, bins=bins, error_count=err)
    return gm, gmu, int(err.item())


# (order, components, mesh, location, particles, records)
CASES = [
    (1, 3, "periodic", "node", 1, "packed"),
    (1, 3, "periodic", "node", 33, "packed"),     # one table and one particle
    (1, 2, "thin", "node", 255, "packed"),
    (1, 1, "closed", "node", 1029, "strided"),
    (1, 3, "closed", "face", 517, "packed"),
    (2, 3, "periodic", "node", 2, "packed"),      # fewer than the streams
    (2, 3, "closed", "node", 31, "packed"),       # a table and one particle
    (2, 3, "thin", "node", 4001, "strided"),
    (2, 2, "periodic", "node", 603, "packed"),
    (2, 1, "closed", "node", 19, "packed"),
]


@pytest.mark.parametrize("form", ["fp64", "fp32", "fixed64"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(map(str, c)))
def test_streams(cuda, case, form):
    order, nc, kind, where, n, records = case
    mesh, hi = _mesh(kind)
    loc = FieldLocation.Node if where == "node" else FieldLocation.Face(1)
    rng = np.random.default_rng(n)
    x = rng.random((n, 3)) * hi
    x[: n // 3] = x[0]  # one stencil ...
    x = x[np.lexsort(np.floor(x * 8).T[::-1])]  # ... and cells in order
    if kind == "closed":
        x[::7] += 10.0
    nm = 8 if order == 1 else 27
    m = rng.uniform(0.5, 1.5, n).astype(np.float32).astype(np.float64)
    u = rng.standard_normal((n, nm, 3))  # rows 1..3: the affine velocity
    u[:, 1:] *= 0.05
    u = u.astype(np.float32).astype(np.float64)
    c = np.ascontiguousarray(u[..., :nc])
    gm, gmu, err = _p2g(mesh, loc, order, form, x, m, u, c, records == "strided")
    sd = create_spline(loc, order, mesh, None).desc
    ext = mesh.extent(loc)
    gm_o = np.zeros(ext)
    gmu_o = np.zeros(ext + ((nc,) if where == "node" else ()))
    inside = np.ones(n, bool) if kind != "closed" else np.arange(n) % 7 != 0
    oracle.polypic_p2g(sd, x[inside], m[inside], u[inside], c[inside], gmu_o, gm_o, DT)
    assert err == int((~inside).sum())
    # FP64: rounding of sums of < 2^13 terms, each of some 100 operations; FP32:
    # the same per particle in 2^-24, cancelling sums up to 8 terms' weight; both
    # with the 2^-37 of a fixed-point term
    tol = 1e-12 if form == "fp64" else 1e-9 if form == "fixed64" else 2e-5
    if form != "fp64":
        perm = rng.permutation(n)
        gm2, gmu2, _ = _p2g(mesh, loc, order, form, x[perm], m[perm], u[perm], c[perm], False)
        assert torch.equal(gm.raw, gm2.raw) and torch.equal(gmu.raw, gmu2.raw)
        gm, gmu = gm.to_float(), gmu.to_float()
    if inside.any():
        assert rel_err(gm.cpu().numpy(), gm_o) <= tol
        assert rel_err(gmu.cpu().numpy(), gmu_o) <= tol


@pytest.mark.parametrize("order,tile", [(1, (4, 4, 8)), (2, (3, 5, 4))])
def test_particles_out_of_their_tile_are_counted(cuda, order, tile):
    """FP32 form with bins: as if the particles that moved into another tile
    since the sort (and only those) were not there."""
    mesh, hi = _mesh("periodic")
    rng = np.random.default_rng(order)
    n, nm = 700, 8 if order == 1 else 27
    x = torch.as_tensor(rng.random((n, 3)) * hi, device="cuda")
    m = rng.uniform(0.5, 1.5, n)
    u = rng.standard_normal((n, nm, 3)) * 0.1
    loc = FieldLocation.Node
    _, perm, bins = cell_sort(create_spline(loc, order, mesh, x), tile, chunk=64)
    xs = permute_members(perm, x)[0].cpu().numpy()
    first = 0 if order == 1 else -1

    def tiles(at):  # the tile of a particle: of its stencil's first node
        s = np.floor(at * 8 + (0.0 if order == 1 else 0.5)).astype(int) + first
        return np.mod(s, (7, 5, 9)) // np.array(tile)

    was = tiles(xs)
    xs[::5, 2] = np.mod(xs[::5, 2] + 4.5 / 8, hi[2])
    stays = (tiles(xs) == was).all(axis=1)
    assert 0 < (~stays).sum() < n
    gm, gmu, err = _p2g(mesh, loc, order, "fp32", xs, m, u, u, False, bins)
    gm2, gmu2, _ = _p2g(mesh, loc, order, "fp32", xs[stays], m[stays], u[stays], u[stays], False)
    assert err == int((~stays).sum())
    assert torch.equal(gm.raw, gm2.raw) and torch.equal(gmu.raw, gmu2.raw)


@pytest.mark.parametrize("case", [c for c in CASES if c[5] == "packed"], ids=lambda c: "-".join(map(str, c)))
def test_fp64_streams_of_sorted_particles(cuda, case):
    """FP64 grids take the streams when the call has bins (linear splines: from 2
    particles per stencil on, here by repeating them); the tolerance of test_streams."""
    order, nc, kind, where, n, _ = case
    mesh, hi = _mesh(kind)
    loc = FieldLocation.Node if where == "node" else FieldLocation.Face(1)
    rng = np.random.default_rng(n)
    n = n if order == 2 else n + 2 * int(np.prod(mesh.extent(loc)))
    x = torch.as_tensor(rng.random((n, 3)) * hi, device="cuda")
    _, perm, bins = cell_sort(create_spline(loc, order, mesh, x), (4, 4, 8), chunk=64)
    x = permute_members(perm, x)[0].cpu().numpy()
    nm = 8 if order == 1 else 27
    m = rng.uniform(0.5, 1.5, n)
    u = rng.standard_normal((n, nm, 3))
    u[:, 1:] *= 0.05
    c = np.ascontiguousarray(u[..., :nc])
    gm, gmu, err = _p2g(mesh, loc, order, "fp64", x, m, u, c, False, bins)
    ext = mesh.extent(loc)
    gm_o, gmu_o = np.zeros(ext), np.zeros(ext + ((nc,) if where == "node" else ()))
    oracle.polypic_p2g(create_spline(loc, order, mesh, None).desc, x, m, u, c, gmu_o, gm_o, DT)
    assert err == 0
    assert rel_err(gm.cpu().numpy(), gm_o) <= 1e-12
    assert rel_err(gmu.cpu().numpy(), gmu_o) <= 1e-12
