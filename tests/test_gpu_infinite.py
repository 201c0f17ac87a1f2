"""FP64 APIC transfers of infinite coefficients, masses and node velocities: the nodes and
the particles that the node by node definition leaves finite, infinite (with their sign) or
NaN are so here, and the finite ones are its values.

Tolerance 1e-12 of the largest finite value: a contribution is a product of some 20
roundings (each 1.1e-16) and a value sums at most a few hundred contributions whose
magnitudes add up to less than 100 times the largest."""

import numpy as np
import pytest
import torch

import oracle
from picasso_b200 import APIC, FieldLocation, UniformMesh, cell_sort, create_spline, permute_members

pytestmark = pytest.mark.gpu
TOL = 1e-12
CELLS = (13, 9, 12)


def _mesh(periodic=True):
    h = 1.0 / 13
    return UniformMesh([0, 0, 0] + [h * n for n in CELLS], cell_size=h, periodic=(periodic,) * 3,
                       halo_cell_width=2)


def _same(got, want):
    fin = np.isfinite(want)
    assert fin.any() and not fin.all()
    assert np.array_equal(np.isfinite(got), fin)
    assert np.array_equal(got[~fin], want[~fin], equal_nan=True)
    assert np.abs(got[fin] - want[fin]).max() <= TOL * np.abs(want[fin]).max()


@pytest.mark.parametrize("order", [1, 2, 3])
@pytest.mark.parametrize("loc,ncomp", [(FieldLocation.Node, 3), (FieldLocation.Cell, 2),
                                       (FieldLocation.Face(1), 3)])
@pytest.mark.parametrize("crowded", [False, True])
@pytest.mark.parametrize("periodic", [True, False])
def test_p2g(cuda, order, loc, ncomp, crowded, periodic):
    stag = loc == FieldLocation.Face(1)
    mesh = _mesh(periodic)
    rng = np.random.default_rng(order)
    n = 400
    x = rng.random((n, 3)) * np.array(CELLS) * mesh.cell_size
    if crowded:  # every stencil in runs of four and more
        x = np.repeat(x[::8], 8, axis=0) + 1e-9 * rng.random((n, 3))
    m, c = rng.uniform(0.5, 1.5, n), rng.standard_normal((n, 4, ncomp))
    for p, (q, d, s) in {3: (0, 0, 1), 40: (1, 1, -1), 101: (2, 1, 1), 202: (3, 0, -1)}.items():
        c[p, q, d] = s * np.inf
    m[333] = np.inf
    if not periodic:  # some of them, and others, out of the mesh
        x[[40, 41, 300]] += [7.0, -9.0, 0.0]
    ext = mesh.extent(loc)
    sdo = create_spline(loc, order, mesh, None).desc
    gm_o, gmu_o = np.zeros(ext), np.zeros(ext if stag else ext + (ncomp,))
    with np.errstate(all="ignore"):
        skipped = oracle.apic_p2g(sdo, x, m, c, gm_o, gmu_o)
    dev = [torch.as_tensor(a, device="cuda") for a in (x, m, c)]
    gm, gmu = mesh.zeros(loc), mesh.zeros(loc, 1 if stag else ncomp)
    if stag:
        gmu = gmu[..., 0]
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    APIC.p2g(dev[1], dev[2], gm, gmu, create_spline(loc, order, mesh, dev[0]), error_count=err)
    assert int(err) == skipped == (0 if periodic else 3)
    _same(gm.cpu().numpy(), gm_o)
    _same(gmu.cpu().numpy(), gmu_o)


@pytest.mark.parametrize("order", [1, 2, 3])
@pytest.mark.parametrize("loc,ncomp", [(FieldLocation.Node, 3), (FieldLocation.Cell, 2),
                                       (FieldLocation.Face(1), 3)])
def test_g2p(cuda, order, loc, ncomp):
    stag = loc == FieldLocation.Face(1)
    mesh = _mesh()
    rng = np.random.default_rng(10 + order)
    n = 1200
    x = rng.random((n, 3)) * np.array(CELLS) * mesh.cell_size
    u = rng.standard_normal(mesh.extent(loc) + (() if stag else (ncomp,)))
    for i, s in (((3, 4, 5), 1), ((9, 2, 7), -1), ((9, 4, 8), 1)):
        u[i] = s * np.inf if stag else [s * np.inf] + [0.5] * (ncomp - 1)
    sdo = create_spline(loc, order, mesh, None).desc
    c_o = np.zeros((n, 4, ncomp))
    with np.errstate(all="ignore"):
        oracle.apic_g2p(sdo, x, u, c_o)
    c = torch.zeros((n, 4, ncomp), dtype=torch.float64, device="cuda")
    APIC.g2p(torch.as_tensor(u, device="cuda"), c,
             create_spline(loc, order, mesh, torch.as_tensor(x, device="cuda")))
    _same(c.cpu().numpy(), c_o)


def test_g2p_from_tiles(cuda):
    """A set large and dense enough for node tiles, some particles out of theirs."""
    mesh = UniformMesh([0, 0, 0, 1, 1, 1], cell_size=1 / 48, periodic=(True,) * 3,
                       halo_cell_width=0)
    g = torch.Generator(device="cuda").manual_seed(4)
    loc, n = FieldLocation.Node, 1_600_000
    x = torch.rand((n, 3), generator=g, device="cuda", dtype=torch.float64)
    _, perm, bins = cell_sort(create_spline(loc, 2, mesh, x), (4, 8, 8), chunk=2048)
    x = permute_members(perm, x)[0]
    x[::1000] = torch.rand((n // 1000, 3), generator=g, device="cuda", dtype=torch.float64)
    u = torch.randn(mesh.extent(loc) + (3,), generator=g, device="cuda", dtype=torch.float64)
    u[::7, 5, ::9, 1] = float("inf")
    out = []
    for b in (bins, None):
        c = torch.zeros((n, 4, 3), dtype=torch.float64, device="cuda")
        APIC.g2p(u, c, create_spline(loc, 2, mesh, x), bins=b)
        out.append(c)
    assert out[1].isinf().any() and not out[1].isnan().any()
    assert torch.equal(out[0], out[1])
