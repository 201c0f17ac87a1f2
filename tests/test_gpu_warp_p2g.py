"""FP64 APIC P2G by warps against the oracle where its runs, batches and wraps
can go wrong: sorted particles (long runs, moves along k), shuffled ones (put
in order inside a warp) and isolated ones (straight to the grid), particle
counts around a warp and a segment, periodic meshes smaller than a stencil,
particles outside a closed mesh, every component count, packed and separate
grid arrays.

Tolerance 1e-12 of the largest value: a contribution is a product of some 20
roundings (each 1.1e-16) and a node sums at most a few hundred contributions
whose magnitudes add up to less than 100 times the largest node value."""

import numpy as np
import pytest
import torch

import oracle
from particles import rel_err
from picasso_b200 import APIC, FieldLocation, UniformMesh, create_spline
from picasso_b200.api import staggered_dim

pytestmark = pytest.mark.gpu
TOL = 1e-12


def _mesh(cells, periodic):
    h = 1.0 / max(cells)
    return UniformMesh([0, 0, 0] + [h * n for n in cells], cell_size=h, periodic=(periodic,) * 3,
                       halo_cell_width=1 if periodic else 2)


def _particles(mesh, cells, count, place, ncomp, seed):
    rng = np.random.default_rng(seed)
    size = np.array(cells) * mesh.cell_size
    x = rng.random((count, 3)) * size
    if place == "sorted":
        q = np.floor(x / mesh.cell_size + 0.5).astype(int)
        x = x[np.lexsort((q[:, 2], q[:, 1], q[:, 0]))]
    elif place == "cells":  # a few crowded cells, random order
        x = (rng.integers(0, 2, (count, 3)) + rng.random((count, 3))) * mesh.cell_size
    c = rng.standard_normal((count, 4, ncomp))
    return x, rng.uniform(0.5, 1.5, count), c


CASES = [((12, 9, 17), True), ((2, 3, 1), True), ((7, 10, 6), False)]


@pytest.mark.parametrize("cells,periodic", CASES)
@pytest.mark.parametrize("place", ["sorted", "random", "cells"])
@pytest.mark.parametrize("order", [1, 2, 3])
@pytest.mark.parametrize("loc,ncomp", [(FieldLocation.Node, 1), (FieldLocation.Cell, 2),
                                       (FieldLocation.Node, 3), (FieldLocation.Face(2), 3),
                                       (FieldLocation.Edge(1), 3)])
def test_against_oracle(cuda, order, loc, ncomp, place, cells, periodic):
    stag = staggered_dim(loc) >= 0
    mesh = _mesh(cells, periodic)
    ext = mesh.extent(loc)
    nv = 1 if stag else ncomp
    for count in (1, 8, 31, 33, 257, 1500):
        x, m, c = _particles(mesh, cells, count, place, ncomp, 100 * order + count)
        if not periodic and count > 8:
            x[::7] -= 100.0 * mesh.cell_size  # outside: skipped and counted
        sdo = create_spline(loc, order, mesh, None).desc
        gm_o = np.zeros(ext)
        gmu_o = np.zeros(ext) if stag else np.zeros(ext + (ncomp,))
        skipped = oracle.apic_p2g(sdo, x, m, c, gm_o, gmu_o)
        sd = create_spline(loc, order, mesh, torch.as_tensor(x, device="cuda"))
        packed = count % 2 == 1
        acc = torch.zeros(ext + (1 + nv,), dtype=torch.float64, device="cuda")
        gm = acc[..., 0] if packed else mesh.zeros(loc)
        gmu = acc[..., 1:] if packed else mesh.zeros(loc, nv)
        if stag:
            gmu = gmu[..., 0]
        err = torch.zeros(1, dtype=torch.int32, device="cuda")
        # one set reads c_p through general strides
        cd = torch.as_tensor(c, device="cuda")
        if count == 33:
            wide = torch.zeros((count, 4 * ncomp + 1), dtype=torch.float64, device="cuda")
            wide[:, 1:] = cd.reshape(count, -1)
            cd = wide[:, 1:].unflatten(1, (4, ncomp))
        APIC.p2g(torch.as_tensor(m, device="cuda"), cd, gm, gmu, sd, error_count=err)
        assert int(err) == skipped
        assert rel_err(gm.cpu().numpy(), gm_o) <= TOL
        assert rel_err(gmu.cpu().numpy(), gmu_o.reshape(tuple(gmu.shape))) <= TOL


@pytest.mark.parametrize("order", [2, 3])
def test_nonfinite_stays_with_its_particle(cuda, order):
    """A particle with a NaN coefficient spoils its own nodes' momentum only:
    not its mass, not the nodes of the particles it is summed next to."""
    mesh = _mesh((16, 16, 16), True)
    loc = FieldLocation.Node
    h = mesh.cell_size
    # two crowded stencils far apart, four particles of each in turn
    x = np.concatenate([np.full((7, 3), 3.2 * h), np.full((6, 3), 11.3 * h)])
    c = np.ones((13, 4, 3))
    c[7, 2, 1] = np.nan
    sd = create_spline(loc, order, mesh, torch.as_tensor(x, device="cuda"))
    gm, gmu = mesh.zeros(loc), mesh.zeros(loc, 3)
    APIC.p2g(torch.ones(13, dtype=torch.float64, device="cuda"), torch.as_tensor(c, device="cuda"),
             gm, gmu, sd)
    gm, gmu = gm.cpu().numpy(), gmu.cpu().numpy()
    assert np.isfinite(gm).all()
    assert np.isfinite(gmu[..., [0, 2]]).all()
    bad = ~np.isfinite(gmu[..., 1])
    lo, n = mesh.halo_cell_width, order + 1
    first = 10 + lo  # floor(11.3) - 1, and floor(11.8) - 1
    assert bad.sum() == n ** 3 and bad[first:first + n, first:first + n, first:first + n].all()
