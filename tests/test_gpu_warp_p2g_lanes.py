"""FP64 APIC P2G of one or two momentum components where the lanes add a particle each:
particles in the order of their cells, some or many per cell, on faces, edges and node
fields, boxes whose stencils wrap around and closed ones with particles outside
(counted), strided members, counts around a warp's 32, against the oracle.

Tolerance 1e-12 of the largest value: sums of fewer than 2^11 terms of some 30 roundings
of 1.1e-16 each."""

import numpy as np
import pytest
import torch

import oracle
from particles import rel_err
from picasso_b200 import APIC, FieldLocation, UniformMesh, create_spline

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("where", ["face0", "face1", "face2", "edge1", "scalar", "pair"])
@pytest.mark.parametrize("order", [1, 2, 3])
def test_cell_order(cuda, order, where, periodic):
    loc = {"face0": FieldLocation.Face(0), "face1": FieldLocation.Face(1),
           "face2": FieldLocation.Face(2), "edge1": FieldLocation.Edge(1),
           "scalar": FieldLocation.Node, "pair": FieldLocation.Cell}[where]
    rng = np.random.default_rng(order)
    for cells, ppc in (((3, 5, 17), 1), ((4, 3, 40), 2), ((6, 7, 1), 3), ((2, 9, 11), 6), ((3, 2, 13), 20)):
        mesh = UniformMesh([0, 0, 0] + [c / 16 for c in cells], cell_size=1 / 16,
                           periodic=(periodic,) * 3, halo_cell_width=0 if periodic else 2)
        cell = np.arange(np.prod(cells)).repeat(ppc)
        x = np.stack([cell // (cells[1] * cells[2]), cell // cells[2] % cells[1], cell % cells[2]],
                     axis=1).astype(float)
        x = (x + rng.random(x.shape)) / 16
        n = x.shape[0]
        inside = np.ones(n, bool)
        if not periodic:
            inside[::9] = False
            x[~inside] += 10.0
        ncomp = {"scalar": 1, "pair": 2}.get(where, 3)
        m = rng.uniform(0.5, 1.5, n)
        c = rng.standard_normal((n, 4, ncomp))
        ext = mesh.extent(loc)
        dev = lambda a: torch.as_tensor(a, device="cuda")
        # members and grids strided
        xd = torch.zeros((n, 4), dtype=torch.float64, device="cuda")[:, 1:]
        xd.copy_(dev(x))
        gm = torch.zeros(ext + (2,), dtype=torch.float64, device="cuda")[..., 1]
        gmu = torch.zeros(ext + ((2,) if ncomp == 2 else ()), dtype=torch.float64, device="cuda")
        err = torch.zeros(1, dtype=torch.int32, device="cuda")
        APIC.p2g(dev(m), dev(c), gm, gmu, create_spline(loc, order, mesh, xd), error_count=err)
        gm_o, gmu_o = np.zeros(ext), np.zeros(ext + ((2,) if ncomp == 2 else ()))
        oracle.apic_p2g(create_spline(loc, order, mesh, None).desc, np.ascontiguousarray(x[inside]),
                        m[inside], np.ascontiguousarray(c[inside]), gm_o, gmu_o)
        assert int(err) == (~inside).sum()
        assert rel_err(gm.cpu().numpy(), gm_o) <= 1e-12
        assert rel_err(gmu.cpu().numpy(), gmu_o) <= 1e-12
