"""Quadratic FP32 P2G of sets large enough for their own ways through the tiles (streams over
thirds of an item from 3.5 M particles, runs from 5 M at 11 and more per cell) against the
FP64 P2G of the same particles.

Tolerance: masses and velocities are positive and the affine part is zero, so that no sum
cancels.  A contribution is a product of some 8 roundings (6e-8 each), a chain in registers
at most 128 particles, and a node's value leaves through at most 64 more additions:
200 * 6e-8 = 1.2e-5 of the largest value."""

import pytest
import torch

from picasso_b200 import APIC, FieldLocation, FixedGrid, UniformMesh, cell_sort, create_spline, permute_members

pytestmark = pytest.mark.gpu
LOC = FieldLocation.Node


@pytest.mark.parametrize("cells,ppc", [((97, 90, 103), 4), ((81, 80, 85), 10), ((76, 77, 80), 11)])
def test_against_fp64(cuda, cells, ppc):
    mesh = UniformMesh([0, 0, 0] + [c / 64 for c in cells], cell_size=1 / 64, periodic=(True,) * 3)
    n = ppc * cells[0] * cells[1] * cells[2]
    g = torch.Generator(device="cuda").manual_seed(ppc)
    x = torch.rand((n, 3), generator=g, device="cuda", dtype=torch.float64)
    x[: n // 4] = x[: n // 4] ** 3  # a quarter of them crowded into a corner
    x *= torch.tensor(cells, dtype=torch.float64, device="cuda") / 64
    _, perm, bins = cell_sort(create_spline(LOC, 2, mesh, x), (4, 8, 8), chunk=4096)
    x = permute_members(perm, x)[0]
    m = torch.rand(n, generator=g, device="cuda") + 0.5
    c = torch.zeros((n, 4, 3), device="cuda")
    c[:, 0] = torch.rand((n, 3), generator=g, device="cuda") + 0.5
    sd = create_spline(LOC, 2, mesh, x)
    ext = mesh.extent(LOC)
    ref = torch.zeros(ext + (4,), dtype=torch.float64, device="cuda")
    APIC.p2g(m.double(), c.double(), ref[..., 0], ref[..., 1:], sd)
    acc = torch.zeros(ext + (4,), dtype=torch.int64, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    APIC.p2g(m, c, FixedGrid(acc[..., 0], 36), FixedGrid(acc[..., 1:], 36), sd, bins=bins,
             error_count=err)
    assert int(err) == 0
    off = (acc.double() * 2.0 ** -36 - ref).abs().amax(dim=(0, 1, 2)) / ref.amax(dim=(0, 1, 2))
    assert off.max() <= 1.2e-5
