"""FP64 G2P from node tiles, which only large dense sets take (1.5 M particles): the same
bits as from global memory without bins, for sorted particles, for particles of which few
or many have left their tiles, and with advection."""

import pytest
import torch

from picasso_b200 import APIC, FieldLocation, UniformMesh, cell_sort, create_spline, permute_members

pytestmark = pytest.mark.gpu
LOC = FieldLocation.Node


@pytest.mark.parametrize("order,tile", [(1, (4, 8, 8)), (2, (4, 8, 8)), (2, (3, 5, 7)), (3, (4, 4, 8))])
@pytest.mark.parametrize("periodic", [True, False])
def test_tiles_repeat_global_memory(cuda, order, tile, periodic):
    cells = (47, 51, 50)
    mesh = UniformMesh([0, 0, 0] + [c / 64 for c in cells], cell_size=1 / 64,
                       periodic=(periodic,) * 3, halo_cell_width=0 if periodic else 2)
    g = torch.Generator(device="cuda").manual_seed(order)
    n = 1_530_007
    hi = torch.tensor(cells, dtype=torch.float64, device="cuda") / 64
    x = torch.rand((n, 3), generator=g, device="cuda", dtype=torch.float64) * hi
    x[:200] += 10.0 if not periodic else 0.0  # (out of the mesh, sorted last, counted)
    _, perm, bins = cell_sort(create_spline(LOC, order, mesh, x), tile, chunk=2048)
    x = permute_members(perm, x)[0]
    u = torch.randn(mesh.extent(LOC) + (3,), generator=g, device="cuda", dtype=torch.float64)
    for moved in (0, 50, n // 3):
        if moved:
            at = torch.randint(0, n - 200, (moved,), generator=g, device="cuda")
            x[at] = torch.rand((moved, 3), generator=g, device="cuda", dtype=torch.float64) * hi
        out = []
        for b in (bins, None):
            for advect in (False, True):
                xc = x.clone()
                sd = create_spline(LOC, order, mesh, xc)
                c = torch.full((n, 4, 3), 7.0, dtype=torch.float64, device="cuda")
                err = torch.zeros(1, dtype=torch.int32, device="cuda")
                if advect:
                    APIC.g2p_advect(u, c, sd, 1e-3, bins=b, error_count=err)
                else:
                    APIC.g2p(u, c, sd, bins=b, error_count=err)
                out.append((c, xc, int(err)))
        for plain, other in ((2, 0), (3, 1)):
            assert torch.equal(out[plain][0], out[other][0])
            assert torch.equal(out[plain][1], out[other][1])
            assert out[plain][2] == out[other][2]
        assert torch.equal(out[0][0], out[1][0])
