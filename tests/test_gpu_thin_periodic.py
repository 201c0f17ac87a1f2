"""FP32 transfers with bins on periodic boxes so thin that a tile with its halo spans
several periods: P2G (separate grids, a packed accumulator whose rows leave by bulk
reductions, from positions and records) and G2P against the oracle, every grid between
guard values that must stay, and PolyPIC G2P against the call without bins."""

import numpy as np
import pytest
import torch

import oracle
from particles import rel_err
from picasso_b200 import (APIC, FieldLocation, FixedGrid, PolyPIC, UniformMesh, cell_sort,
                          create_spline, permute_members, spline_records)

pytestmark = pytest.mark.gpu
LOC = FieldLocation.Node


def _guarded(shape, dtype):
    """(grid, its storage with guards of 20 nodes' rows on both sides)."""
    n, guard = int(np.prod(shape)), 1024
    store = torch.full((n + 2 * guard,), 77, dtype=dtype, device="cuda")
    grid = store[guard:guard + n].view(shape)
    grid.zero_()
    return grid, store


def _intact(store):
    return bool((store[:1024] == 77).all()) and bool((store[-1024:] == 77).all())


@pytest.mark.parametrize("halo", [0, 1])
@pytest.mark.parametrize("cells", [(2, 3, 1), (7, 5, 4), (5, 1, 2), (12, 6, 3)])
@pytest.mark.parametrize("order", [1, 2, 3])
def test_apic(cuda, order, cells, halo):
    mesh = UniformMesh([0, 0, 0] + [c / 8 for c in cells], cell_size=1 / 8, periodic=(True,) * 3,
                       halo_cell_width=halo)
    rng = np.random.default_rng(order)
    # from 4 per cell on quadratic sets are summed in another way
    for n in (3 * int(np.prod(cells)), 10 * int(np.prod(cells))):
        x = torch.as_tensor(rng.random((n, 3)) * np.array(cells) / 8, device="cuda")
        m = torch.as_tensor(rng.uniform(0.5, 1.5, n), dtype=torch.float32, device="cuda")
        c = torch.as_tensor(rng.standard_normal((n, 4, 3)), dtype=torch.float32, device="cuda")
        c[:, 1:] *= 0.1
        _, perm, bins = cell_sort(create_spline(LOC, order, mesh, x), chunk=64)
        x, m, c = permute_members(perm, x, m, c)
        sd = create_spline(LOC, order, mesh, x)
        ext = mesh.extent(LOC)
        sdo = create_spline(LOC, order, mesh, None).desc
        xh, mh, ch = x.cpu().numpy(), m.double().cpu().numpy(), c.double().cpu().numpy()
        gm_o, gmu_o = np.zeros(ext), np.zeros(ext + (3,))
        oracle.apic_p2g(sdo, xh, mh, ch, gm_o, gmu_o)
        err = torch.zeros(1, dtype=torch.int32, device="cuda")
        sums = []
        for records in (False, True):
            if records:
                spline_records(sd, bins)
            for packed in (True, False):
                acc, store = _guarded(ext + (4,), torch.int64)
                gm, gmu = FixedGrid(acc[..., 0], 36), FixedGrid(acc[..., 1:], 36)
                if not packed:
                    gm = FixedGrid(torch.zeros(ext, dtype=torch.int64, device="cuda"), 36)
                APIC.p2g(m, c, gm, gmu, sd, bins=bins, error_count=err)
                assert _intact(store)
                # a node sums at most 27 contributions per particle; their rounding
                # errors, 10 of 6e-8 each, add like a random walk, and the sums are
                # up to 10 times smaller than their terms
                assert rel_err(gm.to_float().cpu().numpy(), gm_o) <= 2e-5
                assert rel_err(gmu.to_float().cpu().numpy(), gmu_o) <= 5e-5
                sums.append(torch.cat([gm.raw.flatten(), gmu.raw.flatten()]))
        assert all(torch.equal(s, sums[0]) for s in sums)
        u, store = _guarded(ext + (3,), torch.float32)
        store[:1024] = store[-1024:] = float("nan")  # must not be read either
        u.copy_(torch.as_tensor(rng.standard_normal(ext + (3,))))
        out_o = np.zeros((n, 4, 3))
        oracle.apic_g2p(sdo, xh, u.double().cpu().numpy(), out_o)
        for b in (bins, cell_sort(sd, chunk=64)[2]):  # records, positions
            out = torch.full_like(c, 7.0)
            APIC.g2p(u, out, sd, bins=b, error_count=err)
            assert rel_err(out.cpu().numpy(), out_o) <= 5e-6  # 64 terms of 10 roundings
        assert int(err) == 0


@pytest.mark.parametrize("cells", [(2, 3, 1), (7, 5, 4)])
@pytest.mark.parametrize("order", [1, 2])
def test_polypic_g2p(cuda, order, cells):
    mesh = UniformMesh([0, 0, 0] + [c / 8 for c in cells], cell_size=1 / 8, periodic=(True,) * 3)
    rng = np.random.default_rng(order)
    n, modes = 100, 8 if order == 1 else 27
    x = torch.as_tensor(rng.random((n, 3)) * np.array(cells) / 8, device="cuda")
    _, perm, bins = cell_sort(create_spline(LOC, order, mesh, x), chunk=64)
    x = permute_members(perm, x)[0]
    sd = create_spline(LOC, order, mesh, x)
    u = torch.as_tensor(rng.standard_normal(mesh.extent(LOC) + (3,)), dtype=torch.float32,
                        device="cuda")
    got, want = (torch.zeros((n, modes, 3), dtype=torch.float32, device="cuda") for _ in range(2))
    PolyPIC.g2p(u, got, sd, bins=bins)
    PolyPIC.g2p(u, want, sd)
    # the same contraction of the same values as without bins (which the oracle checks
    # elsewhere; here whole modes vanish, those along a dimension of one cell)
    assert torch.equal(got, want)
