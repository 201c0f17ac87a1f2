"""Tiles around the limits of shared memory, against the same calls without bins or
the oracle: FP64 G2P tiles on both sides of 48 KB, FP64 batches whose tile does not
fit (they gather from global memory) beside ones whose tile does, and FP32 P2G tiles
that only fit without the padding of their rows."""

import numpy as np
import pytest
import torch

import oracle
from particles import periodic_mesh, rel_err, uniform_particles
from picasso_b200 import (APIC, Batch, BatchInstance, FieldLocation, FixedGrid, UniformMesh,
                          cell_sort, create_spline, permute_members)

pytestmark = pytest.mark.gpu
LOC = FieldLocation.Node


def _sorted(mesh, order, tile, dtype, seed, ppc=1):
    x, m, c = uniform_particles(mesh, ppc, seed=seed)
    dev = [torch.as_tensor(x, device="cuda"), torch.as_tensor(m, dtype=dtype, device="cuda"),
           torch.as_tensor(c, dtype=dtype, device="cuda").contiguous()]
    _, perm, bins = cell_sort(create_spline(LOC, order, mesh, dev[0]), tile, chunk=512)
    x, m, c = permute_members(perm, *dev)
    return create_spline(LOC, order, mesh, x), m, c, bins


# quadratic: (T + 2)^3 nodes of 24 bytes, next to 13 KB (with advection 15 KB)
@pytest.mark.parametrize("tile", [(8, 8, 11), (8, 8, 12), (8, 8, 13), (8, 8, 15), (8, 8, 18)])
def test_fp64_g2p_tiles_around_48_kb(cuda, tile):
    mesh = periodic_mesh(18)
    sd, _, c, bins = _sorted(mesh, 2, tile, torch.float64, 3)
    u = torch.as_tensor(np.random.default_rng(4).standard_normal(mesh.extent(LOC) + (3,)),
                        device="cuda")
    got, want = torch.zeros_like(c), torch.zeros_like(c)
    APIC.g2p(u, got, sd, bins=bins)
    APIC.g2p(u, want, sd)
    # the same contraction of the same values, from the tile or not
    assert torch.equal(got, want)
    x0 = sd.x.clone()
    APIC.g2p_advect(u, got, sd, 1e-3, bins=bins)
    assert torch.equal(got, want) and not torch.equal(sd.x, x0)


@pytest.mark.parametrize("mode", ["fused", "phased"])
def test_fp64_batch_with_a_tile_that_does_not_fit(cuda, mode):
    mesh = periodic_mesh(24)
    made, instances = [], []
    for order, tile in [(1, (24, 24, 24)), (2, (24, 24, 24)), (3, (24, 24, 24)), (2, (4, 8, 8))]:
        sd, m, c, bins = _sorted(mesh, order, tile, torch.float64, order)
        ext = mesh.extent(LOC)
        acc = torch.zeros(ext + (4,), dtype=torch.float64, device="cuda")
        u = torch.zeros(ext + (3,), dtype=torch.float64, device="cuda")
        made.append((order, sd.x.cpu().numpy(), m.cpu().numpy(), c.cpu().numpy(), u, c))
        instances.append(BatchInstance(sd, m, c, acc[..., 0], acc[..., 1:], u, bins, 1e-12))
    Batch(instances, mode=mode).step(graph=False)
    torch.cuda.synchronize()
    for order, x, m, c, u, c_out in made:
        sd = create_spline(LOC, order, mesh, None).desc
        ext = mesh.extent(LOC)
        gm, gmu, gu = np.zeros(ext), np.zeros(ext + (3,)), np.zeros(ext + (3,))
        oracle.apic_p2g(sd, x, m, c, gm, gmu)
        oracle.grid_velocity(mesh.descriptor(LOC), gm, gmu, gu)
        want = np.zeros_like(c)
        oracle.apic_g2p(sd, x, gu, want)
        assert rel_err(u.cpu().numpy(), gu) <= 1e-12
        assert rel_err(c_out.cpu().numpy(), want) <= 1e-12


# nodes x 16 bytes with 4 KB fit in 227 KB, not so with rows padded against bank
# conflicts
@pytest.mark.parametrize("order,tile", [(2, (120, 24, 2)), (2, (92, 13, 8)), (1, (63, 25, 7)),
                                        (3, (120, 6, 9))])
def test_fp32_p2g_tiles_that_fit_unpadded(cuda, order, tile):
    mesh = UniformMesh([0, 0, 0, 120 / 32, 1, 15 / 32], cell_size=1 / 32, periodic=(True,) * 3)
    sd, m, c, bins = _sorted(mesh, order, tile, torch.float32, 5)

    def grid(b):
        ext = mesh.extent(LOC)
        acc = torch.zeros(ext + (4,), dtype=torch.int64, device="cuda")
        gm, gmu = FixedGrid(acc[..., 0], 36), FixedGrid(acc[..., 1:], 36)
        APIC.p2g(m, c, gm, gmu, sd, bins=b)
        return gm.to_float().cpu().numpy(), gmu.to_float().cpu().numpy()

    (gm, gmu), (gm2, gmu2) = grid(bins), grid(None)
    # FP32 sums of one or a few particles per node against single roundings
    assert rel_err(gm, gm2) <= 1e-5 and rel_err(gmu, gmu2) <= 1e-5
    ext = mesh.extent(LOC)
    acc = torch.zeros(ext + (4,), dtype=torch.int64, device="cuda")
    u = torch.zeros(ext + (3,), dtype=torch.float32, device="cuda")
    batch = Batch([BatchInstance(sd, m, c, FixedGrid(acc[..., 0], 36), FixedGrid(acc[..., 1:], 36), u,
                                 bins, 1e-12)], mode="phased")
    batch.step(graph=False)
    assert rel_err(acc[..., 0].double().cpu().numpy() * 2.0 ** -36, gm2) <= 1e-5
