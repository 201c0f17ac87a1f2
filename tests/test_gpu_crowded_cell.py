"""FP32 P2G of thousands of equal particles in one place: the streams of an uncut work
item (a batch with hundreds of tiles) must not add them up one by one.

Tolerance: a stream's sum takes at most 128 particles and the tile the sums of 64 at a
time, half an ulp (2^-24) each, and a contribution has some 10 roundings."""

import math

import numpy as np
import pytest
import torch

import oracle
from picasso_b200 import (Batch, BatchInstance, FieldLocation, FixedGrid, UniformMesh, cell_sort,
                          create_spline, permute_members)

pytestmark = pytest.mark.gpu
LOC = FieldLocation.Node


@pytest.mark.parametrize("order", [1, 2, 3])
@pytest.mark.parametrize("count,chunk", [(4096, 4096), (12288, 16384)])
def test_equal_particles(cuda, order, count, chunk):
    cells = (40, 64, 64)
    mesh = UniformMesh([0, 0, 0] + [c / 64 for c in cells], cell_size=1 / 64, periodic=(True,) * 3)
    x = np.tile(np.array([[17.37, 30.61, 9.23]]) / 64, (count, 1))
    m = np.full(count, 0.7, dtype=np.float32)
    c = np.zeros((count, 4, 3), dtype=np.float32)
    c[:, 0] = (1.3, -0.9, 0.4)
    dev = lambda a: torch.as_tensor(a, device="cuda")
    _, perm, bins = cell_sort(create_spline(LOC, order, mesh, dev(x)), (4, 8, 8), chunk=chunk)
    xs, ms, cs = permute_members(perm, dev(x), dev(m), dev(c))
    ext = mesh.extent(LOC)
    acc = torch.zeros(ext + (4,), dtype=torch.int64, device="cuda")
    gm, gmu = FixedGrid(acc[..., 0], 36), FixedGrid(acc[..., 1:], 36)
    u = torch.zeros(ext + (3,), dtype=torch.float32, device="cuda")
    Batch([BatchInstance(create_spline(LOC, order, mesh, xs), ms, cs, gm, gmu, u, bins, 1e-12)],
          mode="phased").step(graph=False)
    gm_o, gmu_o = np.zeros(ext), np.zeros(ext + (3,))
    oracle.apic_p2g(create_spline(LOC, order, mesh, None).desc, x, m.astype(float), c.astype(float),
                    gm_o, gmu_o)
    streams = {1: 8, 2: 3, 3: 2}[order]
    tol = (128 + streams * math.ceil(count / streams / 60) + 10) * 2.0 ** -24
    for got, want in ((gm, gm_o), (gmu, gmu_o)):
        got = got.to_float().cpu().numpy()
        full = np.abs(want) > 1e-3  # (the others hold less than the fixed point's last bits)
        assert full.sum() > (order + 1) ** 3 // 2
        assert np.max(np.abs(got[full] / want[full] - 1)) <= tol
