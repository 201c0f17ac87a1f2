"""Work items cut into parts: one dense tile among sparse ones, so that its items run
in several parts while the others leave most of theirs empty, items of the smallest
chunk, and a last item shorter than a part, against the oracle.

Tolerance 5e-6 of the largest value: a contribution is about 10 roundings of 6e-8, a
part's stream adds at most 22 of them in registers and a node tile some 40 sums."""

import numpy as np
import pytest
import torch

import oracle
from particles import periodic_mesh, rel_err
from picasso_b200 import APIC, FieldLocation, FixedGrid, cell_sort, create_spline, permute_members

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [1, 2, 3])
@pytest.mark.parametrize("chunk,dense,sparse", [(32, 700, 65), (1000, 2500, 400), (4096, 5000, 64),
                                                (4096, 4097, 0)])
def test_dense_tile(cuda, order, chunk, dense, sparse):
    mesh = periodic_mesh(16, halo=1)
    rng = np.random.default_rng(dense)
    n = dense + sparse
    x = rng.random((n, 3))
    x[:dense] = 0.27 + 0.2 * x[:dense]
    m = rng.uniform(0.5, 1.5, n).astype(np.float32)
    c = rng.standard_normal((n, 4, 3)).astype(np.float32)
    c[:, 1:] *= 0.1
    loc = FieldLocation.Node
    dev = lambda a: torch.as_tensor(a, device="cuda")
    sd0 = create_spline(loc, order, mesh, dev(x))
    _, perm, bins = cell_sort(sd0, (4, 8, 8), chunk=chunk)
    xs, ms, cs = permute_members(perm, sd0.x, dev(m), dev(c))
    ext = mesh.extent(loc)
    acc = torch.zeros(ext + (4,), dtype=torch.int64, device="cuda")
    gm, gmu = FixedGrid(acc[..., 0], 36), FixedGrid(acc[..., 1:], 36)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    sd = create_spline(loc, order, mesh, xs)
    APIC.p2g(ms, cs, gm, gmu, sd, bins=bins, error_count=err)
    u = torch.as_tensor(rng.standard_normal(ext + (3,)).astype(np.float32), device="cuda")
    out = torch.zeros_like(cs)
    APIC.g2p(u, out, sd, bins=bins, error_count=err)
    sdo = create_spline(loc, order, mesh, None).desc
    gm_o, gmu_o = np.zeros(ext), np.zeros(ext + (3,))
    xh = xs.cpu().numpy()
    oracle.apic_p2g(sdo, xh, ms.double().cpu().numpy(), cs.double().cpu().numpy(), gm_o, gmu_o)
    out_o = np.zeros((n, 4, 3))
    oracle.apic_g2p(sdo, xh, u.double().cpu().numpy(), out_o)
    assert int(err) == 0
    assert rel_err(gm.to_float().cpu().numpy(), gm_o) <= 5e-6
    assert rel_err(gmu.to_float().cpu().numpy(), gmu_o) <= 5e-6
    assert rel_err(out[:, 0].cpu().numpy(), out_o[:, 0]) <= 5e-6  # 64 terms of 10 roundings
