"""The FP32 loop of linear splines and of sparse quadratic sets rounds its sums as it
always has: FP64 positions follow FP32 velocities, so another order of the P2G's sums,
or another rounding of the G2P's, moves a particle to another place (1e-9 of the box
away).  The digests are those of the sums in runs of 32 per work item, with nvcc 12.9;
they hold for the accumulators of the P2G, from positions and from records and with the
grid update in it, and for the positions after G2P with advection.

A batch and staggered fields move no particle and may sum in another order."""

import hashlib

import numpy as np
import pytest
import torch

from picasso_b200 import (APIC, FieldLocation, FixedGrid, UniformMesh, cell_sort, create_spline,
                          grid_velocity, permute_members, spline_records)

pytestmark = pytest.mark.gpu
LOC = FieldLocation.Node


def _sequence(n, columns, first):
    """n x columns values in [0, 1): multiples of irrational steps, the same anywhere."""
    roots = np.sqrt(np.array([2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37, 41, 43, 47, 53, 59.0]))
    return np.mod(np.arange(1, n + 1)[:, None] * roots[first:first + columns], 1.0)


def _digest(t):
    return hashlib.sha256(np.ascontiguousarray(t.cpu().numpy()).tobytes()).hexdigest()[:16]


def step(order, cells, n, dense, periodic, tile, chunk):
    """(digest of the accumulators, of the advected positions) of one FP32 step."""
    h = 1.0 / max(cells)
    hi = np.array(cells) * h
    mesh = UniformMesh([0, 0, 0] + list(hi), cell_size=h, periodic=(periodic,) * 3,
                       halo_cell_width=0 if periodic else 2)
    x = _sequence(n, 3, 0) * hi
    x[:dense] = hi * (0.3 + 0.25 * x[:dense] / hi)  # a dense corner
    dev = lambda a, t: torch.as_tensor(a, dtype=t, device="cuda")
    m = dev(_sequence(n, 1, 3)[:, 0] + 0.5, torch.float32)
    c = dev((4.0 * _sequence(n, 12, 4) - 2.0).reshape(n, 4, 3), torch.float32)
    sd = create_spline(LOC, order, mesh, dev(x, torch.float64))
    _, perm, bins = cell_sort(sd, tile, chunk=chunk)
    x, m, c = permute_members(perm, sd.x, m, c)
    sd = create_spline(LOC, order, mesh, x)
    ext = mesh.extent(LOC)
    sums = []
    for how in ("positions", "records") + (("fused",) if periodic else ()):
        if how == "records":
            spline_records(sd, bins)
        acc = torch.zeros(ext + (4,), dtype=torch.int64, device="cuda")
        gm, gmu = FixedGrid(acc[..., 0], 36), FixedGrid(acc[..., 1:], 36)
        u = torch.zeros(ext + (3,), dtype=torch.float32, device="cuda")
        if how == "fused":
            APIC.p2g_update(m, c, gm, gmu, u, sd, bins=bins)
        else:
            APIC.p2g(m, c, gm, gmu, sd, bins=bins)
            grid_velocity(mesh.descriptor(LOC), gm, gmu, u, 1e-12)
        sums.append(_digest(acc))
    assert len(set(sums)) == 1
    APIC.g2p_advect(u, c, sd, 0.1 * h, bins=bins)
    return sums[0], _digest(x)


# order, cells, particles, of these in a dense corner, periodic, tile, chunk
CASES = {
    "linear": ((1, (10, 9, 11), 8000, 2000, True, (4, 8, 8), 4096),
              ("d4af937a9f58c3de", "f66a98652e1233f2")),
    "linear_sparse_closed": ((1, (9, 12, 8), 700, 0, False, (4, 4, 8), 97),
                            ("0046069f61159c3c", "fa1ecd9773ac3221")),
    "linear_dense_tile": ((1, (8, 8, 8), 9000, 8000, True, (8, 8, 8), 4096),
                         ("9be5ea4657196234", "54228420132df236")),
    "quadratic_sparse": ((2, (10, 9, 11), 3900, 1000, True, (4, 8, 8), 4096),
                        ("5921cc1b4b5b4746", "20e3ec207171d81f")),
    "quadratic_one_per_cell": ((2, (9, 12, 8), 864, 0, True, (3, 5, 4), 128),
                              ("7f90b1d16e6c0309", "fd4d7451bedd0ddb")),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_sums_and_positions_repeat(cuda, name):
    args, want = CASES[name]
    assert step(*args) == want
