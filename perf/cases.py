"""Workloads whose speed this framework is judged by, and their exact results.

Every case is what a particle-in-cell / material-point program does with the
library between two of its own steps: the APIC and PolyPIC transfers with the
grid velocity between them, the time loop with its re-sort and advection, the
first sort of a particle set, staggered (face) fields and batches of small
problems.  Positions, velocities, masses and affine / polynomial modes have
the distributions of the benchmark configurations (v ~ N(0, 1),
m ~ U[0.5, 1.5], C ~ N(0, 0.1), higher modes ~ N(0, 0.05); uniform in every
cell, or 70 % in 32 Gaussian blobs of two cells and 30 % uniform).

A pass leaves its inputs as they are: the transfers write their particle
results into arrays of their own, so that every pass does the same work (the
batch, whose instances own their particles, steps them in place).  The
fixed-point accumulators of the FP32 form are an intermediate of the pass;
what a program goes on with -- grid velocities, particle values, positions --
is returned whole.
"""

import itertools
import math
import random

import torch

import picasso_b200 as pb

FIXED_BITS = 36
THRESHOLD = 1e-12
GRAVITY = (0.0, 0.0, -9.81)

# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------


def _case(kind, cells, ppc, order, form, place="uniform", sort=False, periodic=True):
    """kind: step, loop, poly, sort or faces.  cells: "NX x NY x NZ".  place:
    uniform (ppc per cell, in cell order), shuffled (the same in random order)
    or clustered (random order).  sort: the particles are cell-sorted and the
    transfers get their bins."""
    return {"kind": kind, "nx": cells[0], "ny": cells[1], "nz": cells[2], "ppc": ppc,
            "order": order, "form": form, "place": place, "sort": sort, "periodic": periodic}


def _batch(count, max_edge, max_ppc, form, shapes):
    """`count` instances, edges from {16, 24, ..., max_edge}, 1 .. max_ppc
    particles per cell, order 2 or 3, all drawn from the seed `shapes`."""
    return {"kind": "batch", "count": count, "max_edge": max_edge, "max_ppc": max_ppc,
            "form": form, "shapes": shapes}


def listed():
    def named(name, case):
        return dict(case, name=name)

    return [
        # the headline workload: a large clustered set, FP32 form, sorted once
        named("step_fp32_256", _case("step", (256, 256, 256), 8, 2, "fp32", "clustered", True)),
        # the drop-in replacement of the reference: FP64, no sort, 64^3
        named("step_fp64_64", _case("step", (64, 64, 64), 8, 2, "fp64")),
        # the same arithmetic on a program's sorted, clustered particles
        named("step_fp64_sorted_128",
              _case("step", (128, 128, 128), 8, 2, "fp64", "clustered", True)),
        # cubic time loop with re-sort, permutation and advection, both forms
        named("loop_fp32_128", _case("loop", (128, 128, 128), 8, 3, "fp32")),
        named("loop_fp64_64", _case("loop", (64, 64, 64), 8, 3, "fp64")),
        # a debugging-size time loop, quadratic: launches and latency
        named("loop_fp32_12", _case("loop", (12, 12, 12), 4, 2, "fp32")),
        # PolyPIC with 27 modes in both forms, and with 8 modes on an odd box
        named("poly27_fp32_96", _case("poly", (96, 96, 96), 8, 2, "fp32", sort=True)),
        named("poly27_fp64_48", _case("poly", (48, 48, 48), 8, 2, "fp64", sort=True)),
        named("poly8_fp32_odd",
              _case("poly", (101, 67, 83), 5, 1, "fp32", "uniform", True, False)),
        # first sort of a random set: keys, permutation of the members, records
        named("sort_fp32_128", _case("sort", (128, 128, 128), 8, 2, "fp32", "clustered")),
        # staggered velocities on the three faces of an odd, closed box
        named("faces_fp64_odd", _case("faces", (45, 38, 53), 6, 2, "fp64", "shuffled", False,
                                      False)),
        # many small independent problems stepped from one captured graph
        named("batch_fp32", _batch(24, 64, 16, "fp32", 4)),
    ]


def draw(rng):
    kind = rng.choice(["step", "step", "step", "loop", "loop", "poly", "poly", "sort", "faces",
                       "batch"])
    form = rng.choice(["fp32", "fp64"])
    if kind == "batch":
        return _batch(rng.randint(6, 24), rng.choice([32, 40, 48, 56, 64]), rng.choice([4, 8, 16]),
                      form, rng.randint(0, 10 ** 6))
    # particles, spread over the logarithm of the kind's range
    most = {"step": 2e7, "loop": 1e7, "poly": 4e6, "sort": 2e7, "faces": 1e6}[kind]
    if form == "fp64":
        most /= 4
    total = math.exp(rng.uniform(math.log(3e3), math.log(most)))
    place = rng.choice(["uniform", "shuffled", "clustered"])
    # (a clustered set's background is about a third of its mean density)
    ppc = rng.randint(4 if place == "clustered" else 1, 16)
    edge = max(8.0, (total / ppc) ** (1.0 / 3.0))
    cells = [max(8, int(round(edge * rng.uniform(0.7, 1.4)))) for _ in range(3)]
    order = rng.choice([1, 2]) if kind == "poly" else rng.choice([1, 2, 2, 3])
    if kind == "faces":
        place = "uniform" if place == "uniform" else "shuffled"
        return _case(kind, cells, ppc, order, "fp64", place, False, rng.random() < 0.5)
    if kind in ("loop", "sort"):
        return _case(kind, cells, ppc, order, form, place)
    sort = form == "fp32" or rng.random() < 0.5
    # a closed box has nearly empty nodes at its sides, whose fixed-point
    # velocities only the bit-exact per-contribution sums (PolyPIC) repeat
    closed = (kind == "poly" or form == "fp64") and place != "clustered" and rng.random() < 0.4
    return _case(kind, cells, ppc, order, form, place, sort, not closed)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------


def _tile(case):
    return (4, 4, 8) if case["order"] == 3 else (4, 8, 8)


def _chunk(case):
    return 1024 if case["kind"] == "poly" else 4096


def _cell_size(case):
    return 1.0 / max(case["nx"], case["ny"], case["nz"])


def _dt(case):
    return 0.1 * _cell_size(case)


def _total(case):
    return case["nx"] * case["ny"] * case["nz"] * case["ppc"]


def _modes(case):
    return (8 if case["order"] == 1 else 27) if case["kind"] == "poly" else 4


def _particles(case, seed):
    """(x FP64, m, c) in the program's order, before any sort."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    dims = torch.tensor([case["nx"], case["ny"], case["nz"]], dtype=torch.float64, device="cuda")
    h = _cell_size(case)
    total = _total(case)

    def rand(*shape):
        return torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)

    if case["place"] == "clustered":
        blobs = int(total * 0.7)
        centre = rand(32, 3) * dims
        which = torch.randint(0, 32, (blobs,), generator=g, device="cuda")
        x = torch.empty((total, 3), device="cuda", dtype=torch.float64)
        x[:blobs] = 2.0 * torch.randn((blobs, 3), generator=g, device="cuda", dtype=torch.float64)
        x[:blobs] += centre[which]
        x[blobs:] = rand(total - blobs, 3) * dims
        x.remainder_(dims)
        x *= h
        x = torch.where(x >= dims * h, torch.zeros_like(x), x)
    else:
        cell = torch.arange(total, device="cuda") // case["ppc"]
        if case["place"] == "shuffled":
            cell = cell[torch.randperm(total, generator=g, device="cuda")]
        nz, ny = case["nz"], case["ny"]
        x = torch.stack([cell // (ny * nz), (cell // nz) % ny, cell % nz], dim=1).double()
        del cell
        x += rand(total, 3)
        x *= h
    real = torch.float32 if case["form"] == "fp32" else torch.float64
    m = (rand(total) + 0.5).to(real)
    modes = _modes(case)
    c = torch.randn((total, modes, 3), generator=g, device="cuda", dtype=real)
    c[:, 1:] *= 0.1 if modes == 4 else 0.05
    return x, m, c


def _mesh(case):
    h = _cell_size(case)
    return pb.UniformMesh([0.0, 0.0, 0.0, case["nx"] * h, case["ny"] * h, case["nz"] * h],
                          cell_size=h, periodic=(case["periodic"],) * 3,
                          halo_cell_width=0 if case["periodic"] else 2)


def _grids(mesh, loc, form):
    """Accumulator (mass, momentum), its two views and the velocity grid."""
    ext = mesh.extent(loc)
    if form == "fp32":
        acc = torch.zeros(ext + (4,), dtype=torch.int64, device="cuda")
        return (pb.FixedGrid(acc, FIXED_BITS), pb.FixedGrid(acc[..., 0], FIXED_BITS),
                pb.FixedGrid(acc[..., 1:], FIXED_BITS),
                torch.zeros(ext + (3,), dtype=torch.float32, device="cuda"))
    acc = torch.zeros(ext + (4,), dtype=torch.float64, device="cuda")
    return (acc, acc[..., 0], acc[..., 1:],
            torch.zeros(ext + (3,), dtype=torch.float64, device="cuda"))


def _drifted(case, seed):
    """Particles of a running time loop: sorted one step ago, then moved."""
    x, m, c = _particles(case, seed)
    sd = pb.create_spline(pb.FieldLocation.Node, case["order"], _mesh(case), x)
    perm = pb.cell_sort(sd, _tile(case), chunk=_chunk(case))[1]
    x, m, c = pb.permute_members(perm, x, m, c)
    x += _dt(case) * c[:, 0].double()
    size = torch.tensor([case["nx"], case["ny"], case["nz"]], dtype=torch.float64,
                        device="cuda") * _cell_size(case)
    x = torch.where(x < 0.0, x + size, x)
    x = torch.where(x >= size, x - size, x)
    return x.contiguous(), m, c


def _shapes(case):
    r = random.Random(case["shapes"])
    edges = list(range(16, case["max_edge"] + 1, 8))
    return [(r.choice(edges), r.randint(1, case["max_ppc"]), r.choice([2, 3]))
            for _ in range(case["count"])]


def _prepare_batch(case, seed):
    loc = pb.FieldLocation.Node
    instances, out = [], []
    for q, (edge, ppc, order) in enumerate(_shapes(case)):
        one = _case("step", (edge, edge, edge), ppc, order, case["form"])
        x, m, c = _particles(one, seed * 1000 + q)
        mesh = _mesh(one)
        sd = pb.create_spline(loc, order, mesh, x)
        perm, bins = pb.cell_sort(sd, _tile(one), chunk=4096)[1:]
        x, m, c = pb.permute_members(perm, x, m, c)
        _, gm, gmu, u = _grids(mesh, loc, case["form"])
        instances.append(pb.BatchInstance(pb.create_spline(loc, order, mesh, x), m, c, gm, gmu, u,
                                          bins, THRESHOLD))
        out.append((u, c))
    return {"kind": "batch", "batch": pb.Batch(instances, mode="phased"), "out": out}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return _prepare_batch(case, seed)
    loc = pb.FieldLocation.Node
    mesh = _mesh(case)
    order, form = case["order"], case["form"]
    s = {"kind": kind, "case": case, "mesh": mesh, "order": order, "form": form}
    if kind == "faces":
        x, m, c = _particles(case, seed)
        s.update(m=m, c=c, faces=[])
        for d in range(3):
            face = pb.FieldLocation.Face(d)
            s["faces"].append({"sd": pb.create_spline(face, order, mesh, x),
                               "desc": mesh.descriptor(face), "m_i": mesh.zeros(face),
                               "mu_i": mesh.zeros(face), "u_i": mesh.zeros(face),
                               "c": torch.zeros_like(c)})
        return s
    s["desc"] = mesh.descriptor(loc)
    if kind != "sort":
        s["acc"], s["gm"], s["gmu"], s["u"] = _grids(mesh, loc, form)
    x, m, c = _drifted(case, seed) if kind == "loop" else _particles(case, seed)
    sd = pb.create_spline(loc, order, mesh, x)
    if kind in ("loop", "sort"):
        s.update(x=x, m=m, c=c, sd=sd, bufs=pb.SortBuffers(sd, _tile(case)),
                 x_out=torch.empty_like(x), m_out=torch.empty_like(m), c_out=torch.empty_like(c))
        if form == "fp32":
            s["rec"] = torch.empty((x.shape[0], 4), dtype=torch.float32, device="cuda")
        return s
    bins = None
    if case["sort"]:
        perm, bins = pb.cell_sort(sd, _tile(case), chunk=_chunk(case))[1:]
        x, m, c = pb.permute_members(perm, x, m, c)
        sd = pb.create_spline(loc, order, mesh, x)
        if form == "fp32" and kind == "step":
            pb.spline_records(sd, bins)
    s.update(x=x, m=m, c=c, sd=sd, bins=bins, c_out=torch.zeros_like(c))
    return s


# ---------------------------------------------------------------------------
# passes
# ---------------------------------------------------------------------------


def run(s):
    return _RUN[s["kind"]](s)


def _grid_out(s):
    return {"u": s["u"], "grid": s["acc"]} if s["form"] == "fp64" else {"u": s["u"]}


def _run_step(s):
    pb.grid_fill(s["desc"], s["acc"], 0.0, ncomp=4)
    pb.APIC.p2g(s["m"], s["c"], s["gm"], s["gmu"], s["sd"], bins=s["bins"])
    pb.grid_velocity(s["desc"], s["gm"], s["gmu"], s["u"], THRESHOLD)
    pb.APIC.g2p(s["u"], s["c_out"], s["sd"], bins=s["bins"])
    return dict(_grid_out(s), c=s["c_out"])


def _run_poly(s):
    pb.grid_fill(s["desc"], s["acc"], 0.0, ncomp=4)
    pb.PolyPIC.p2g(s["m"], s["c"], s["c"], s["gmu"], s["gm"], _dt(s["case"]), s["sd"],
                   bins=s["bins"])
    pb.grid_velocity(s["desc"], s["gm"], s["gmu"], s["u"], THRESHOLD)
    pb.PolyPIC.g2p(s["u"], s["c_out"], s["sd"], bins=s["bins"])
    return dict(_grid_out(s), c=s["c_out"])


def _sorted(s):
    """Sort and permutation into the second member set; the sorted spline."""
    key, perm, bins = pb.cell_sort(s["sd"], _tile(s["case"]), chunk=_chunk(s["case"]),
                                   out=s["bufs"])
    for name in ("x", "m", "c"):
        pb.permute(perm, s[name], s[name + "_out"])
    sd = pb.create_spline(pb.FieldLocation.Node, s["order"], s["mesh"], s["x_out"])
    if s["form"] == "fp32":
        pb.spline_records(sd, bins, out=s["rec"])
    return key, perm, bins, sd


def _run_sort(s):
    key, perm, bins, _ = _sorted(s)
    out = {"key": key, "perm": perm, "x": s["x_out"], "m": s["m_out"], "c": s["c_out"],
           "tile_offset": bins.tile_offset, "tile_items": bins.tile_items}
    if s["form"] == "fp32":
        out["rec"] = s["rec"]
    return out


def _run_loop(s):
    _, perm, bins, sd = _sorted(s)
    dt = _dt(s["case"])
    pb.grid_fill(s["desc"], s["acc"], 0.0, ncomp=4)
    pb.APIC.p2g(s["m_out"], s["c_out"], s["gm"], s["gmu"], sd, bins=bins)
    pb.grid_update(s["desc"], s["gm"], s["gmu"], s["u"], dt, gravity=GRAVITY,
                   mass_threshold=THRESHOLD)
    pb.APIC.g2p_advect(s["u"], s["c_out"], sd, dt, bins=bins)
    return dict(_grid_out(s), perm=perm, x=s["x_out"], m=s["m_out"], c=s["c_out"])


def _run_faces(s):
    out = []
    for f in s["faces"]:
        pb.grid_fill(f["desc"], f["m_i"])
        pb.grid_fill(f["desc"], f["mu_i"])
        pb.APIC.p2g(s["m"], s["c"], f["m_i"], f["mu_i"], f["sd"])
    for f in s["faces"]:
        pb.grid_velocity(f["desc"], f["m_i"], f["mu_i"], f["u_i"], THRESHOLD)
        pb.APIC.g2p(f["u_i"], f["c"], f["sd"])
        out.append({"m": f["m_i"], "mu": f["mu_i"], "u": f["u_i"], "c": f["c"]})
    return out


def _run_batch(s):
    s["batch"].step(graph=True)
    return s["out"]


_RUN = {"step": _run_step, "poly": _run_poly, "sort": _run_sort, "loop": _run_loop,
        "faces": _run_faces, "batch": _run_batch}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------


def work(case):
    """Inputs read once, outputs written once; the multiplications and
    additions of the stencil sums."""
    if case["kind"] == "batch":
        parts = [work(_case("step", (e, e, e), p, o, case["form"], sort=True))
                 for e, p, o in _shapes(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n = _total(case)
    nodes = case["nx"] * case["ny"] * case["nz"]
    knots = (case["order"] + 1) ** 3
    real = 4 if case["form"] == "fp32" else 8
    state = real * (1 + 3 * _modes(case))  # mass and modes
    if case["kind"] == "sort":
        return {"bytes": n * (2 * (24 + state) + 8 + (16 if case["form"] == "fp32" else 0)),
                "flops": 0}
    grid_out = nodes * (3 * real if case["form"] == "fp32" else 7 * real)
    flops = n * knots * (2 + 3 * 8 + 1 + 3 * 8)
    if case["kind"] == "poly":
        flops = n * knots * 2 * 3 * (_modes(case) * 2)
    if case["kind"] == "loop":
        return {"bytes": n * (2 * 24 + 2 * state + 4) + grid_out, "flops": flops}
    if case["kind"] == "faces":
        return {"bytes": n * (24 + state + 3 * 12 * real) + 3 * nodes * 3 * real,
                "flops": 3 * n * knots * (2 + 8 + 1 + 8)}
    x = 16 if case["form"] == "fp32" and case["sort"] and case["kind"] == "step" else 24
    return {"bytes": n * (x + state + state - real) + grid_out, "flops": flops}


# ---------------------------------------------------------------------------
# exact results: plain torch in 64 bits
# ---------------------------------------------------------------------------
_SLAB = 1 << 21  # particles at a time


class _Grid:
    """Nodes of one field: first coordinate, spacing and count per dimension.
    offset: 0 on nodes, 1/2 between them."""

    def __init__(self, case, offset=(0.0, 0.0, 0.0)):
        h = _cell_size(case)
        halo = 0 if case["periodic"] else 2
        cells = (case["nx"], case["ny"], case["nz"])
        self.h, self.periodic = h, case["periodic"]
        self.n = [cells[d] + 2 * halo + (1 if offset[d] == 0.0 and not case["periodic"] else 0)
                  for d in range(3)]
        corner = 0.0 - halo * h
        self.lo = [corner + (0.0 + offset[d]) * h for d in range(3)]
        self.dx = [corner + (1.0 + offset[d]) * h - self.lo[d] for d in range(3)]

    def start(self, x, d, order):
        """First stencil node of every particle along d (not wrapped)."""
        q = (x[:, d] - self.lo[d]) * (1.0 / self.dx[d]) + (0.5 if order == 2 else 0.0)
        return torch.floor(q).long() - (0 if order == 1 else 1)

    def spline(self, x, d, order):
        """Node indices, weights, distances and weight gradients, (N, K)."""
        k = torch.arange(order + 1, device=x.device)
        node = self.start(x, d, order)[:, None] + k
        dist = self.lo[d] + node.double() * self.dx[d] - x[:, d:d + 1]
        r = dist / self.dx[d]
        a = r.abs()
        if order == 1:
            w, g = 1.0 - a, torch.where(k == 0, -1.0, 1.0).double().expand_as(a) / self.dx[d]
        elif order == 2:
            w = torch.where(k == 1, 0.75 - a * a, 0.5 * (1.5 - a) ** 2)
            g = None
        else:
            inner = 2.0 / 3.0 - a * a + 0.5 * a ** 3
            w = torch.where((k == 1) | (k == 2), inner, (2.0 - a) ** 3 / 6.0)
            g = None
        if self.periodic:
            node = node.remainder(self.n[d])
        return node, w, dist, g

    def stencil(self, x, order):
        """(flat node, knot triple, the three splines) of every stencil node."""
        sp = [self.spline(x, d, order) for d in range(3)]
        for ijk in itertools.product(range(order + 1), repeat=3):
            flat = (sp[0][0][:, ijk[0]] * self.n[1] + sp[1][0][:, ijk[1]]) * self.n[2] \
                + sp[2][0][:, ijk[2]]
            yield flat, ijk, sp


def _order_of(case, x):
    """The stable (tile, cell) order of the particles."""
    g = _Grid(case)
    tile = _tile(case)
    t, b = 0, 0
    for d in range(3):
        s = g.start(x, d, case["order"])
        if g.periodic:
            s = s.remainder(g.n[d])
        t = t * -(-g.n[d] // tile[d]) + s // tile[d]
        b = b * tile[d] + s % tile[d]
    return torch.argsort(t * (tile[0] * tile[1] * tile[2]) + b, stable=True)


def _slabs(*arrays):
    for a in range(0, arrays[0].shape[0], _SLAB):
        yield [v[a:a + _SLAB] for v in arrays]


def _weight(sp, ijk):
    return sp[0][1][:, ijk[0]] * sp[1][1][:, ijk[1]] * sp[2][1][:, ijk[2]]


def _distance(sp, ijk):
    return [sp[d][2][:, ijk[d]] for d in range(3)]


def _apic_to_grid(g, order, x, m, c, cols=(0, 1, 2)):
    acc = torch.zeros((g.n[0] * g.n[1] * g.n[2], 1 + len(cols)), dtype=torch.float64,
                      device=x.device)
    inertia = {1: 0.0, 2: 4.0, 3: 3.0}[order] / g.dx[0] ** 2
    for xs, ms, cs in _slabs(x, m.double(), c):
        cs = cs.double()[:, :, list(cols)]
        for flat, ijk, sp in g.stencil(xs, order):
            w = _weight(sp, ijk)
            if order == 1:
                v = w[:, None] * cs[:, 0]
                for a in range(3):
                    dw = [sp[d][3 if d == a else 1][:, ijk[d]] for d in range(3)]
                    v = v + (dw[0] * dw[1] * dw[2])[:, None] * cs[:, 1 + a]
            else:
                v = cs[:, 0].clone()
                for a, dist in enumerate(_distance(sp, ijk)):
                    v += inertia * dist[:, None] * cs[:, 1 + a]
                v *= w[:, None]
            acc.index_add_(0, flat, torch.cat([w[:, None], v], dim=1) * ms[:, None])
    return acc


def _apic_to_particles(g, order, x, u, cols=(0, 1, 2)):
    out = torch.zeros((x.shape[0], 4, 3), dtype=torch.float64, device=x.device)
    for xs, os in _slabs(x, out):
        for flat, ijk, sp in g.stencil(xs, order):
            wu = _weight(sp, ijk)[:, None] * u[flat]
            os[:, 0, list(cols)] += wu
            for a, dist in enumerate(_distance(sp, ijk)):
                os[:, 1 + a, list(cols)] += wu * dist[:, None]
    return out


def _velocity(acc, dt=0.0, gravity=(0.0, 0.0, 0.0)):
    keep = acc[:, :1] > THRESHOLD
    kick = dt * torch.tensor(gravity[:acc.shape[1] - 1], dtype=torch.float64, device=acc.device)
    return torch.where(keep, acc[:, 1:] / torch.where(keep, acc[:, :1], 1.0) + kick, 0.0)


def _degrees(order):
    first = [(0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (1, 0, 1), (0, 1, 1), (1, 1, 1)]
    return first + [t for t in itertools.product(range(order + 1), repeat=3) if t not in first]


def _poly_to_grid(g, order, x, m, c, dt):
    acc = torch.zeros((g.n[0] * g.n[1] * g.n[2], 4), dtype=torch.float64, device=x.device)
    degrees = _degrees(order)
    for xs, ms, cs in _slabs(x, m.double(), c):
        cs = cs.double()
        back = torch.linalg.inv(torch.eye(3, dtype=torch.float64, device=x.device) + dt * cs[:, 1:4])
        for flat, ijk, sp in g.stencil(xs, order):
            xi = (back @ torch.stack(_distance(sp, ijk), dim=1)[:, :, None])[:, :, 0]
            power = []
            for d in range(3):
                h, r = g.dx[d], xi[:, d]
                p = [torch.ones_like(r), r]
                if order == 2:
                    off = -sp[d][2][:, 1]
                    p.append(r * r - h * h / 4 - off * (h * h - 4 * off * off) / (h * h) * r)
                power.append(p)
            v = torch.zeros((xs.shape[0], 3), dtype=torch.float64, device=x.device)
            for q, (a, b, e) in enumerate(degrees):
                v += (power[0][a] * power[1][b] * power[2][e])[:, None] * cs[:, q]
            w = _weight(sp, ijk)[:, None]
            acc.index_add_(0, flat, torch.cat([w, w * v], dim=1) * ms[:, None])
    return acc


def _poly_to_particles(g, order, x, u):
    degrees = _degrees(order)
    out = torch.zeros((x.shape[0], len(degrees), 3), dtype=torch.float64, device=x.device)
    for xs, os in _slabs(x, out):
        for flat, ijk, sp in g.stencil(xs, order):
            factor = []
            for d in range(3):
                _, w, dist, grad = sp[d]
                k, h = ijk[d], g.dx[d]
                f = [w[:, k], grad[:, k] if order == 1 else 4.0 * w[:, k] * dist[:, k] / (h * h)]
                if order == 2:
                    f.append(torch.full_like(f[0], (0.5, -1.0, 0.5)[k] / (h * h)))
                factor.append(f)
            for q, (a, b, e) in enumerate(degrees):
                os[:, q] += (factor[0][a] * factor[1][b] * factor[2][e])[:, None] * u[flat]
    return out


def exact(case, seed):
    kind = case["kind"]
    # the batch steps its particles in place; a sort computes no numbers
    if kind in ("batch", "sort"):
        return None
    order = case["order"]
    if kind == "faces":
        x, m, c = _particles(case, seed)
        out = []
        for d in range(3):
            offset = [0.5, 0.5, 0.5]
            offset[d] = 0.0
            g = _Grid(case, offset)
            acc = _apic_to_grid(g, order, x, m, c, (d,))
            u = _velocity(acc)
            out.append({"m": acc[:, 0].reshape(g.n), "mu": acc[:, 1].reshape(g.n),
                        "u": u.reshape(g.n), "c": _apic_to_particles(g, order, x, u, (d,))})
        return out
    x, m, c = _drifted(case, seed) if kind == "loop" else _particles(case, seed)
    if kind == "loop" or case["sort"]:
        perm = _order_of(case, x)
        x, m, c = x[perm], m[perm], c[perm]
    g = _Grid(case)
    dt = _dt(case)
    if kind == "poly":
        acc = _poly_to_grid(g, order, x, m, c, dt)
        u = _velocity(acc)
        out = {"c": _poly_to_particles(g, order, x, u)}
    else:
        acc = _apic_to_grid(g, order, x, m, c)
        u = _velocity(acc, dt, GRAVITY) if kind == "loop" else _velocity(acc)
        out = {"c": _apic_to_particles(g, order, x, u)}
    out["u"] = u.reshape(g.n + [3])
    if case["form"] == "fp64":
        out["grid"] = acc.reshape(g.n + [4])
    if kind == "loop":
        out.update(perm=None, m=None)
        size = torch.tensor([case["nx"], case["ny"], case["nz"]], dtype=torch.float64,
                            device="cuda") * _cell_size(case)
        x = x + dt * out["c"][:, 0]
        out["x"] = torch.where(x < 0.0, x + size, torch.where(x >= size, x - size, x))
    return out
