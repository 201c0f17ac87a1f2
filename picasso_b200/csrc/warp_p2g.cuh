// APIC P2G in FP64 by warps, on the FP64 tensor cores.
//
// A warp takes a contiguous segment of the particles, 32 at a time.  First
// every lane evaluates one particle into a shared table: its stencil weights
// with the mass folded in, and its affine velocity relative to the stencil's
// centre knot n0,
//   v(n) = E + sum_q G_q (n_q - n0),  E = v_p + D B dist(n0),  G = D dx B
// (Picasso_APIC.hpp:94-139).  A run of particles with the same stencil is then
// one contraction over its particles p,
//   C[node, (field, E | G_0 | G_1 | G_2)] = sum_p w_node(p) m(p) coef(p),
// done four particles at a time by mma.m8n8k4.f64 (IEEE FMAs), and node n of a
// field is C_E + sum_q (n_q - n0) C_Gq.  The columns are laid out so that a
// lane's accumulators hold all four coefficients of one field of its nodes and
// the four lanes of a row the four fields: the node values need no exchange
// and a grid addition covers whole nodes (one 32-byte sector of a packed
// accumulator).  A stencil that moves one node up along k keeps its other
// k-planes: the finished plane is added to the grid, the rest carried over.
// The particles may come in any order.  Where many of a warp's 32 particles
// change the stencil they are first put in the order of their stencils; where
// most still do (no neighbours among them), every particle's node values go
// straight to the grid, without the contraction.
//
// Measured (B200, against one thread per particle adding every contribution to
// the grid, which the L2's 200 G additions/s bound): quadratic 128^3 8 per cell
// clustered and sorted 31.7 -> 1.52 ms, 64^3 unsorted 1.28 -> 0.49 ms, shuffled
// 1.03 -> 0.52 ms (108 additions per particle at 440 G/s: whole sectors);
// cubic 64^3 sorted 4.83 -> 0.32 ms; linear 128^3 sorted 3.51 -> 1.10 ms; the
// faces of a 45 x 38 x 53 box, shuffled, 0.48 -> 0.35 ms.  A sorted quadratic
// particle costs about 60 ps plus 290 ps per stencil; what bounds it is the
// latency of a run's chain (table, contraction, node values) at 16 warps per
// SM, no unit is over half busy (tensor pipe 34 %, shared memory 41 %).
//
// Linear splines (gradient form, Picasso_APIC.hpp:276-318, 8 nodes) give every
// lane one (node, field) and take the particles one or two at a time.
#pragma once

#include "common.cuh"
#include "transfer.cuh"

namespace pb {

// D += A B: A 8x4 (row lane / 4, column lane % 4), B 4x8 (row lane % 4, column
// lane / 4), D 8x8 (row lane / 4, columns 2 (lane % 4), + 1).
__device__ __forceinline__ void mma_f64(double (&d)[2], double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

// p + s g for a small compile-time integer s (0: p exactly).
__device__ __forceinline__ double add_steps_f64(int s, double p, double g)
{
    return s == 0 ? p : (s == 1 ? p + g : (s == -1 ? p - g : fma((double)s, g, p)));
}

template <int ORDER, int NC, bool STAG>
struct WarpP2G {
    static constexpr int K = SplineTraits<ORDER>::K;
    static constexpr int KK = K * K;
    static constexpr int KKK = K * K * K;
    static constexpr int NV = STAG ? 1 : NC;   // momentum components of the grid
    static constexpr int NF = 1 + NV;          // grid fields
    static constexpr int NCI = STAG ? 3 : NC;  // columns of c_p
    // The nodes in row tiles of 8 (order >= 2).  The tile dimension is the last
    // of (D0, D1, D2), a row is a pair (n_D0, n_D1), D1 fastest.  Quadratic:
    // tile t < 3 holds the first 8 of the 9 pairs at n_D2 = t, tile 3 the ninth
    // pair at n_D2 = 0, 1, 2.  Cubic: tile t holds half t % 2 of the 16 pairs at
    // n_D2 = t / 2.  With several momentum components a node's fields fill a
    // sector and the k-planes are whole tiles (D2 = k); with one, the rows run
    // along k so that a grid addition covers consecutive nodes.
    static constexpr int MT = ORDER == 1 ? 1 : (ORDER == 2 ? 4 : 8);
    static constexpr bool KROWS = NV == 1;
    static constexpr int D0 = KROWS ? 1 : 0, D1 = KROWS ? 2 : 1, D2 = KROWS ? 0 : 2;
    static constexpr int NT = NF <= 2 ? 1 : 2;  // column tiles: 4 fields (2 for one tile)
    // linear: lanes per particle and particles at a time
    static constexpr int LP = 8 * NF;
    static constexpr int PER = ORDER == 1 ? 32 / LP : (NT == 1 ? 2 : 1);
    // Table: rows of 32 particles, 36 doubles apart (a quarter of the banks
    // further per row, so that the 4 particles x 8 rows a warp reads at once
    // are conflict-free).  Weights: the 9 or 16 pairs' w_D0 w_D1 m times w_D2
    // (quadratic: a row per node), or followed by w_D2 (cubic); linear w_x,
    // w_y, w_z.  Then 4 coefficients per momentum component (linear: per field),
    // coefficient r of component d in row r CF + d (the lanes of a value's fields
    // read consecutive rows), and the element offsets of the stencil's first node in the mass and
    // momentum arrays (-1: the stencil wraps or is none).
    static constexpr int ROW = 36;
    static constexpr int WROWS = ORDER == 1 ? 6 : (ORDER == 2 ? KKK : KK + K);
    static constexpr int CF = ORDER == 1 ? NF : NV;
    static constexpr int CROWS = 4 * CF;
    static constexpr int DOUBLES = (WROWS + CROWS + 2) * ROW;
    // Share of the 32 particles that start a new stencil from which on they go
    // straight to the grid: a run costs 290-400 ps more than its particles, the
    // direct way about 250 ps per particle with 4 fields and 190 ps with 2.
    static constexpr int kDirectNum = NT == 2 ? 5 : 3, kDirectDen = 8;
    // With one or two momentum components, particles in few rows (i, j) of which many
    // move the stencil are added by the lanes of their own: neighbouring lanes' nodes
    // then lie along k and an addition of the warp covers whole sectors.  Of 32 particles
    // at most kLaneRows rows, more than kLaneMoves moves.  1 M particles in cell order,
    // ms, as runs or node by node / this way / one thread per particle.  A face field:
    // linear 1 per cell 0.104 / 0.073 / 0.067, 8 per cell 0.131 / 0.080 / 0.083, 32 per
    // cell 0.092 / 0.110 / 0.156; quadratic 1 per cell 0.240 / 0.151 / 0.156, 4 per cell
    // 0.266 / 0.174 / 0.217, 12 per cell 0.167 / 0.209 / 0.376; cubic 1 per cell 0.450 /
    // 0.447 / 0.400, 6 per cell 0.687 / 0.418 / 0.588.  Two components: linear 1 per cell
    // 0.176 / 0.077 / 0.067; quadratic 2 per cell 0.425 / 0.327 / 0.322, 8 per cell 0.281
    // / 0.324 / 0.438; cubic 1 per cell 0.936 / 0.560 / 0.533, 2 per cell 0.401 / 0.592 /
    // 0.617.
    static constexpr int kLaneRows = 10;
    static constexpr int kLaneMoves =
        ORDER == 1 ? 4 : NV == 1 ? 9 : (ORDER == 2 ? 18 : 20);
};

// c_p packed (rows of 4 x NCI doubles, a multiple of 16 bytes) from a 16-byte
// aligned base: its rows may be read in 16-byte words.
template <int NCI>
inline bool wide_rows(const PField& c)
{
    return c.shift == 0 && c.tile_stride == 4 * NCI && c.comp_stride == 1 &&
           reinterpret_cast<uintptr_t>(c.data) % 16 == 0;
}

// A particle whose mass or coefficients are not all finite, node by node as it is defined
// (others: nothing): relative to the centre knot an infinite coefficient would make NaN,
// inf - inf or 0 inf, of nodes that are infinite.  Called at the segment's end: inside the
// loop it spills (quadratic 3 M sorted 0.282 -> 0.295 ms, this way 0.289).
template <int ORDER, int NC, bool STAG>
__device__ __forceinline__ void p2g_odd_particle(const MeshP& mp, int64_t p, const PField& x,
                                                 const PField& m, const PField& c,
                                                 const GField& gm, const GField& gmu, int stag)
{
    using W = WarpP2G<ORDER, NC, STAG>;
    constexpr int K = W::K;
    const double D = inertial_scaling<ORDER == 1 ? 2 : ORDER, double>(mp.dx[0]);
    unsigned top = high_bits(m.get<double>(p, 0));
    for (int q = 0; q < 4; ++q) {
        for (int d = 0; d < W::NV; ++d)
            top = max(top, high_bits(c.get<double>(p, q * W::NCI + (STAG ? stag : d))));
    }
    if (top < kNotFinite) return;
#pragma unroll 1
    for (int e = 0; e < W::KKK; ++e) {
        double w = m.get<double>(p, 0), dist[3];
        int g[3];
        bool ok = true;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const int n = d == 0 ? e / W::KK : (d == 1 ? e / K % K : e % K);
            const double xd = x.get<double>(p, d);
            const double x0 = logical_coord(xd, mp.lo[d], mp.rdx[d], SplineTraits<ORDER>::shift);
            Spline1D<ORDER, double> sp;
            spline_eval_f64<ORDER>(xd, mp.lo[d], mp.dx[d], mp.rdx[d], sp);
            w *= select<K>(sp.w, n);
            dist[d] = select<K>(sp.d, n);
            int idx[K];
            ok = resolve_stencil<K>(mp, d, (int)floor(x0) + SplineTraits<ORDER>::first, idx) && ok;
            g[d] = select<K>(idx, n);
        }
        if (!ok) return;  // out of the mesh, counted already
        atomicAdd(gm.ptr<double>(g[0], g[1], g[2], 0), w);
#pragma unroll 1
        for (int d = 0; d < W::NV; ++d) {
            const int col = STAG ? stag : d;
            double v = 0.0;
#pragma unroll
            for (int q = 0; q < 3; ++q) v = fma(c.get<double>(p, (1 + q) * W::NCI + col), dist[q], v);
            atomicAdd(gmu.ptr<double>(g[0], g[1], g[2], d),
                      w * fma(D, v, c.get<double>(p, col)));
        }
    }
}

// Adds the particles [a, b) to the grid; called by a whole warp.  sm:
// WarpP2G::DOUBLES doubles of the warp.  wide: wide_rows(c).
template <int ORDER, int NC, bool STAG>
__device__ __forceinline__ void apic_p2g_warp(const MeshP& mp, int64_t a, int64_t b,
                                              const PField& x, const PField& m, const PField& c,
                                              bool wide, const GField& gm, const GField& gmu,
                                              int stag, int* err, double* sm)
{
    using W = WarpP2G<ORDER, NC, STAG>;
    constexpr int K = W::K, KK = W::KK, NV = W::NV, NF = W::NF, NCI = W::NCI;
    constexpr int MT = W::MT, NT = W::NT, ROW = W::ROW, PER = W::PER;
    constexpr int CS = W::CF * ROW;  // between the coefficients of a component
    constexpr int D0 = W::D0, D1 = W::D1, D2 = W::D2;
    constexpr unsigned kAll = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    const int lg = lane >> 2, lt = lane & 3;  // row and column group of the lane
    double* coef = sm + W::WROWS * ROW;
    long long* first = reinterpret_cast<long long*>(coef + W::CROWS * ROW);

    // field of the grid values the lane holds, its place among the PER lanes
    // that hold the same value, and whether it has one at all
    const int field = ORDER == 1 ? lane % NF : (NT == 2 ? lt : lt >> 1);
    const int par = ORDER == 1 ? lane / W::LP : (PER == 2 ? lt & 1 : 0);
    const bool holds = ORDER == 1 ? lane < PER * W::LP : field < NF;
    // Node (n_D0, n_D1, n_D2) number t of the lane.  r0, r1: the pair of its row
    // (cubic: of the first half; linear: the node's i, j and in r2 its k).
    const int r0 = ORDER == 1 ? lane % W::LP / NF >> 1 & 1 : lg / K;
    const int r1 = ORDER == 1 ? lane % W::LP / NF & 1 : lg % K;
    const int r2 = ORDER == 1 ? lane % W::LP / NF >> 2 : 0;
    auto node_of = [&](int t, int (&n)[3]) {
        n[D0] = ORDER == 2 && t == 3 ? 2 : (ORDER == 3 && (t & 1) ? r0 + 2 : r0);
        n[D1] = ORDER == 2 && t == 3 ? 2 : r1;
        n[D2] = ORDER == 1 ? r2 : (ORDER == 2 ? (t == 3 ? lg : t) : t >> 1);
        if (ORDER == 1) n[0] = r0, n[1] = r1, n[2] = r2;
    };
    auto has_node = [&](int t, bool plane) {
        int n[3];
        node_of(t, n);
        return (ORDER != 2 || t < 3 || lg < 3) && (!plane || n[2] == 0);
    };
    const double o0 = r0 - 1, o1 = r1 - 1, o3 = lg - 1;
    // E + sum_q (n_q - n0) G_q for the lane's node number t
    auto affine = [&](int t, double E, double g0, double g1, double g2) {
        if (ORDER == 2 && t == 3) return fma(o3, g2, E + g0 + g1);
        const double v = fma(ORDER == 3 && (t & 1) ? o0 + 2.0 : o0, g0, fma(o1, g1, E));
        return add_steps_f64((ORDER == 3 ? t >> 1 : t) - 1, v, g2);
    };

    // wrap of a stencil index: [0, lim) then + off
    int lim[3], off[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        lim[d] = mp.periodic[d] ? mp.own_n[d] : 0x7FFFFFFF;
        off[d] = mp.periodic[d] ? mp.own_lo[d] : 0;
    }
    // place of each of the lane's nodes from the stencil's first node, in
    // elements of its field's array (a stencil that wraps, or strides past 32
    // bits, computes the addresses at every addition)
    bool near = gmu.s[3] <= (1 << 27);
#pragma unroll
    for (int d = 0; d < 3; ++d) near = near && gm.s[d] <= (1 << 27) && gmu.s[d] <= (1 << 27);
    int rel[MT];
#pragma unroll
    for (int t = 0; t < MT; ++t) {
        int n[3];
        node_of(t, n);
        const GField& g = field == 0 ? gm : gmu;
        rel[t] = n[0] * (int)g.s[0] + n[1] * (int)g.s[1] + n[2] * (int)g.s[2] +
                 (field == 0 ? 0 : (field - 1) * (int)g.s[3]);
    }
    double* const array = reinterpret_cast<double*>(field == 0 ? gm.data : gmu.data);
    const long long* my_first = first + (field == 0 ? 0 : ROW);
    // the lane's values of the nodes (of the first k-plane) of a stencil: from
    // the element offset of its first node, or (a stencil that wraps) from its
    // start
    auto add_at = [&](long long at, bool on, bool plane, const double (&v)[MT]) {
#pragma unroll
        for (int t = 0; t < MT; ++t)
            if (on && has_node(t, plane)) atomicAdd(array + at + rel[t], v[t]);
    };
    auto add_wrapped = [&](const int (&st)[3], bool on, bool plane, const double (&v)[MT]) {
#pragma unroll
        for (int t = 0; t < MT; ++t) {
            if (!on || !has_node(t, plane)) continue;
            int g[3];
            node_of(t, g);
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                g[d] += st[d];
                while (g[d] >= lim[d]) g[d] -= lim[d];
                g[d] += off[d];
            }
            atomicAdd(field == 0 ? gm.ptr<double>(g[0], g[1], g[2], 0)
                                 : gmu.ptr<double>(g[0], g[1], g[2], field - 1),
                      v[t]);
        }
    };
    // linear: the lane's node value of the particle in column q,
    //   m (c_0 www + sum_d c_d dw_d),  dw_d = +-1/dx w w of the other dimensions
    // (mass and 1/dx are in the coefficients, the signs are the node's)
    const int flip0 = r0 ? 0 : 0x80000000, flip1 = r1 ? 0 : 0x80000000, flip2 = r2 ? 0 : 0x80000000;
    auto flipped = [](double v, int flip) {
        return __hiloint2double(__double2hiint(v) ^ flip, __double2loint(v));
    };
    auto linear_value = [&](int q) {
        const double wx = sm[r0 * ROW + q], wy = sm[(2 + r1) * ROW + q],
                     wz = sm[(4 + (r2 & 1)) * ROW + q];
        const double* cf = coef + field * ROW + q;
        const double yz = fma(flipped(cf[3 * CS], flip2), wy, flipped(cf[2 * CS], flip1) * wz);
        return fma(fma(wx, cf[0], flipped(cf[CS], flip0)), wy * wz, wx * yz);
    };

    // The current run: offset of its stencil's first node (-1: it wraps, its
    // start is in `start`; -2: no run).
    long long cur = -2;
    int start[3] = {-1, -1, -1};
    // Sums of the current run: node values carried over from the previous
    // stencil (linear: the sums themselves) and the contraction's accumulators.
    double carry[MT], C[ORDER == 1 ? 1 : MT][NT][2];
    auto zero_c = [&] {
#pragma unroll
        for (int t = 0; t < (ORDER == 1 ? 1 : MT); ++t)
#pragma unroll
            for (int n = 0; n < NT; ++n) C[t][n][0] = C[t][n][1] = 0.0;
    };
    auto zero_carry = [&] {
#pragma unroll
        for (int t = 0; t < MT; ++t) carry[t] = 0.0;
    };
    zero_c();
    zero_carry();
    // The sums to the grid: all nodes, or (plane) those of the first k-plane,
    // with the rest carried one node down along k.
    auto flush = [&](bool plane) {
        double v[MT];
#pragma unroll
        for (int t = 0; t < MT; ++t) {
            if constexpr (ORDER == 1) {
                v[t] = carry[t];
                if (PER == 2) v[t] += __shfl_xor_sync(kAll, v[t], 16);
            } else if constexpr (NT == 2) {
                const double s = affine(t, C[t][0][0], C[t][0][1], C[t][NT - 1][0], C[t][NT - 1][1]);
                v[t] = carry[t] + (field == 0 ? C[t][0][0] : s);
            } else {
                // even lanes hold E, G_0, odd ones G_1, G_2
                const bool odd = lt & 1;
                const double h = affine(t, odd ? 0.0 : C[t][0][0], odd ? 0.0 : C[t][0][1],
                                        odd ? C[t][0][0] : 0.0, odd ? C[t][0][1] : 0.0);
                const double s = h + __shfl_xor_sync(kAll, h, 1);
                v[t] = carry[t] + (field == 0 ? C[t][0][0] : s);
            }
        }
        zero_c();
        if (cur >= 0) add_at(cur, holds && par == 0, plane, v);
        else add_wrapped(start, holds && par == 0, plane, v);
        if (!plane) {
            zero_carry();
            return;
        }
        if constexpr (ORDER == 1) {  // the lanes of k = 1 come LP / 2 later
            const double up = __shfl_down_sync(kAll, v[0], W::LP / 2);
            carry[0] = par == 0 && r2 == 0 ? up : 0.0;
        } else if constexpr (!W::KROWS) {  // k-planes are tiles
            if constexpr (ORDER == 2) {
                const double up = __shfl_down_sync(kAll, v[3], 4);
                carry[0] = v[1];
                carry[1] = v[2];
                carry[2] = 0.0;
                carry[3] = lg < 2 ? up : 0.0;
            } else {
#pragma unroll
                for (int t = 0; t < MT; ++t) carry[t] = t + 2 < MT ? v[t + 2 < MT ? t + 2 : 0] : 0.0;
            }
        } else {  // rows run along k; the quadratic ninth pair is in tile 3
#pragma unroll
            for (int t = 0; t < MT; ++t) {
                if (ORDER == 2 && t == 3) {
                    carry[t] = 0.0;
                } else {
                    double up = __shfl_down_sync(kAll, v[t], 4);
                    if (ORDER == 2) {
                        const double ninth = __shfl_sync(kAll, v[MT - 1], 4 * t + lt);
                        if (lg == 7) up = ninth;
                    }
                    carry[t] = r1 == K - 1 ? 0.0 : up;
                }
            }
        }
        // (lanes that share a value: one of them keeps it)
        if (PER == 2 && ORDER >= 2) {
#pragma unroll
            for (int t = 0; t < MT; ++t) carry[t] = par == 0 ? carry[t] : 0.0;
        }
    };

    int last[3] = {-1, -1, -1};  // stencil start of the previous particle
    bool odd = false;  // the lane has had a particle that p2g_odd_particle takes
    for (int64_t p0 = a; p0 < b; p0 += 32) {
        const int cnt = (int)min((int64_t)32, b - p0);
        int64_t p = p0 + lane;
        int s[3] = {-1, -1, -1};
        bool ok = lane < cnt;
        if (ok) {
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const double x0 = logical_coord(x.get<double>(p, d), mp.lo[d], mp.rdx[d],
                                                SplineTraits<ORDER>::shift);
                ok = stencil_start<K>(mp, d, (int)floor(x0) + SplineTraits<ORDER>::first, s[d]) && ok;
            }
            if (!ok) s[0] = s[1] = s[2] = -1;
        }
        if (p + 32 < b) {  // the next particles, into L2
            asm volatile("prefetch.global.L2 [%0];\n" ::"l"(
                reinterpret_cast<const double*>(x.data) + x.index(p + 32, 0)));
            asm volatile("prefetch.global.L2 [%0];\n" ::"l"(
                reinterpret_cast<const double*>(c.data) + c.index(p + 32, 0)));
        }
        // stencil changes against the previous particle, and the changes by
        // one node along k
        unsigned chg, step, rows;
        auto changes = [&] {
            int pv[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                pv[d] = __shfl_up_sync(kAll, s[d], 1);
                if (lane == 0) pv[d] = last[d];
            }
            const bool same2 = s[0] == pv[0] && s[1] == pv[1];
            const bool live = lane < cnt;
            chg = __ballot_sync(kAll, live && !(same2 && s[2] == pv[2]));
            step = __ballot_sync(kAll, live && same2 && s[0] >= 0 && s[2] == pv[2] + 1);
            rows = __ballot_sync(kAll, live && !same2);
        };
        changes();
        if (__popc(chg & ~step) > 8) {
            // the lane's particle becomes the one of its rank
            const unsigned key = warp_sort_by_stencil(
                lane < cnt, ((unsigned)s[0] * (unsigned)mp.ext[1] + (unsigned)s[1]) *
                                    (unsigned)mp.ext[2] + (unsigned)s[2]);
            const int src = key & 31;
            p = p0 + src;
            ok = __shfl_sync(kAll, ok, src);
#pragma unroll
            for (int d = 0; d < 3; ++d) s[d] = __shfl_sync(kAll, s[d], src);
            changes();
        }
        __syncwarp();  // the previous particles have been read
        if (lane < cnt) {
            if (!ok) {
                if (err) atomicAdd(err, 1);
                first[lane] = first[ROW + lane] = -1;
            } else {
                const bool inside = near && s[0] + K <= lim[0] && s[1] + K <= lim[1] &&
                                    s[2] + K <= lim[2];
                first[lane] =
                    inside ? gm.index(s[0] + off[0], s[1] + off[1], s[2] + off[2], 0) : -1;
                first[ROW + lane] =
                    inside ? gmu.index(s[0] + off[0], s[1] + off[1], s[2] + off[2], 0) : -1;
                Spline1D<ORDER, double> sp[3];
#pragma unroll
                for (int d = 0; d < 3; ++d)
                    spline_eval_f64<ORDER>(x.get<double>(p, d), mp.lo[d], mp.dx[d], mp.rdx[d], sp[d]);
                double cp[4 * NCI];
                if (wide) {
                    const double2* row =
                        reinterpret_cast<const double2*>(reinterpret_cast<const double*>(c.data) +
                                                         p * (4 * NCI));
#pragma unroll
                    for (int q = 0; q < 2 * NCI; ++q) {
                        const double2 v = __ldg(row + q);
                        cp[2 * q] = v.x;
                        cp[2 * q + 1] = v.y;
                    }
                } else {
#pragma unroll
                    for (int q = 0; q < 4 * NCI; ++q) cp[q] = c.get<double>(p, q);
                }
                const double mass = m.get<double>(p, 0);
                double* wt = sm + lane;
                if constexpr (ORDER == 1) {
#pragma unroll
                    for (int n = 0; n < K; ++n) {
                        wt[n * ROW] = sp[0].w[n];
                        wt[(K + n) * ROW] = sp[1].w[n];
                        wt[(2 * K + n) * ROW] = sp[2].w[n];
                        coef[n * CS + lane] = n == 0 ? mass : 0.0;
                        coef[(2 + n) * CS + lane] = 0.0;
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < K; ++i)
#pragma unroll
                        for (int j = 0; j < K; ++j) {
                            const double w2 = sp[D0].w[i] * mass * sp[D1].w[j];
                            if (ORDER == 3) {
                                wt[(i * K + j) * ROW] = w2;
                            } else {
#pragma unroll
                                for (int k = 0; k < K; ++k)
                                    wt[(k * KK + i * K + j) * ROW] = w2 * sp[D2].w[k];
                            }
                        }
                    if (ORDER == 3) {
#pragma unroll
                        for (int k = 0; k < K; ++k) wt[(KK + k) * ROW] = sp[D2].w[k];
                    }
                }
                const double D =
                    ORDER == 1 ? 1.0 : inertial_scaling<ORDER == 1 ? 2 : ORDER, double>(mp.dx[0]);
                unsigned top = high_bits(mass);
#pragma unroll
                for (int d = 0; d < NV; ++d) {
                    double v[4];
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        v[r] = cp[r * NCI + d];
                        if constexpr (STAG)
                            v[r] = stag == 0 ? v[r] : (stag == 1 ? cp[r * 3 + 1] : cp[r * 3 + 2]);
                    }
                    if constexpr (ORDER >= 2) {
#pragma unroll
                        for (int r = 0; r < 4; ++r) top = max(top, high_bits(v[r]));
                        const double bd =
                            fma(v[3], sp[2].d[1], fma(v[2], sp[1].d[1], v[1] * sp[0].d[1]));
                        v[0] = fma(D, bd, v[0]);
                        const double g[3] = {v[1] * (D * mp.dx[0]), v[2] * (D * mp.dx[1]),
                                             v[3] * (D * mp.dx[2])};
                        v[1] = g[D0];
                        v[2] = g[D1];
                        v[3] = g[D2];
                    } else {
                        v[0] *= mass;
#pragma unroll
                        for (int q = 0; q < 3; ++q) v[1 + q] *= mp.rdx[q] * mass;
                    }
#pragma unroll
                    for (int r = 0; r < 4; ++r)
                        coef[r * CS + (ORDER == 1 ? d + 1 : d) * ROW + lane] = v[r];
                }
                if constexpr (ORDER >= 2) {
                    if (top >= kNotFinite) {
                        odd = true;  // and the table without it
#pragma unroll 1
                        for (int r = 0; r < W::WROWS + W::CROWS; ++r) sm[r * ROW + lane] = 0.0;
                    }
                }
            }
        }
        const unsigned valid = __ballot_sync(kAll, s[0] >= 0);
        __syncwarp();
        if constexpr (NV < 3) {
            // every lane its own particle (kLaneRows)
            if (__popc(rows) <= W::kLaneRows && __popc(chg) * 32 > cnt * W::kLaneMoves) {
                if (cur >= -1) flush(false);
                cur = -2;
                if (s[0] >= 0) {
                    int node[3][K];  // grid indices of the stencil
#pragma unroll
                    for (int d = 0; d < 3; ++d)
#pragma unroll
                        for (int q = 0; q < K; ++q) {
                            int g = s[d] + q;
                            while (g >= lim[d]) g -= lim[d];
                            node[d][q] = g + off[d];
                        }
                    const double* wt = sm + lane;
                    double cf[NV][4];
#pragma unroll
                    for (int f = 0; f < NV; ++f)
#pragma unroll
                        for (int r = 0; r < 4; ++r)
                            cf[f][r] = coef[r * CS + (ORDER == 1 ? f + 1 : f) * ROW + lane];
#pragma unroll 1
                    for (int i = 0; i < K; ++i) {
                        const int gi = select<K>(node[0], i);
#pragma unroll
                        for (int j = 0; j < K; ++j) {
                            double* pm = gm.ptr<double>(gi, node[1][j], 0, 0);
                            double* pmu = gmu.ptr<double>(gi, node[1][j], 0, 0);
#pragma unroll
                            for (int k = 0; k < K; ++k) {
                                const int n[3] = {i, j, k};
                                const int pair = n[D0] * K + n[D1];
                                double w, v[NV];
                                if constexpr (ORDER == 1) {  // linear_value of all fields
                                    const double wx = wt[i * ROW], wy = wt[(2 + j) * ROW],
                                                 wz = wt[(4 + k) * ROW];
                                    w = coef[lane] * (wx * (wy * wz));
#pragma unroll
                                    for (int f = 0; f < NV; ++f) {
                                        const double x1 = i ? cf[f][1] : -cf[f][1], y1 = j ? cf[f][2] : -cf[f][2],
                                                     z1 = k ? cf[f][3] : -cf[f][3];
                                        v[f] = fma(fma(wx, cf[f][0], x1), wy * wz, wx * fma(z1, wy, y1 * wz));
                                    }
                                } else {
                                    w = ORDER == 3 ? wt[pair * ROW] * wt[(KK + n[D2]) * ROW]
                                                   : wt[(n[D2] * KK + pair) * ROW];
#pragma unroll
                                    for (int f = 0; f < NV; ++f)
                                        v[f] = w * fma((double)(n[D2] - 1), cf[f][3],
                                                       fma((double)(n[D1] - 1), cf[f][2],
                                                           fma((double)(n[D0] - 1), cf[f][1], cf[f][0])));
                                }
                                atomicAdd(pm + (int64_t)node[2][k] * gm.s[2], w);
#pragma unroll
                                for (int f = 0; f < NV; ++f)
                                    atomicAdd(pmu + (int64_t)node[2][k] * gmu.s[2] + f * gmu.s[3], v[f]);
                            }
                        }
                    }
                }
#pragma unroll
                for (int d = 0; d < 3; ++d) last[d] = -1;  // no run to continue
                continue;
            }
        }
        // table row of the weight of the lane's node number t (cubic: of its pair)
        auto wrow = [&](int t) {
            if (ORDER == 3) return ((t & 1) * 8 + lg) * ROW;
            return (t < 3 ? t * KK + lg : (lg < 3 ? lg : 0) * KK + KK - 1) * ROW;
        };
        if (__popc(chg) * W::kDirectDen > cnt * W::kDirectNum) {
            // no neighbours: node values straight to the grid, PER particles
            // at a time
            if (cur >= -1) flush(false);
            cur = -2;
#pragma unroll 2
            for (int q0 = 0; q0 < cnt; q0 += PER) {
                const int q = min(q0 + par, 31);
                const bool on = holds && q0 + par < cnt;
                const long long at = my_first[q];
                double v[MT];
                if constexpr (ORDER == 1) {
                    v[0] = linear_value(q);
                } else {
                    const double* cf = coef + (field == 0 || field >= NF ? 0 : field - 1) * ROW + q;
                    const double E = cf[0], g0 = cf[CS], g1 = cf[2 * CS], g2 = cf[3 * CS];
#pragma unroll
                    for (int t = 0; t < MT; ++t) {
                        double w = sm[wrow(t) + q];
                        if (ORDER == 3) w *= sm[(KK + (t >> 1)) * ROW + q];
                        v[t] = field == 0 ? w : w * affine(t, E, g0, g1, g2);
                    }
                }
                if (__any_sync(kAll, on && at < 0)) {
                    int st[3];
#pragma unroll
                    for (int d = 0; d < 3; ++d) st[d] = __shfl_sync(kAll, s[d], q);
                    add_wrapped(st, on && st[0] >= 0, false, v);
                } else {
                    add_at(at, on, false, v);
                }
            }
#pragma unroll
            for (int d = 0; d < 3; ++d) last[d] = -1;  // no run to continue
            continue;
        }
        for (int q = 0; q < cnt;) {
            if ((chg >> q) & 1u) {
                if (cur >= -1) flush((step >> q) & 1u);
                cur = (valid >> q) & 1u ? my_first[q] : -2;
                if (cur < 0) {
#pragma unroll
                    for (int d = 0; d < 3; ++d) start[d] = __shfl_sync(kAll, s[d], q);
                }
            }
            const unsigned later = q < 31 ? chg & (0xFFFFFFFEu << q) : 0u;
            const int end = later ? __ffs(later) - 1 : cnt;
            if (!((valid >> q) & 1u)) {
                q = end;
                continue;
            }
            if constexpr (ORDER == 1) {
#pragma unroll 2
                for (; q < end; q += PER)
                    if (PER == 1 || q + par < end) carry[0] += linear_value(q + par);
            } else {
                // column lg of the coefficients: its field and coefficients
                const int bf = NT == 2 ? lg >> 1 : lg >> 2;
                const int br = NT == 2 ? lg & 1 : lg & 3;
                const bool unit = bf == 0 && br == 0;
                const double* bp = coef + br * CS + (bf > 0 ? bf - 1 : 0) * ROW;
                // four particles; TAIL: past the run's end zeros (both factors,
                // so that no other particle's value enters)
                auto contract = [&](auto tail) {
                    constexpr bool TAIL = decltype(tail)::value;
                    const int pc = q + lt;
                    const bool in = !TAIL || pc < end;
                    double B[NT];
#pragma unroll
                    for (int n = 0; n < NT; ++n) {
                        B[n] = unit && n == 0 ? 1.0 : 0.0;
                        if (in && bf > 0 && bf < NF) B[n] = bp[2 * n * CS + pc];
                    }
#pragma unroll
                    for (int t = 0; t < MT; ++t) {
                        double A = in ? sm[wrow(t) + pc] : 0.0;
                        if (ORDER == 3) A *= in ? sm[(KK + (t >> 1)) * ROW + pc] : 0.0;
#pragma unroll
                        for (int n = 0; n < NT; ++n) mma_f64(C[t][n], A, B[n]);
                    }
                };
#pragma unroll 1
                for (; q + 4 <= end; q += 4) contract(std::false_type{});
                if (q < end) contract(std::true_type{});
            }
            q = end;
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) last[d] = __shfl_sync(kAll, s[d], cnt - 1);
    }
    if (cur >= -1) flush(false);
    if (ORDER >= 2 && __any_sync(kAll, odd)) {
        for (int64_t p = a + lane; p < b; p += 32)
            p2g_odd_particle<ORDER, NC, STAG>(mp, p, x, m, c, gm, gmu, stag);
    }
}

}  // namespace pb
