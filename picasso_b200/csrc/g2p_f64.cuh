// APIC G2P in FP64: one thread per particle (Picasso_APIC.hpp:407-544), its
// stencil contracted one dimension at a time, the results of a warp's 32
// particles written together.
//
// With the distances taken from the centre knot n0 (dist_q(n) = dist_q(n0) +
// (n_q - n0) dx),
//   u_p = sum w u,  M_q = sum w u (n_q - n0),  B_p(:, q) = dx M_q + dist_q(n0) u_p,
// and the sums over k, j and i in turn cost about 240 FP64 instructions per
// quadratic particle of three components instead of 440 node by node.  A thread
// storing its own row of 12 values touches a sector per value (a warp: 384
// sector writes for 3 KB); packed rows leave through shared memory, 32 rows at a
// time, in whole lines.  What bounds it are the L1 wavefronts of the gather, 81
// loads per quadratic particle:
//   * particles in any order read u_i from global memory, in the order of their
//     stencils inside a warp where they have little locality (linear, quadratic;
//     64^3 cells of 8: 0.214 ms as they come, 0.170 ms ordered, 90 % of the L1 data
//     pipe);
//   * large dense sets of cell-sorted particles (bins; g2p_tiles_pay) read it from a
//     node tile in shared memory (128^3 8 per cell clustered: 0.97 ms from global
//     memory, 0.74 ms).
// Against the form it replaces (node by node, every thread storing its row):
// sorted quadratic 128^3 1.28 -> 0.74 ms, cubic with advection 64^3 0.44 -> 0.17
// ms, unsorted quadratic 64^3 0.224 -> 0.170 ms, the faces of a 45 x 38 x 53 box
// 0.38 -> 0.14 ms.
#pragma once

#include "common.cuh"
#include "gridops.cuh"
#include "tiled.cuh"
#include "transfer.cuh"

namespace pb {

// Results of a warp: 4 x NCO values of c_p and, with advection, 3 coordinates
// per particle, at an odd stride.
template <int NCO, bool ADV>
struct WarpRows {
    static constexpr int NV = 4 * NCO;
    static constexpr int STRIDE = (NV + (ADV ? 3 : 0)) | 1;
    static constexpr int DOUBLES = 32 * STRIDE;
};

// Weights, and the distance to the centre knot, of one dimension: the formulas of
// spline_eval_f64 with every rounding written out, so that all kernels that
// gather (with and without advection, from a tile or not) get the same bits.
template <int ORDER>
__device__ __forceinline__ void g2p_spline(double x, double lo, double dx, double rdx, int& s0,
                                           double (&w)[SplineTraits<ORDER>::K], double& dist0)
{
    constexpr int N0 = ORDER == 1 ? 0 : 1;
    const double x0 = logical_coord(x, lo, rdx, SplineTraits<ORDER>::shift);
    const double fl = floor(x0);
    const double t = __dsub_rn(x0, fl);
    s0 = (int)fl + SplineTraits<ORDER>::first;
    if constexpr (ORDER == 1) {
        w[0] = __dsub_rn(1.0, t);
        w[1] = t;
    } else if constexpr (ORDER == 2) {
        const double a = __dsub_rn(t, 0.5), h = 0.5 * a;
        w[0] = __dadd_rn(fma(h, a, -h), 0.125);
        w[1] = fma(-a, a, 0.75);
        w[2] = __dadd_rn(fma(h, a, h), 0.125);
    } else {
        const double v = __dsub_rn(1.0, t), t2 = __dmul_rn(t, t), v2 = __dmul_rn(v, v);
        w[0] = __dmul_rn(__dmul_rn(v2, v), 1.0 / 6.0);
        w[1] = __dadd_rn(__dsub_rn(2.0 / 3.0, t2), __dmul_rn(0.5 * t, t2));
        w[2] = __dadd_rn(__dsub_rn(2.0 / 3.0, v2), __dmul_rn(0.5 * v, v2));
        w[3] = __dmul_rn(__dmul_rn(t2, t), 1.0 / 6.0);
    }
    dist0 = __dsub_rn(fma((double)(s0 + N0), dx, lo), x);
}

// u_p and B_p of one particle; load(i, j, k, d): component d at stencil node
// (i, j, k).
template <int ORDER, int NU, class Load>
__device__ __forceinline__ void g2p_contract(const MeshP& mp,
                                             const double (&ws)[3][SplineTraits<ORDER>::K],
                                             const double (&dist0)[3], double (&up)[NU],
                                             double (&B)[NU][3], Load&& load)
{
    constexpr int K = SplineTraits<ORDER>::K;
    constexpr int N0 = ORDER == 1 ? 0 : 1;
    double M[NU][3];
#pragma unroll
    for (int d = 0; d < NU; ++d) up[d] = M[d][0] = M[d][1] = M[d][2] = 0.0;
#pragma unroll
    for (int i = 0; i < K; ++i) {
        double A0[NU], A1[NU], A2[NU];
#pragma unroll
        for (int d = 0; d < NU; ++d) A0[d] = A1[d] = A2[d] = 0.0;
#pragma unroll
        for (int j = 0; j < K; ++j) {
            double S0[NU], S1[NU];
#pragma unroll
            for (int d = 0; d < NU; ++d) S0[d] = S1[d] = 0.0;
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const double w = ws[2][k], wk = w * (double)(k - N0);
#pragma unroll
                for (int d = 0; d < NU; ++d) {
                    const double v = load(i, j, k, d);
                    S0[d] = fma(w, v, S0[d]);
                    if (k != N0) S1[d] = fma(wk, v, S1[d]);
                }
            }
            const double w = ws[1][j], wj = w * (double)(j - N0);
#pragma unroll
            for (int d = 0; d < NU; ++d) {
                A0[d] = fma(w, S0[d], A0[d]);
                if (j != N0) A1[d] = fma(wj, S0[d], A1[d]);
                A2[d] = fma(w, S1[d], A2[d]);
            }
        }
        const double w = ws[0][i], wi = w * (double)(i - N0);
#pragma unroll
        for (int d = 0; d < NU; ++d) {
            up[d] = fma(w, A0[d], up[d]);
            if (i != N0) M[d][0] = fma(wi, A0[d], M[d][0]);
            M[d][1] = fma(w, A1[d], M[d][1]);
            M[d][2] = fma(w, A2[d], M[d][2]);
        }
    }
#pragma unroll
    for (int d = 0; d < NU; ++d)
#pragma unroll
        for (int q = 0; q < 3; ++q) B[d][q] = fma(mp.dx[q], M[d][q], __dmul_rn(dist0[q], up[d]));
}

// Results of the warp's particles p0 + at (ok: the lane has one): c_p(0, d) =
// u_p(d); c_p(1 + q, d) = B_p(d, q) (APIC.hpp:464-471), the gathered component of
// a staggered location in column stag, the others 0; with ADV the moved
// positions.  rows: the warp's shared buffer when c_p (and x_p) is packed, else
// null.
template <int NC, bool STAG, bool ADV>
__device__ __forceinline__ void g2p_store(int64_t p0, int at, bool ok, const double xp[3],
                                          const double (&up)[STAG ? 1 : NC],
                                          const double (&B)[STAG ? 1 : NC][3], const PField& x,
                                          const PField& c, int stag, const Advect* adv, double* rows)
{
    constexpr int NCO = STAG ? 3 : NC;
    using R = WarpRows<NCO, ADV>;
    const int lane = threadIdx.x & 31;
    const int64_t p = p0 + at;
    auto emit = [&](auto&& store) {
#pragma unroll
        for (int d = 0; d < NCO; ++d) {
            const int s = STAG ? 0 : d;
            const bool mine = !STAG || d == stag;
            store(d, mine ? up[s] : 0.0);
#pragma unroll
            for (int q = 0; q < 3; ++q) store((1 + q) * NCO + d, mine ? B[s][q] : 0.0);
        }
    };
    if (rows) {
        __syncwarp();  // the previous rows have been read
        if (ok) {
            double* mine = rows + at * R::STRIDE;
            emit([&](int v, double val) { mine[v] = val; });
            if constexpr (ADV) {
                const double uo[3] = {up[0], up[1], up[2]};
                advect_particle(*adv, p, xp, uo, [&](int d, double v) { mine[R::NV + d] = v; });
            }
        }
        const unsigned done = __reduce_or_sync(0xFFFFFFFFu, ok ? 1u << at : 0u);
        __syncwarp();
        double* dst = reinterpret_cast<double*>(c.data) + p0 * R::NV;
#pragma unroll
        for (int r = 0; r < R::NV; ++r) {
            const int e = lane + 32 * r, q = e / R::NV;
            if ((done >> q) & 1u) dst[e] = rows[q * R::STRIDE + (e - q * R::NV)];
        }
        if constexpr (ADV) {
            double* xd = reinterpret_cast<double*>(x.data) + p0 * 3;
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                const int e = lane + 32 * r, q = e / 3;
                if ((done >> q) & 1u) xd[e] = rows[q * R::STRIDE + R::NV + (e - q * 3)];
            }
        }
    } else if (ok) {
        emit([&](int v, double val) { c.set<double>(p, v, val); });
        if constexpr (ADV) {
            const double uo[3] = {up[0], up[1], up[2]};
            advect_particle(*adv, p, xp, uo, [&](int d, double v) { x.set<double>(p, d, v); });
        }
    }
}

// B_p of particle p node by node as it is defined, for the components whose u_p (in `up`)
// is not finite: relative to the centre knot an infinite node velocity makes NaN, inf - inf,
// of sums that are infinite.  After g2p_store (whose registers it then does not add to),
// by whole warps.  With advection the particle's position is not finite either, and stays.
template <int NU>
__device__ __forceinline__ bool g2p_odd(const double (&up)[NU])
{
    unsigned top = 0;
#pragma unroll
    for (int d = 0; d < NU; ++d) top = max(top, high_bits(up[d]));
    return top >= kNotFinite;
}
template <int ORDER, int NC, bool STAG, bool CG>
__device__ __forceinline__ void g2p_store_odd(const MeshP& mp, int64_t p, bool odd, const PField& x,
                                              const GField& u, const PField& c, int stag)
{
    constexpr int K = SplineTraits<ORDER>::K, NU = STAG ? 1 : NC, NCO = STAG ? 3 : NC;
    if (!__any_sync(0xFFFFFFFFu, odd)) return;  // (and the row has been written)
    if (!odd) return;
#pragma unroll 1
    for (int d = 0; d < NU; ++d) {
        double up = 0.0, b[3] = {0.0, 0.0, 0.0};
#pragma unroll 1
        for (int e = 0; e < K * K * K; ++e) {
            double w = 1.0, dist[3];
            int g[3];
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const int n = q == 0 ? e / (K * K) : (q == 1 ? e / K % K : e % K);
                const double xq = x.get<double>(p, q);
                double ws[K], dist0;
                int s0, idx[K];
                g2p_spline<ORDER>(xq, mp.lo[q], mp.dx[q], mp.rdx[q], s0, ws, dist0);
                resolve_stencil<K>(mp, q, s0, idx);
                w *= select<K>(ws, n);
                dist[q] = fma((double)(s0 + n), mp.dx[q], mp.lo[q]) - xq;
                g[q] = select<K>(idx, n);
            }
            const double* a = u.ptr<double>(g[0], g[1], g[2], d);
            const double wu = w * (CG ? __ldcg(a) : __ldg(a));
            up += wu;
#pragma unroll
            for (int q = 0; q < 3; ++q) b[q] = fma(wu, dist[q], b[q]);
        }
        if (high_bits(up) < kNotFinite) continue;
#pragma unroll
        for (int q = 0; q < 3; ++q) c.set<double>(p, (1 + q) * NCO + (STAG ? stag : d), b[q]);
    }
}

// u_p and B_p of a particle at xp gathered from u_i in global memory.  False (counted in
// err) if the stencil leaves a non-periodic mesh.  CG: u_i is read through L2 only
// (written earlier in the same launch).  UNIT: the components of u_i are adjacent.
template <int ORDER, int NU, bool CG, bool UNIT>
__device__ __forceinline__ bool g2p_gather(const MeshP& mp, const double (&xp)[3], const GField& u,
                                           int* err, double (&up)[NU], double (&B)[NU][3])
{
    constexpr int K = SplineTraits<ORDER>::K;
    double w[3][K], dist0[3];
    int idx[3][K];
    bool ok = true;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        int s0;
        g2p_spline<ORDER>(xp[d], mp.lo[d], mp.dx[d], mp.rdx[d], s0, w[d], dist0[d]);
        ok = resolve_stencil<K>(mp, d, s0, idx[d]) && ok;
    }
    if (!ok) {
        if (err) atomicAdd(err, 1);
        return false;
    }
    int64_t nk[K];
#pragma unroll
    for (int k = 0; k < K; ++k) nk[k] = (int64_t)idx[2][k] * u.s[2];
    const int64_t sc = UNIT ? 1 : u.s[3];
    g2p_contract<ORDER, NU>(mp, w, dist0, up, B, [&](int i, int j, int k, int d) {
        const double* a = reinterpret_cast<const double*>(u.data) +
                          (int64_t)idx[0][i] * u.s[0] +
                          (int64_t)idx[1][j] * u.s[1] + nk[k] + d * sc;
        return CG ? __ldcg(a) : __ldg(a);
    });
    return true;
}

// Particles p0 .. p0 + cnt - 1 (cnt <= 32) by a whole warp, gathered from global memory.
// ORDERED: the particles are taken as they come.  rows: see g2p_store.
template <int ORDER, int NC, bool STAG, bool CG, bool ADV, bool UNIT, bool ORDERED>
__device__ __forceinline__ void apic_g2p_warp(const MeshP& mp, int64_t p0, int cnt, const PField& x,
                                              const GField& u, const PField& c, int stag, int* err,
                                              const Advect* adv, double* rows)
{
    constexpr int K = SplineTraits<ORDER>::K;
    constexpr int NU = STAG ? 1 : NC;  // components of u_i
    constexpr unsigned kAll = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    int at = lane;  // the lane's particle among the warp's 32
    bool ok = lane < cnt;
    if constexpr (!ORDERED) {
        int s[3] = {-1, -1, -1};
        if (ok) {
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const double x0 = logical_coord(x.get<double>(p0 + lane, d), mp.lo[d], mp.rdx[d],
                                                SplineTraits<ORDER>::shift);
                stencil_start<K>(mp, d, (int)floor(x0) + SplineTraits<ORDER>::first, s[d]);
            }
        }
        const int prev0 = __shfl_up_sync(kAll, s[0], 1);
        const int prev1 = __shfl_up_sync(kAll, s[1], 1);
        const bool moved = s[0] != prev0 || s[1] != prev1;
        if (__popc(__ballot_sync(kAll, moved)) > 8)
            at = warp_sort_by_stencil(lane < cnt,
                                      ((unsigned)s[0] * (unsigned)mp.ext[1] + (unsigned)s[1]) *
                                              (unsigned)mp.ext[2] + (unsigned)s[2]) & 31;
    }
    double up[NU], B[NU][3], xp[3] = {0.0, 0.0, 0.0};
    if (ok) {
#pragma unroll
        for (int d = 0; d < 3; ++d) xp[d] = x.get<double>(p0 + at, d);
        ok = g2p_gather<ORDER, NU, CG, UNIT>(mp, xp, u, err, up, B);
    }
    const bool odd = !ADV && ok && g2p_odd(up);
    g2p_store<NC, STAG, ADV>(p0, at, ok, xp, up, B, x, c, stag, adv, rows);
    if (!ADV) g2p_store_odd<ORDER, NC, STAG, CG>(mp, p0 + at, odd, x, u, c, stag);
}

// A tile of node velocities in shared memory: `u` holds NU doubles per node of
// tile `ob` (bin origin) of tp.
struct NodeTile {
    const double* u;
    const TileP* tp;
    int ob[3];
    int i_lo, i_hi;  // bin rows staged
};

// u_p and B_p of one particle at xp gathered from global memory, the rows of its stencil
// in a loop (the same operations as g2p_contract, in few registers): for the particles
// that are not in the tile they were sorted into.  False if the stencil leaves a
// non-periodic mesh.  (A row at a time, its values in flight together; node by node
// quadratic sets of 8 per cell that had drifted since the sort took 1.6 times as long: 5 M
// drifted by 0.1 cells 0.75 ms, now 0.46, from global memory alone 0.32; as a loop of its
// own over the warps concerned, or with g2p_contract, the tile's gather spills and sorted
// sets lose 5 to 40 %.)
template <int ORDER, bool CG>
__device__ __forceinline__ bool g2p_stray(const MeshP& mp, const double xp[3], const GField& u,
                                          double (&up)[3], double (&B)[3][3])
{
    constexpr int K = SplineTraits<ORDER>::K;
    constexpr int N0 = ORDER == 1 ? 0 : 1;
    double w[3][K], dist0[3];
    int idx[3][K];
    bool ok = true;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        int s0;
        g2p_spline<ORDER>(xp[d], mp.lo[d], mp.dx[d], mp.rdx[d], s0, w[d], dist0[d]);
        ok = resolve_stencil<K>(mp, d, s0, idx[d]) && ok;
    }
    if (!ok) return false;
    double M[3][3];
#pragma unroll
    for (int d = 0; d < 3; ++d) up[d] = M[d][0] = M[d][1] = M[d][2] = 0.0;
    double A0[3] = {0.0, 0.0, 0.0}, A1[3] = {0.0, 0.0, 0.0}, A2[3] = {0.0, 0.0, 0.0};
#pragma unroll 1
    for (int e = 0; e < K * K; ++e) {
        const int i = e / K, j = e - i * K;
        const double* row = reinterpret_cast<const double*>(u.data) +
                            (int64_t)select<K>(idx[0], i) * u.s[0] + (int64_t)select<K>(idx[1], j) * u.s[1];
        double v[K][3];
#pragma unroll
        for (int k = 0; k < K; ++k)
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const double* a = row + (int64_t)idx[2][k] * u.s[2] + d * u.s[3];
                v[k][d] = CG ? __ldcg(a) : __ldg(a);
            }
        const double wy = select<K>(w[1], j), wj = wy * (double)(j - N0);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            double S0 = 0.0, S1 = 0.0;
#pragma unroll
            for (int k = 0; k < K; ++k) {
                S0 = fma(w[2][k], v[k][d], S0);
                if (k != N0) S1 = fma(w[2][k] * (double)(k - N0), v[k][d], S1);
            }
            A0[d] = fma(wy, S0, A0[d]);
            if (j != N0) A1[d] = fma(wj, S0, A1[d]);
            A2[d] = fma(wy, S1, A2[d]);
        }
        if (j == K - 1) {
            const double wx = select<K>(w[0], i), wi = wx * (double)(i - N0);
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                up[d] = fma(wx, A0[d], up[d]);
                if (i != N0) M[d][0] = fma(wi, A0[d], M[d][0]);
                M[d][1] = fma(wx, A1[d], M[d][1]);
                M[d][2] = fma(wx, A2[d], M[d][2]);
                A0[d] = A1[d] = A2[d] = 0.0;
            }
        }
    }
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
        for (int q = 0; q < 3; ++q) B[d][q] = fma(mp.dx[q], M[d][q], __dmul_rn(dist0[q], up[d]));
    return true;
}

// Particles p0 .. p0 + cnt - 1 of a tile, three components, by a whole warp:
// gathered from the tile.
template <int ORDER, bool CG, bool ADV>
__device__ __forceinline__ void g2p_tile_warp(const MeshP& mp, const NodeTile& nt, int64_t p0,
                                              int cnt, const PField& x, const GField& u,
                                              const PField& c, int* err, const Advect* adv,
                                              double* rows)
{
    constexpr int K = SplineTraits<ORDER>::K;
    const int lane = threadIdx.x & 31;
    const TileP& tp = *nt.tp;
    bool ok = lane < cnt;
    double xp[3] = {0.0, 0.0, 0.0}, up[3], B[3][3];
    if (ok) {
        int lb[3];
        bool mine = true;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            xp[d] = x.get<double>(p0 + lane, d);
            const int s0 = (int)floor(logical_coord(xp[d], mp.lo[d], mp.rdx[d],
                                                    SplineTraits<ORDER>::shift)) +
                           SplineTraits<ORDER>::first;
            if (!mp.periodic[d] && (s0 < 0 || s0 > mp.ext[d] - K)) mine = false;
            lb[d] = bin_of(mp, tp, d, s0) - nt.ob[d];
            if (lb[d] < 0 || lb[d] >= tp.T[d]) mine = false;
        }
        if (mine && lb[0] >= nt.i_lo && lb[0] <= nt.i_hi) {
            double w[3][K], dist0[3];
            int s0;
#pragma unroll
            for (int d = 0; d < 3; ++d)
                g2p_spline<ORDER>(xp[d], mp.lo[d], mp.dx[d], mp.rdx[d], s0, w[d], dist0[d]);
            const int e2 = tp.NT[2], e12 = tp.NT[1] * e2;
            const double* base = nt.u + 3 * ((lb[0] * tp.NT[1] + lb[1]) * e2 + lb[2]);
            g2p_contract<ORDER, 3>(mp, w, dist0, up, B, [&](int i, int j, int k, int d) {
                return base[3 * (i * e12 + j * e2 + k) + d];
            });
        } else {
            ok = g2p_stray<ORDER, CG>(mp, xp, u, up, B);
            if (!ok && err) atomicAdd(err, 1);
        }
    }
    const bool odd = !ADV && ok && g2p_odd(up);
    g2p_store<3, false, ADV>(p0, lane, ok, xp, up, B, x, c, -1, adv, rows);
    if (!ADV) g2p_store_odd<ORDER, 3, false, CG>(mp, p0 + lane, odd, x, u, c, -1);
}

// One work item (tile t, particles [a, b)) of cell-sorted particles by NTHR
// threads: the node velocities the item's bin rows can touch are staged in
// `nodes` (3 doubles per tile node), then every warp takes 32 particles at a
// time.  Particles that are not in the tile (they have moved since the sort) are
// gathered from global memory.  rows: a WarpRows buffer per warp, or null.
template <int ORDER, int NTHR, bool CG, bool ADV>
__device__ __forceinline__ void g2p_item_f64(const MeshP& mp, const TileP& tp, int64_t t, int64_t a,
                                             int64_t b, const PField& x, const GField& u,
                                             const PField& c, int* err, const Advect* adv,
                                             double* nodes, double* rows, int tid)
{
    constexpr int K = SplineTraits<ORDER>::K;
    NodeTile nt;
    nt.u = nodes;
    nt.tp = &tp;
    tile_origin(tp, t, nt.ob);
    nt.i_lo = 0;
    nt.i_hi = tp.T[0] - 1;
    {   // bin rows of the first and last particle (keys are i-major in a tile)
        const double shift = SplineTraits<ORDER>::shift;
        int r[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const double x0 = logical_coord(x.get<double>(q ? b - 1 : a, 0), mp.lo[0], mp.rdx[0], shift);
            r[q] = bin_of(mp, tp, 0, (int)floor(x0) + SplineTraits<ORDER>::first) - nt.ob[0];
        }
        if (r[0] >= 0 && r[0] <= r[1] && r[1] < tp.T[0]) {
            nt.i_lo = r[0];
            nt.i_hi = r[1];
        }
    }
    auto sync = [] {
        if (NTHR == 32) __syncwarp();
        else __syncthreads();
    };
    sync();  // the previous item's threads are done with the tile (and, with
             // advection, every thread has read the two positions)
    const int e2 = tp.NT[2], e1 = tp.NT[1];
    const int rows_n = (nt.i_hi - nt.i_lo + K) * e1;
    for (int e = tid; e < rows_n * e2; e += NTHR) {
        const int k = e % e2, ij = e / e2;
        const int j = ij % e1, i = nt.i_lo + ij / e1;
        int g[3] = {nt.ob[0] + i, nt.ob[1] + j, nt.ob[2] + k};
        bool inside = true;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            if (mp.periodic[d]) {
                while (g[d] >= tp.nb[d]) g[d] -= tp.nb[d];
                g[d] += mp.own_lo[d];
            } else {
                inside = inside && g[d] < mp.ext[d];
            }
        }
        if (inside) {
            const double* src = u.ptr<double>(g[0], g[1], g[2], 0);
            double* dst = nodes + 3 * ((i * e1 + j) * e2 + k);
#pragma unroll
            for (int d = 0; d < 3; ++d) dst[d] = CG ? __ldcg(src + d * u.s[3]) : __ldg(src + d * u.s[3]);
        }
    }
    sync();
    double* mine = rows ? rows + (tid >> 5) * WarpRows<3, ADV>::DOUBLES : nullptr;
    for (int64_t p0 = a + (tid & ~31); p0 < b; p0 += NTHR)
        g2p_tile_warp<ORDER, CG, ADV>(mp, nt, p0, (int)min((int64_t)32, b - p0), x, u, c, err, adv,
                                      mine);
}

// Whether the bins' node tiles pay against gathering from global memory: enough particles
// per staged node, and tiles small enough for 4 CTAs on an SM.  2 M sorted particles,
// tile / global memory, ms: linear tile (4, 8, 8) 8 per cell 0.077 / 0.084 and 4 per cell
// (2.5 per node) 0.084 / 0.084; quadratic 4 per cell (1.7) 0.107 / 0.123, 2 per cell
// 0.137 / 0.139, 1 per cell 0.211 / 0.164, tile (4, 4, 8) 4 per cell (1.4) 0.121 / 0.122,
// (2, 2, 2) 1 per cell 1.98 / 0.17; cubic 2 per cell (0.6) 0.197 / 0.219, tile (4, 4, 8)
// 2 per cell (0.5) 0.230 / 0.218; (8, 16, 16), 2 CTAs, 8 per cell, quadratic 0.176 /
// 0.121.
inline bool g2p_tiles_pay(const TileP& tp, int order, int64_t n)
{
    const double per_node = (double)n / ((double)tp.ntiles * tp.nodes);
    return 3 * sizeof(double) * (size_t)tp.nodes <= 40 * 1024 &&
           per_node >= (order == 1 ? 4.5 : order == 2 ? 1.5 : 0.55);
}

// c_p (ncv values per particle) and, with adv, x_p are packed rows.
inline bool packed_rows_f64(const PField& x, const PField& c, int ncv, bool adv)
{
    return c.shift == 0 && c.tile_stride == ncv && c.comp_stride == 1 &&
           (!adv || (x.shift == 0 && x.tile_stride == 3 && x.comp_stride == 1));
}

}  // namespace pb
