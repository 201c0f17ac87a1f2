// Work items of the shared-memory tiled APIC transfers (FP32 precision form)
// on cell-sorted particles in packed storage: x_p (N,3) FP64, m_p (N) FP32,
// c_p (N,4,3) FP32.  Used by the single-call kernels (tiled.cu) and by the
// persistent batched kernel (batch.cu).
//
// Work items are chunks of at most `chunk` particles of one tile (the sort
// writes the per-tile item prefix).
//
// P2G item (one warp; linear splines and sparse quadratic sets: run_p2g.cuh): the item's
// sorted particles are cut into S contiguous
// streams (3 for quadratic, 2 for cubic, 8 for linear splines) that the warp
// sweeps side by side.  The lanes first evaluate the next 32 / S particles of
// every stream, one particle each (splines, the affine velocity relative to the
// stencil's centre knot), into a shared table; then, step by step, K^2 lanes per
// stream -- one for every k-row of the stencil -- add the stream's next particle
// to their K nodes' sums in registers.  When a stream's stencil moves, its lanes
// add the nodes that are finished (one k-plane for a move along k, else all) to
// the warp's FP32 node tile ((T + K - 1)^3 nodes), stream after stream: a fixed
// order without atomics, so the tile sums are reproducible.  At the end of the
// item the touched box of the tile is rounded to 64-bit fixed point and added to
// HBM with integer reductions, whose result does not depend on their order; P2G
// is deterministic for a given particle order.
//
// G2P item (one warp or one CTA): the item's node velocities are staged once
// in a shared float4 tile and every thread gathers its particles' stencils
// from there, contracting the stencil one dimension at a time.
//
// Both read either the FP64 positions or, when the bins carry them, spline
// records (in-cell fractions as FP32 + sort key, written by
// picasso_spline_records from the same FP64 arithmetic): same splines and
// bins, 16 instead of 24 bytes per particle, no FP64 instruction.  Staggered
// locations (Face / Edge) accumulate two grid fields (mass and the entity's
// momentum component) instead of four.  The P2G can also apply the grid
// update to the nodes whose sums are complete (fused_update_arrive).
#pragma once

#include "common.cuh"
#include "gridops.cuh"
#include "transfer.cuh"

namespace pb {

constexpr unsigned kFull = 0xFFFFFFFFu;

struct TileP {
    int T[3];    // bins per tile
    int nt[3];   // tiles per dimension
    int nb[3];   // bins per dimension
    int NT[3];   // nodes per tile dimension (T + K - 1)
    int nodes;   // NT0 * NT1 * NT2
    int SJ, SI;  // P2G node-tile strides along j and i (k stride 1), padded so
                 // that a plane's nodes fall on distinct banks
    int P;       // node slots of the P2G tile (NT0 * SI, in runs padded too)
    bool runs;   // P2G in runs (run_p2g.cuh)
    int chunk;
    int split;       // parts an item of the bins is cut into at most (set_parts)
    int part;        // particles of a part, if `split` parts suffice
    int64_t items_max;  // items of the bins, at most
    int tsh[3];      // log2(T[d]) when T[d] is a power of two, else -1
    uint32_t tsize;  // bins per tile (sort keys of tile t start at t * tsize)
    int64_t ntiles;
    const int64_t* off;     // tile particle offsets (ntiles + 1)
    const uint32_t* items;  // tile work-item prefix (ntiles + 1)
};

// Neighbour grids of a slab decomposition along x: the local x-planes below
// lo_end are the lower neighbour's planes (index + lo_shift there), those
// from hi_begin on the upper neighbour's (index + hi_shift); the neighbours'
// grids have the local strides.  P2G adds the sums of those nodes into the
// neighbour's grid (lo[0] / hi[0]: mass, [1]: momentum) and G2P reads their
// velocities from it ([0]): the halo exchange happens inside the transfers,
// through peer memory when the neighbour is another GPU.
struct HaloPeers {
    int on;
    int lo_end, hi_begin;
    int lo_shift, hi_shift;
    char* lo[2];
    char* hi[2];
};

// Grid base holding local x-plane gi (own, or a neighbour's field f) and the
// plane's index there.
__device__ __forceinline__ char* halo_route(const HaloPeers& hp, int f, char* own, int gi, int& gx)
{
    gx = gi;
    if (hp.on) {
        if (gi < hp.lo_end) {
            gx = gi + hp.lo_shift;
            return hp.lo[f];
        }
        if (gi >= hp.hi_begin) {
            gx = gi + hp.hi_shift;
            return hp.hi[f];
        }
    }
    return own;
}

// Per-call (per-instance) arguments of the tiled kernels.
struct P2GArgs {
    MeshP mp;
    TileP tp;
    int stag;          // staggered location: the entity's dimension (else -1)
    const double* x;
    const float* rec;  // spline records (4 floats per particle) or null
    const float* m;
    const float* c;
    GField gm;
    GField gmu;
    float scale_m;
    float scale_mu;
    int* err;
    // gm and gmu are one packed accumulator (a node's mass and momentum are 4
    // consecutive 64-bit words, 16-byte aligned): the item's flush adds whole
    // k-rows with bulk reductions (flush_rows_bulk)
    int bulk_flush;
    HaloPeers hp;
};

struct G2PArgs {
    MeshP mp;
    TileP tp;
    int stag;           // staggered location: the entity's dimension (else -1)
    const double* x;
    const float4* rec;  // spline records or null
    GField u;
    float* c;
    int* err;
    double* x_out;  // G2P with advection: positions updated in place (= x)
    Advect adv;
    HaloPeers hp;
};

// Static shared memory of the batch's kernels, which copy these arguments there: the
// launch that runs all phases holds both.
constexpr int kBatchStaticSmem = (int)((sizeof(P2GArgs) + 15) / 16 * 16 + (sizeof(G2PArgs) + 15) / 16 * 16);

__device__ __forceinline__ int bin_of(const MeshP& mp, const TileP& tp, int d, int s0)
{
    if (mp.periodic[d]) {
        const int nb = tp.nb[d];
        int r = s0 - mp.own_lo[d];
        if (r < 0) r += nb;          // one period covers every particle inside or
        else if (r >= nb) r -= nb;   // next to the owned box
        if ((unsigned)r >= (unsigned)nb) {
            r %= nb;
            if (r < 0) r += nb;
        }
        return r;
    }
    return s0;
}

// Node of the tile with bin origin ob along d.  (A tile with its halo can span several
// periods of a thin mesh.)
__device__ __forceinline__ int node_global(const MeshP& mp, const TileP& tp, int d, int ob,
                                           int local)
{
    int g = ob + local;
    if (mp.periodic[d]) {
        const int nb = tp.nb[d];
        if (g >= nb) {
            g -= nb;
            if (g >= nb) g %= nb;
        }
        return mp.own_lo[d] + g;
    }
    return g;
}

// Work item w -- part w / items_max of item w % items_max of the bins, so that the
// parts beyond an item's last are launched after the others -> tile t (-1 past the
// last item) and particle range [a, b); called by whole warps.  False if it has
// no particles.  The tile is searched 32 at a time: the dependent loads of a binary
// search (11 for 1224 tiles) are what an empty part costs.
__device__ __forceinline__ bool item_range(const TileP& tp, int64_t w, int64_t& t, int64_t& a,
                                           int64_t& b)
{
    int part = 0;
    if (tp.split > 1) {
        part = (int)(w / tp.items_max);
        w -= part * tp.items_max;
    }
    t = -1;
    const int lane = threadIdx.x & 31;
    const int64_t items = (int64_t)__ldg(tp.items + tp.ntiles);
    int64_t lo = 0, hi = tp.ntiles - 1;  // last t with items[t] <= w
    while (lo < hi) {
        const int64_t step = (hi - lo + 32) >> 5;
        const int64_t at = lo + lane * step;
        const unsigned below = __ballot_sync(0xFFFFFFFFu, at <= hi && (int64_t)__ldg(tp.items + at) <= w);
        lo += (__popc(below | 1u) - 1) * step;
        hi = min(hi, lo + step - 1);
    }
    if (w >= items) return false;
    t = lo;
    a = __ldg(tp.off + t) + (w - (int64_t)__ldg(tp.items + t)) * tp.chunk;
    b = min(a + (int64_t)tp.chunk, (int64_t)__ldg(tp.off + t + 1));
    if (tp.split > 1) {  // equal parts of whole warps, the rest empty
        const int np = max(1, min(tp.split, (int)((b - a + tp.part - 1) / tp.part)));
        const int64_t len = ((b - a + np - 1) / np + 31) & ~int64_t(31);
        a += part * len;
        b = min(a + len, b);
    }
    return a < b;
}

__device__ __forceinline__ void tile_origin(const TileP& tp, int64_t t, int ob[3])
{
    ob[2] = (int)(t % tp.nt[2]) * tp.T[2];
    ob[1] = (int)((t / tp.nt[2]) % tp.nt[1]) * tp.T[1];
    ob[0] = (int)(t / ((int64_t)tp.nt[1] * tp.nt[2])) * tp.T[0];
}

// Spline of a particle at x and its bin inside the tile with bin origin ob;
// false if the particle is not in this tile (or not in the mesh).
template <int ORDER>
__device__ __forceinline__ bool locate(const MeshP& mp, const TileP& tp, const double xp[3],
                                       const int ob[3], Spline1D<ORDER, float> sp[3], int lb[3])
{
    constexpr int K = SplineTraits<ORDER>::K;
    bool ok = true;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        eval_spline<ORDER>(xp[d], mp.lo[d], mp.dx[d], mp.rdx[d], sp[d]);
        if (!mp.periodic[d] && (sp[d].s0 < 0 || sp[d].s0 > mp.ext[d] - K)) ok = false;
        lb[d] = bin_of(mp, tp, d, sp[d].s0) - ob[d];
        if (lb[d] < 0 || lb[d] >= tp.T[d]) ok = false;
    }
    return ok;
}

// ---------------------------------------------------------------------------
// bulk reductions (shared -> global through the tensor memory accelerator;
// both addresses 16-byte aligned, size a multiple of 16 bytes)
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned smem_addr(const void* p)
{
    return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void bulk_add_u64(long long* dst, const long long* src, int bytes)
{
    asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.u64 [%0], [%1], %2;\n"
                 ::"l"(dst), "r"(smem_addr(src)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;\n" ::: "memory"); }
// the shared-memory sources of this thread's committed bulk operations have
// been read (the buffer may be rewritten)
__device__ __forceinline__ void bulk_wait_read()
{
    asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");
}
// shared-memory writes of this thread become visible to the bulk operations
__device__ __forceinline__ void fence_proxy_async_smem()
{
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
}

// ---------------------------------------------------------------------------
// P2G
// ---------------------------------------------------------------------------
// Field g of a node n = (a, b, c) of a bin receives
//   w_n m (e_d + sum_q G_dq (n_q - n0))                     (order 2 / 3)
//   m (c0 www + cx gww + cy wgw + cz wwg)                    (order 1)
// for the momentum components d = g - 1 and w_n m for the mass (g = 0), with
// n0 the stencil's centre knot, e_d = v_d + D sum_q B_dq dist_q(n0) and
// G_dq = D dx B_dq: the affine term D B dist (APIC.hpp:110-139) written
// relative to the centre knot, where dist_q(n) - dist_q(n0) = (n_q - n0) dx,
// so the nodes next to the centre need one addition and the centre none.
// Order 1: APIC.hpp:287-318 with D = 1; the gradients are +-w w / dx, so a k-row
// (a, b) of weight w_ab = w_a w_b receives (c0 m w_ab + cx m gx_a w_b + cy m gy_b
// w_a) w_c +- (cz m / dx) w_ab.
//
// STAG: a staggered location (Face<D> / Edge<D>, APIC.hpp:148-232): two
// grid fields, the mass and the one momentum component of the entity's
// dimension, which comes from column `stag` of c_p.
template <int ORDER, bool STAG>
struct P2GCfg {
    static constexpr int K = SplineTraits<ORDER>::K;
    static constexpr int KK = K * K;            // lanes per stream, a k-row each
    static constexpr int NV = STAG ? 1 : 3;     // momentum components
    static constexpr int NF = 1 + NV;           // grid fields
    static constexpr int S = 32 / KK;           // streams
    static constexpr int B = 32 / S;            // table slots per stream
    // Table entry of a particle: (E, G_x, G_y, G_z) per component (linear: m times
    // c0 and the gradient coefficients), w_z, (linear: m), the tile offset of its
    // stencil's first node (-1: skipped).  20 floats: the 16-byte stores of 8
    // lanes fall on distinct banks.
    static constexpr int ENTRY = 20, WZ = 4 * NV, AT = WZ + K + (ORDER == 1 ? 1 : 0);
    static_assert(AT < ENTRY, "a particle's entry");
    // entries of a stream; linear and cubic ones 4 floats further apart, so that the
    // streams' reads (16 bytes, one address each) fall on distinct banks
    static constexpr int SE = B * ENTRY + (ORDER == 2 ? 0 : 4);
    static constexpr int TABLE = ORDER == 2 ? 32 * ENTRY : S * SE;
    // then w_x w_y m per k-row (linear: w_x, w_y) in rows of 33
    static constexpr int WROWS = ORDER == 1 ? 2 * K : KK, WROW = 33;
    static constexpr int TILE_OFF = (TABLE + WROWS * WROW + 3) & ~3;
};

// Single-warp CTAs per SM the P2G register budget is sized for.
constexpr int kP2GOccupancy = 16;

template <int ORDER, bool STAG = false>
__host__ __device__ constexpr int p2g_warp_floats(int P)
{
    return P2GCfg<ORDER, STAG>::TILE_OFF + P2GCfg<ORDER, STAG>::NF * P;
}

// p + s g for a small integer s (s = 0: p exactly).  Called with unrolled
// loop indices, so the branch folds at compile time.
__device__ __forceinline__ float add_steps(int s, float p, float g)
{
    if (s == 0) return p;
    if (s == 1) return p + g;
    if (s == -1) return p - g;
    return fmaf((float)s, g, p);
}

// Bin inside tile t of a particle from its sort key; false if the key is
// not one of the tile's bins (another tile, or outside the mesh).
__device__ __forceinline__ bool bin_of_key(const TileP& tp, int64_t t, uint32_t key, int lb[3])
{
    const uint32_t ll = key - (uint32_t)t * tp.tsize;
    uint32_t r;
    if (tp.tsh[2] >= 0) {
        lb[2] = (int)(ll & (uint32_t)(tp.T[2] - 1));
        r = ll >> tp.tsh[2];
    } else {
        r = ll / (uint32_t)tp.T[2];
        lb[2] = (int)(ll - r * (uint32_t)tp.T[2]);
    }
    if (tp.tsh[1] >= 0) {
        lb[1] = (int)(r & (uint32_t)(tp.T[1] - 1));
        lb[0] = (int)(r >> tp.tsh[1]);
    } else {
        const uint32_t r2 = r / (uint32_t)tp.T[1];
        lb[1] = (int)(r - r2 * (uint32_t)tp.T[1]);
        lb[0] = (int)r2;
    }
    return ll < tp.tsize;
}

// Spline of a particle from its record (in-cell fractions, key) and its bin
// inside tile t; false if the particle is not in this tile.
template <int ORDER>
__device__ __forceinline__ bool locate_record(const MeshP& mp, const TileP& tp, int64_t t,
                                              float4 r, Spline1D<ORDER, float> sp[3], int lb[3])
{
    const bool ok = bin_of_key(tp, t, __float_as_uint(r.w), lb);
    spline_from_frac<ORDER, float>(r.x, (float)mp.dx[0], mp.rdx[0], sp[0]);
    spline_from_frac<ORDER, float>(r.y, (float)mp.dx[1], mp.rdx[1], sp[1]);
    spline_from_frac<ORDER, float>(r.z, (float)mp.dx[2], mp.rdx[2], sp[2]);
    return ok;
}

// Flush of a P2G item's node box (bin rows [i_lo, i_hi] plus the halo, the
// whole tile along j and k) into a packed accumulator: the box's k-rows are
// rounded to fixed point into `buf` (room for buf_nodes nodes of 4 words, a
// group of rows at a time) and each row is added to HBM by one bulk
// reduction (one more for every time it wraps around a periodic boundary; rows and
// nodes past a non-periodic mesh end are left out -- no stencil reaches them).
// The integer sums do not depend on the order of the reductions.
template <int ORDER, class Values>
__device__ __forceinline__ void flush_rows_bulk(const P2GArgs& A, Values&& values, int i_lo, int i_hi,
                                                const int ob[3], float* buf_f, int buf_nodes,
                                                int lane)
{
    constexpr int K = SplineTraits<ORDER>::K;
    const MeshP& mp = A.mp;
    const TileP& tp = A.tp;
    long long* buf = reinterpret_cast<long long*>(buf_f);
    const int e1 = tp.NT[1], e2 = tp.NT[2];
    const int rows = (i_hi - i_lo + K) * e1;
    const int per = buf_nodes / e2;  // rows per group (>= 1, checked by the host)
    // nodes of a row before the periodic wrap or the mesh end along k
    const int gk0 = node_global(mp, tp, 2, ob[2], 0);
    const int n0 = mp.periodic[2] ? min(e2, tp.nb[2] - ob[2]) : min(e2, mp.ext[2] - gk0);
    const int nk = mp.periodic[2] ? e2 : n0;  // nodes of a row to add
    for (int r0 = 0; r0 < rows; r0 += per) {
        const int nr = min(per, rows - r0);
        if (r0 > 0) {  // the previous group's rows have been read
            bulk_wait_read();
            __syncwarp();
        }
        for (int node = lane; node < nr * e2; node += 32) {  // node of the group
            const int q = node / e2;
            const int k = node - q * e2;
            const int row = r0 + q;
            const int i = i_lo + row / e1, j = row - (row / e1) * e1;
            const int idx = i * tp.SI + j * tp.SJ + k;
            float x[4];
            values(idx, x);
            long long w[4];
#pragma unroll
            for (int f = 0; f < 4; ++f)
                w[f] = x[f] != 0.f ? to_fixed(f == 0 ? A.gm : A.gmu,
                                              x[f] * (f == 0 ? A.scale_m : A.scale_mu))
                                   : 0LL;
            longlong2* d = reinterpret_cast<longlong2*>(buf + 4 * node);
            d[0] = make_longlong2(w[0], w[1]);
            d[1] = make_longlong2(w[2], w[3]);
        }
        fence_proxy_async_smem();
        __syncwarp();
        for (int q = lane; q < nr; q += 32) {
            const int row = r0 + q;
            const int i = i_lo + row / e1, j = row - (row / e1) * e1;
            const int gi = node_global(mp, tp, 0, ob[0], i);
            const int gj = node_global(mp, tp, 1, ob[1], j);
            if ((!mp.periodic[0] && gi >= mp.ext[0]) || (!mp.periodic[1] && gj >= mp.ext[1]))
                continue;
            const long long* src = buf + (size_t)q * e2 * 4;
            if (n0 > 0) bulk_add_u64(A.gm.ptr<long long>(gi, gj, gk0, 0), src, n0 * 32);
            for (int k = n0; k < nk; k += tp.nb[2])
                bulk_add_u64(A.gm.ptr<long long>(gi, gj, mp.own_lo[2], 0), src + 4 * k,
                             min(nk - k, tp.nb[2]) * 32);
        }
        bulk_commit();
    }
    bulk_wait_read();  // the buffer is the next item's table
    __syncwarp();
}

// A P2G item's node box (values(idx, x): the NF fields at tile index idx), rounded to
// fixed point and added to HBM: by bulk reductions of whole k-rows into a packed
// accumulator (`buf`, room for buf_nodes nodes, holds the rounded rows), else node by
// node (nodes that received nothing are skipped).  any: the item added something.
template <int ORDER, int NF, class Values>
__device__ __forceinline__ void flush_tile(const P2GArgs& A, Values&& values, bool any, int i_lo,
                                           int i_hi, const int ob[3], float* buf, int buf_nodes,
                                           int lane)
{
    constexpr int K = SplineTraits<ORDER>::K;
    const MeshP& mp = A.mp;
    const TileP& tp = A.tp;
    if (!any) return;
    if (NF == 4 && A.bulk_flush) {
        if constexpr (NF == 4) flush_rows_bulk<ORDER>(A, values, i_lo, i_hi, ob, buf, buf_nodes, lane);
        return;
    }
    const int e1 = tp.NT[1], e2 = tp.NT[2];
    const int total = (i_hi - i_lo + K) * e1 * e2;
    for (int e = lane; e < total; e += 32) {
        const int k = e % e2;
        const int j = (e / e2) % e1;
        const int i = i_lo + e / (e1 * e2);
        const int idx = i * tp.SI + j * tp.SJ + k;
        const int gi = node_global(mp, tp, 0, ob[0], i);
        const int gj = node_global(mp, tp, 1, ob[1], j);
        const int gk = node_global(mp, tp, 2, ob[2], k);
        // this rank's grids, or the neighbour's that owns plane gi
        int gx_m, gx_mu;
        char* bm = halo_route(A.hp, 0, A.gm.data, gi, gx_m);
        char* bmu = halo_route(A.hp, 1, A.gmu.data, gi, gx_mu);
        float v[NF];
        values(idx, v);
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            if (v[f] != 0.f) {
                const long long q =
                    to_fixed(f == 0 ? A.gm : A.gmu, v[f] * (f == 0 ? A.scale_m : A.scale_mu));
                unsigned long long* dst =
                    f == 0 ? reinterpret_cast<unsigned long long*>(bm) + A.gm.index(gx_m, gj, gk, 0)
                           : reinterpret_cast<unsigned long long*>(bmu) +
                                 A.gmu.index(gx_mu, gj, gk, NF == 2 ? 0 : f - 1);
                atomicAdd(dst, (unsigned long long)q);
            }
        }
    }
}

// Bin rows [i_lo, i_hi] spanned by an item's particles [a, b) (keys are i-major within
// a tile): the first and last particle bound them; the item's node box is these rows
// plus the halo, over the whole tile along j and k.
template <int ORDER, bool REC>
__device__ __forceinline__ void p2g_rows(const P2GArgs& A, int64_t t, int64_t a, int64_t b,
                                         const int ob[3], int& i_lo, int& i_hi)
{
    const MeshP& mp = A.mp;
    const TileP& tp = A.tp;
    i_lo = 0;
    i_hi = tp.T[0] - 1;
    int la[3], lz[3];
    bool oka, okb;
    if constexpr (REC) {
        oka = bin_of_key(tp, t, __float_as_uint(__ldg(A.rec + 4 * a + 3)), la);
        okb = bin_of_key(tp, t, __float_as_uint(__ldg(A.rec + 4 * (b - 1) + 3)), lz);
    } else {
        Spline1D<ORDER, float> sp[3];
        const double xa[3] = {A.x[3 * a], A.x[3 * a + 1], A.x[3 * a + 2]};
        const double xb[3] = {A.x[3 * (b - 1)], A.x[3 * (b - 1) + 1], A.x[3 * (b - 1) + 2]};
        oka = locate<ORDER>(mp, tp, xa, ob, sp, la);
        okb = locate<ORDER>(mp, tp, xb, ob, sp, lz);
    }
    if (oka && okb && lz[0] >= la[0]) {
        i_lo = la[0];
        i_hi = lz[0];
    }
}

// One P2G work item (tile t, particles [a, b)) by the calling warp.  `warp_smem`
// holds p2g_warp_floats<ORDER, STAG>(P) floats (16-byte aligned).  REC: the
// particles' positions arrive as spline records (in-cell fraction of the
// logical position along each dimension in FP32, and the sort key of the bin)
// instead of the FP64 positions.
//
// Bound: issue slots and shared-memory wavefronts together (quadratic 128^3
// clustered: 28 warp instructions per particle, 60 % of the issue slots and of
// the shared-memory pipe at 14 warps per SM; 20 warps, tile (4, 4, 8), are no
// faster).  Measured against one lane (cubic: 4) per particle and stream, with
// up to 108 sums per lane: cubic 128^3 8 per cell 1.52 -> 0.85 ms, quadratic 256^3
// 8 per cell clustered 5.53 -> 5.33 ms, a batch of 24 small problems 2.16 -> 1.07
// ms.  The next step's entry is read before the current one is used (quadratic
// 5.80 -> 5.35 ms, cubic 0.95 -> 0.85 ms).  Not kept: the streams that move found
// one by one (5.50 ms instead of testing each); packed FP32 pairs, whose
// coefficients need more shared-memory reads than they save instructions.
template <int ORDER, bool REC = false, bool STAG = false>
__device__ void p2g_item(const P2GArgs& A, int64_t t, int64_t a, int64_t b, float* warp_smem)
{
    using C = P2GCfg<ORDER, STAG>;
    constexpr int K = C::K, KK = C::KK, NV = C::NV, NF = C::NF, S = C::S, B = C::B;
    const MeshP& mp = A.mp;
    const TileP& tp = A.tp;
    const int lane = threadIdx.x & 31;
    float* table = warp_smem;
    float* wrow = warp_smem + C::TABLE;
    float* tile = warp_smem + C::TILE_OFF;

    int ob[3], i_lo, i_hi;
    tile_origin(tp, t, ob);
    p2g_rows<ORDER, REC>(A, t, a, b, ob, i_lo, i_hi);

    for (int i = lane; i < NF * tp.P / 2; i += 32)
        reinterpret_cast<float2*>(tile)[i] = make_float2(0.f, 0.f);
    const float D = (ORDER >= 2) ? inertial_scaling<ORDER, float>(mp.dx[0]) : 1.f;
    const float Dh = D * (float)mp.dx[0];

    // the lane as evaluator: slot es of stream eg
    const int U = (int)((b - a + S - 1) / S);  // particles per stream
    const int eg = lane / B, es = lane - eg * B;
    const int64_t p_first = a + (int64_t)eg * U;
    const int ecnt = eg < S ? (int)max((int64_t)0, min(p_first + U, b) - p_first) : 0;
    // its next particle, read one table ahead
    float4 nc[3], nrec = make_float4(0.f, 0.f, 0.f, 0.f);
    double nx[3] = {0.0, 0.0, 0.0};
    float nm = 0.f;
    auto fetch = [&](int s0) {
        if (s0 + es < ecnt) {
            const int64_t p = p_first + s0 + es;
            if constexpr (REC) {
                nrec = __ldg(reinterpret_cast<const float4*>(A.rec) + p);
            } else {
#pragma unroll
                for (int d = 0; d < 3; ++d) nx[d] = __ldg(A.x + 3 * p + d);
            }
#pragma unroll
            for (int v = 0; v < 3; ++v) nc[v] = __ldg(reinterpret_cast<const float4*>(A.c) + 3 * p + v);
            nm = __ldg(A.m + p);
        }
    };
    auto evaluate = [&](int s0) {
        float* e = table + eg * C::SE + es * C::ENTRY;
        float out[C::ENTRY], wxy[C::WROWS];
#pragma unroll
        for (int v = 0; v < C::ENTRY; ++v) out[v] = 0.f;
#pragma unroll
        for (int v = 0; v < C::WROWS; ++v) wxy[v] = 0.f;
        int at = -1;
        if (s0 + es < ecnt) {
            Spline1D<ORDER, float> sp[3];
            int lb[3];
            bool ok;
            if constexpr (REC) {
                ok = locate_record<ORDER>(mp, tp, t, nrec, sp, lb);
            } else {
                ok = locate<ORDER>(mp, tp, nx, ob, sp, lb);
            }
            // a particle out of the item's rows (the particles are not sorted)
            // is skipped like one of another tile
            ok = ok && lb[0] >= i_lo && lb[0] <= i_hi;
            if (!ok) {
                if (A.err) atomicAdd(A.err, 1);
            } else {
                at = lb[0] * tp.SI + lb[1] * tp.SJ + lb[2];
                // c_p(r, d) is element 3 r + d
                const float cp[12] = {nc[0].x, nc[0].y, nc[0].z, nc[0].w, nc[1].x, nc[1].y,
                                      nc[1].z, nc[1].w, nc[2].x, nc[2].y, nc[2].z, nc[2].w};
#pragma unroll
                for (int f = 0; f < NV; ++f) {
                    const int d = STAG ? A.stag : f;
                    float v[4];
#pragma unroll
                    for (int r = 0; r < 4; ++r)
                        v[r] = d == 0 ? cp[3 * r] : (d == 1 ? cp[3 * r + 1] : cp[3 * r + 2]);
                    if constexpr (ORDER >= 2) {
                        const float bd =
                            fmaf(v[3], sp[2].d[1], fmaf(v[2], sp[1].d[1], v[1] * sp[0].d[1]));
                        out[4 * f] = fmaf(D, bd, v[0]);
#pragma unroll
                        for (int r = 1; r < 4; ++r) out[4 * f + r] = Dh * v[r];
                    } else {
                        out[4 * f] = v[0] * nm;
#pragma unroll
                        for (int r = 1; r < 4; ++r) out[4 * f + r] = v[r] * nm * (float)mp.rdx[r - 1];
                    }
                }
#pragma unroll
                for (int k = 0; k < K; ++k) out[C::WZ + k] = sp[2].w[k];
                if constexpr (ORDER == 1) {
                    out[C::WZ + K] = nm;
#pragma unroll
                    for (int k = 0; k < K; ++k) {
                        wxy[k] = sp[0].w[k];
                        wxy[K + k] = sp[1].w[k];
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < K; ++i) {
                        const float wx = sp[0].w[i] * nm;
#pragma unroll
                        for (int j = 0; j < K; ++j) wxy[i * K + j] = wx * sp[1].w[j];
                    }
                }
            }
        }
        out[C::AT] = __int_as_float(at);
#pragma unroll
        for (int v = 0; v < (C::AT + 4) / 4; ++v)
            reinterpret_cast<float4*>(e)[v] =
                make_float4(out[4 * v], out[4 * v + 1], out[4 * v + 2], out[4 * v + 3]);
#pragma unroll
        for (int v = 0; v < C::WROWS; ++v) wrow[v * C::WROW + lane] = wxy[v];
    };

    // the lane as k-row (ri, rj) of stream g
    const bool act = lane < S * KK;
    const int g = act ? lane / KK : 0, row = act ? lane - g * KK : 0;
    const int ri = row / K, rj = row - ri * K;
    const float oi = (float)(ri - 1), oj = (float)(rj - 1);
    float* trow = tile + NF * (ri * tp.SI + rj * tp.SJ);
    float acc[NF][K];
#pragma unroll
    for (int f = 0; f < NF; ++f)
#pragma unroll
        for (int k = 0; k < K; ++k) acc[f][k] = 0.f;
    int cur = -1;  // tile offset of the sums' stencil
    auto add_node = [&](int k) {
        if constexpr (NF == 4) {
            float4* d = reinterpret_cast<float4*>(trow + 4 * (cur + k));
            const float4 v = *d;
            *d = make_float4(v.x + acc[0][k], v.y + acc[1][k], v.z + acc[NF - 2][k], v.w + acc[NF - 1][k]);
        } else {
            float2* d = reinterpret_cast<float2*>(trow + 2 * (cur + k));
            const float2 v = *d;
            *d = make_float2(v.x + acc[0][k], v.y + acc[1][k]);
        }
    };
    // The lanes whose stream moves (mine; step: by one node along k) add their
    // finished nodes to the tile, stream after stream; `moved`: ballot of mine.
    auto merge = [&](unsigned moved, bool mine, bool step) {
#pragma unroll
        for (int q = 0; q < S; ++q) {
            if (!((moved >> (q * KK)) & 1u)) continue;
            if (mine && g == q) {
                add_node(0);
                if (!step) {
#pragma unroll
                    for (int k = 1; k < K; ++k) add_node(k);
                }
            }
            __syncwarp();
        }
        if (mine) {
#pragma unroll
            for (int f = 0; f < NF; ++f)
#pragma unroll
                for (int k = 0; k < K; ++k)
                    acc[f][k] = step && k + 1 < K ? acc[f][k + 1 < K ? k + 1 : k] : 0.f;
        }
    };

    // A stream that stays in one stencil hands its sums to the tile every 60 to 64 steps,
    // so that no FP32 sum is a chain of more than 128 particles, however crowded a cell
    // and long an item (4096 equal masses in one cell: error 1.8e-5, with it 2e-6).
    constexpr int kTables = 64 / B;
    int tables = 0, was = -1;  // tables since the last look, the stencil then

    fetch(0);
    for (int s0 = 0; s0 < U; s0 += B) {
        if (tables == kTables) {
            const bool stayed = cur >= 0 && cur == was;
            const unsigned all = __ballot_sync(kFull, stayed);
            if (all) merge(all, stayed, false);
            was = cur;
            tables = 0;
        }
        ++tables;
        __syncwarp();  // the table has been read
        evaluate(s0);
        __syncwarp();
        fetch(s0 + B);
        const int steps = min(B, U - s0);
        const float* e = table + g * C::SE;
        const float* w = wrow + g * B;
        // a particle's entry as the lane reads it, one step ahead of its use
        // (past the last step: the words after the entries, not used)
        struct Entry {
            float4 v[NV];
            float wz[K], wa, wb;  // wa: w_x w_y m of the k-row (linear: w_x; wb: w_y), m
            float m;
            int at;
        };
        auto read = [&](int q) {
            Entry r;
            const float* p = e + q * C::ENTRY;
#pragma unroll
            for (int f = 0; f < NV; ++f) r.v[f] = *reinterpret_cast<const float4*>(p + 4 * f);
            const float4 z = *reinterpret_cast<const float4*>(p + C::WZ);
            const float zz[4] = {z.x, z.y, z.z, z.w};
#pragma unroll
            for (int k = 0; k < K; ++k) r.wz[k] = zz[k];
            const int at = __float_as_int(K < 4 ? z.w : p[C::AT]);
            r.at = act ? at : -1;
            r.m = ORDER == 1 ? z.z : 0.f;
            r.wa = ORDER == 1 ? w[ri * C::WROW + q] : w[row * C::WROW + q];
            r.wb = ORDER == 1 ? w[(K + rj) * C::WROW + q] : 0.f;
            return r;
        };
        Entry next = read(0);
#pragma unroll 2
        for (int q = 0; q < steps; ++q) {
            const Entry r = next;
            next = read(q + 1);
            const bool mine = r.at >= 0 && cur >= 0 && r.at != cur;
            const unsigned moved = __ballot_sync(kFull, mine);
            if (moved) merge(moved, mine, r.at == cur + 1);
            if (r.at >= 0) cur = r.at;
            if constexpr (ORDER == 1) {
                const float wx = r.wa, wy = r.wb;
                const float wab = wx * wy, mab = r.m * wab;
                const float sx = ri ? wy : -wy, sy = rj ? wx : -wx;
                acc[0][0] = fmaf(mab, r.wz[0], acc[0][0]);
                acc[0][1] = fmaf(mab, r.wz[1], acc[0][1]);
#pragma unroll
                for (int f = 0; f < NV; ++f) {
                    const float p = fmaf(r.v[f].z, sy, fmaf(r.v[f].y, sx, r.v[f].x * wab));
                    const float c = r.v[f].w * wab;
                    acc[1 + f][0] += fmaf(p, r.wz[0], -c);
                    acc[1 + f][1] += fmaf(p, r.wz[1], c);
                }
            } else {
                float wn[K];
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    wn[k] = r.wa * r.wz[k];
                    acc[0][k] += wn[k];
                }
#pragma unroll
                for (int f = 0; f < NV; ++f) {
                    const float p = fmaf(oj, r.v[f].z, fmaf(oi, r.v[f].y, r.v[f].x));
#pragma unroll
                    for (int k = 0; k < K; ++k)
                        acc[1 + f][k] = fmaf(wn[k], add_steps(k - 1, p, r.v[f].w), acc[1 + f][k]);
                }
            }
        }
    }
    const unsigned last = __ballot_sync(kFull, cur >= 0);
    if (last) merge(last, cur >= 0, false);
    auto values = [&](int idx, float (&x)[NF]) {
        if constexpr (NF == 4) {
            const float4 v = reinterpret_cast<const float4*>(tile)[idx];
            x[0] = v.x, x[1] = v.y, x[NF - 2] = v.z, x[NF - 1] = v.w;
        } else {
            const float2 v = reinterpret_cast<const float2*>(tile)[idx];
            x[0] = v.x, x[1] = v.y;
        }
    };
    flush_tile<ORDER, NF>(A, values, last != 0, i_lo, i_hi, ob, warp_smem, C::TILE_OFF / 8, lane);
    __syncwarp();
}

// ---------------------------------------------------------------------------
// P2G with the grid update in its flush
// ---------------------------------------------------------------------------
// A node's value is final once every work item that can touch it has added
// its tile box.  Every node belongs to the tile of the bin with its index
// (for a non-periodic mesh the last tile along a dimension also takes the
// K - 1 nodes past the last bin), and a tile's nodes form 8 regions by
// whether each local index is below K - 1: those nodes are also touched by
// the items of the previous tile along that dimension, the others only by
// the tile's own items (tiles of at least K - 1 bins).  An item that has
// flushed counts its arrival at every region it can touch (27: the tile and
// its successors along each dimension, their low parts); the item whose
// arrival completes a region's count (the items of the up to 8 tiles that
// touch it) converts the region's nodes with the grid update.  The
// accumulators are exact integer sums, so the conversion sees the same
// values as a separate update pass after P2G: results are bit-identical.
struct FusedUpdate {
    GridUpdate P;
    GField gf, gu, gu64;  // force (optional, FP64), velocity, FP64 velocity (optional)
    uint32_t* count;      // 8 arrival counters per tile, zero at launch
};

// Local node range [lo, hi) of the region part `low` of tile q along d.
__device__ __forceinline__ void region_range(const TileP& tp, int d, int q, int low, int K, int& lo,
                                             int& hi)
{
    lo = low ? 0 : K - 1;
    hi = low ? K - 1 : min(tp.T[d], tp.nb[d] - q * tp.T[d]);
}

__device__ __forceinline__ uint32_t tile_items_of(const TileP& tp, int64_t s)
{
    return (__ldg(tp.items + s + 1) - __ldg(tp.items + s)) * (uint32_t)tp.split;
}

// Items of the tiles that touch region `reg` of tile (q0, q1, q2).
__device__ __forceinline__ uint32_t region_items(const MeshP& mp, const TileP& tp, const int q[3],
                                                 int reg)
{
    uint32_t expected = 0;
    for (int mm = 0; mm < 8; ++mm) {
        if (mm & ~reg) continue;
        int pp[3];
        bool ok = true;
        for (int d = 0; d < 3; ++d) {
            pp[d] = q[d] - ((mm >> d) & 1);
            if (pp[d] < 0) {
                if (mp.periodic[d]) pp[d] += tp.nt[d];
                else ok = false;
            }
        }
        if (ok) expected += tile_items_of(tp, ((int64_t)pp[0] * tp.nt[1] + pp[1]) * tp.nt[2] + pp[2]);
    }
    return expected;
}

// Global node of local index g[d] in tile q along d.
__device__ __forceinline__ void region_node(const MeshP& mp, const TileP& tp, const int q[3],
                                            int g[3])
{
    for (int d = 0; d < 3; ++d) {
        g[d] += q[d] * tp.T[d];
        if (mp.periodic[d]) g[d] += mp.own_lo[d];
    }
}

// Called by the whole warp after p2g_item(A, t, ...) has flushed its box.
template <int ORDER>
__device__ void fused_update_arrive(const P2GArgs& A, const FusedUpdate& F, int64_t t)
{
    constexpr int K = SplineTraits<ORDER>::K;
    const MeshP& mp = A.mp;
    const TileP& tp = A.tp;
    const int lane = threadIdx.x & 31;
    __threadfence();  // this lane's reductions are visible before its item counts
    __syncwarp();
    const int q[3] = {(int)(t / ((int64_t)tp.nt[1] * tp.nt[2])),
                      (int)((t / tp.nt[2]) % tp.nt[1]), (int)(t % tp.nt[2])};
    bool last = false;
    int64_t tt = 0;
    int reg = 0;
    if (lane < 27) {
        // per dimension: 0 = this tile, high part; 1 = this tile, low part;
        // 2 = the next tile, low part
        const int o[3] = {lane / 9, (lane / 3) % 3, lane % 3};
        int qq[3];
        bool exists = true;
        for (int d = 0; d < 3; ++d) {
            qq[d] = q[d] + (o[d] == 2);
            if (qq[d] >= tp.nt[d]) {
                if (mp.periodic[d]) qq[d] = 0;
                else exists = false;
            }
            reg |= (o[d] >= 1) << d;
        }
        if (exists) {
            tt = ((int64_t)qq[0] * tp.nt[1] + qq[1]) * tp.nt[2] + qq[2];
            // the items of the tiles that touch the region: qq and, along
            // the region's low dimensions, the previous tile
            const uint32_t expected = region_items(mp, tp, qq, reg);
            const uint32_t old = atomicAdd(F.count + tt * 8 + reg, 1u);
            last = old + 1 == expected;
        }
    }
    unsigned lm = __ballot_sync(kFull, last);
    while (lm) {
        const int src = __ffs(lm) - 1;
        lm &= lm - 1;
        const int64_t ct = __shfl_sync(kFull, tt, src);
        const int cr = __shfl_sync(kFull, reg, src);
        __threadfence();  // every arrival counted: their reductions are visible
        const int cq[3] = {(int)(ct / ((int64_t)tp.nt[1] * tp.nt[2])),
                           (int)((ct / tp.nt[2]) % tp.nt[1]), (int)(ct % tp.nt[2])};
        int lo[3], hi[3];
        for (int d = 0; d < 3; ++d) region_range(tp, d, cq[d], (cr >> d) & 1, K, lo[d], hi[d]);
        const int n1 = hi[1] - lo[1], n2 = hi[2] - lo[2];
        const int total = (hi[0] - lo[0]) * n1 * n2;
        for (int e = lane; e < total; e += 32) {
            int g[3] = {lo[0] + e / (n1 * n2), lo[1] + (e / n2) % n1, lo[2] + e % n2};
            region_node(mp, tp, cq, g);
            update_node<long long, double, float, true>(F.P, A.gm, A.gmu, F.gf, F.gu, F.gu64,
                                                        g[0], g[1], g[2]);
        }
    }
}

// Regions no work item touches are converted by no item: one thread per
// (tile, region) writes them the update of an empty node, 0.
template <int ORDER>
__global__ void zero_untouched_regions_kernel(MeshP mp, TileP tp, FusedUpdate F)
{
    constexpr int K = SplineTraits<ORDER>::K;
    const int64_t total = tp.ntiles * 8;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < total;
         r += (int64_t)gridDim.x * blockDim.x) {
        const int64_t t = r / 8;
        const int reg = (int)(r % 8);
        const int q[3] = {(int)(t / ((int64_t)tp.nt[1] * tp.nt[2])),
                          (int)((t / tp.nt[2]) % tp.nt[1]), (int)(t % tp.nt[2])};
        if (region_items(mp, tp, q, reg) != 0) continue;
        int lo[3], hi[3];
        for (int d = 0; d < 3; ++d) region_range(tp, d, q[d], (reg >> d) & 1, K, lo[d], hi[d]);
        for (int i = lo[0]; i < hi[0]; ++i)
            for (int j = lo[1]; j < hi[1]; ++j)
                for (int k = lo[2]; k < hi[2]; ++k) {
                    int g[3] = {i, j, k};
                    region_node(mp, tp, q, g);
                    for (int c = 0; c < 3; ++c) {
                        *F.gu.ptr<float>(g[0], g[1], g[2], c) = 0.f;
                        if (F.gu64.data) *F.gu64.ptr<double>(g[0], g[1], g[2], c) = 0.0;
                    }
                }
    }
}

// ---------------------------------------------------------------------------
// G2P
// ---------------------------------------------------------------------------
// Term n of the sum of w_n v_n: the first one sets it.
__device__ __forceinline__ float add_term(int n, float w, float v, float sum)
{
    return n == 0 ? __fmul_rn(w, v) : fmaf(w, v, sum);
}

// Term n of S0 = sum w_n v_n and S1 = sum (n - n0) w_n v_n, n0 the stencil's centre
// knot (0 linear, else 1), in few instructions: 3 (linear), 4 (quadratic) and 6 (cubic)
// for all terms.  (Linear: the product twice, once in the sum's FMA, as the velocities
// that advected positions follow have always been rounded; run_sums in tiled.cu.)
template <int ORDER>
__device__ __forceinline__ void add_moments(int n, float w, float v, float& S0, float& S1)
{
    if constexpr (ORDER == 1) {
        if (n == 0) {
            S0 = __fmul_rn(w, v);
        } else {
            S1 = __fmul_rn(w, v);
            S0 = fmaf(w, v, S0);
        }
    } else {
        if (n == 0) {
            S0 = __fmul_rn(w, v);
            return;
        }
        if (n == 2) S1 = fmaf(w, v, -S1);
        if (n == 1) S1 = S0;  // the first term, to be subtracted
        if (n == 3) S1 = fmaf(2.f * w, v, S1);
        S0 = fmaf(w, v, S0);
    }
}

// One G2P work item by NTHR threads (a warp or a CTA) sharing `tile`
// (tp.nodes float4).  Threads are numbered tid in [0, NTHR).
// Bound by the instructions of the contraction together with its 16-byte reads of
// shared memory (quadratic, 128^3 cells 8 per cell clustered: 66 % of the issue slots
// and 73 % of the L1 data pipe of a busy SM, 390 instructions and 78 shared-memory
// wavefronts per 32 particles; DRAM at 42 %).  Taking the moments in fused
// multiply-adds (add_moments), walking the rows by one pointer and staging the tile
// without divisions took 440 instructions to 390: 256^3 2.16 -> 2.06 ms, 128^3 0.326
// -> 0.301 ms, cubic with advection 128^3 0.66 -> 0.635 ms.  More warps at fewer
// registers lose more to spills (64 instead of 72: 2.51 ms).
// ADV: each particle is then moved, x += dt u_p (FP64, as picasso_advect).
// The positions of the item's first and last particle are read before the
// tile barrier, so no thread reads a position another thread has moved.
// REC: the particles' splines come from their records (not with ADV).
// STAG: a staggered location (APIC.hpp:477-544): the grid field is the scalar
// velocity component of the entity's dimension, which lands in column `stag`
// of c_p (the other columns are written as zero, as the plain kernel does).
template <int ORDER, int NTHR, bool ADV = false, bool REC = false, bool STAG = false>
__device__ void g2p_item(const G2PArgs& A, int64_t t, int64_t a, int64_t b, float4* tile,
                         int tid)
{
    static_assert(!(ADV && REC), "the advection reads the FP64 positions");
    static_assert(!(ADV && STAG), "the advection moves by the 3-component velocity");
    constexpr int NU = STAG ? 1 : 3;  // velocity components gathered
    constexpr int K = SplineTraits<ORDER>::K;
    constexpr int N0 = ORDER == 1 ? 0 : 1;  // centre knot of the stencil
    const MeshP& mp = A.mp;
    const TileP& tp = A.tp;
    auto sync = [] {
        if (NTHR == 32) __syncwarp();
        else __syncthreads();
    };
    int ob[3];
    tile_origin(tp, t, ob);
    // bin rows spanned by the item: the first and last particle bound the
    // slowest tile dimension (keys are i-major within a tile)
    int i_lo = 0, i_hi = tp.T[0] - 1;
    if constexpr (REC) {
        int la[3], lz[3];
        const bool oka = bin_of_key(tp, t, __float_as_uint(__ldg(&A.rec[a].w)), la);
        const bool okb = bin_of_key(tp, t, __float_as_uint(__ldg(&A.rec[b - 1].w)), lz);
        if (oka && okb && lz[0] >= la[0]) {
            i_lo = la[0];
            i_hi = lz[0];
        }
    } else {
        Spline1D<ORDER, float> sp[3];
        int lb[3];
        const double xa[3] = {A.x[3 * a], A.x[3 * a + 1], A.x[3 * a + 2]};
        const double xb[3] = {A.x[3 * (b - 1)], A.x[3 * (b - 1) + 1], A.x[3 * (b - 1) + 2]};
        const bool oka = locate<ORDER>(mp, tp, xa, ob, sp, lb);
        const int la = lb[0];
        const bool okb = locate<ORDER>(mp, tp, xb, ob, sp, lb);
        if (oka && okb && lb[0] >= la) {
            i_lo = la;
            i_hi = lb[0];
        }
    }
    const int plane = tp.NT[1] * tp.NT[2];
    const int total = (i_hi - i_lo + K) * plane;
    sync();  // the previous item's threads are done with the tile
    // node e = tid, tid + NTHR, ...: (i, j, k) by carries, not by divisions
    const int step_k = NTHR % tp.NT[2], step_j = NTHR / tp.NT[2] % tp.NT[1], step_i = NTHR / plane;
    int k = tid % tp.NT[2], j = tid / tp.NT[2] % tp.NT[1], i = i_lo + tid / plane;
    for (int e = tid; e < total; e += NTHR) {
        const int gi = node_global(mp, tp, 0, ob[0], i);
        const int gj = node_global(mp, tp, 1, ob[1], j);
        const int gk = node_global(mp, tp, 2, ob[2], k);
        const bool inside = (mp.periodic[0] || gi < mp.ext[0]) &&
                            (mp.periodic[1] || gj < mp.ext[1]) &&
                            (mp.periodic[2] || gk < mp.ext[2]);
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (inside) {  // through L2: the batched kernel writes u_i in the same launch
            int gx;
            const float* ub =
                reinterpret_cast<const float*>(halo_route(A.hp, 0, A.u.data, gi, gx));
            v.x = __ldcg(ub + A.u.index(gx, gj, gk, 0));
            if (!STAG) {
                v.y = __ldcg(ub + A.u.index(gx, gj, gk, 1));
                v.z = __ldcg(ub + A.u.index(gx, gj, gk, 2));
            }
        }
        tile[i_lo * plane + e] = v;
        k += step_k;
        j += step_j;
        i += step_i;
        if (k >= tp.NT[2]) {
            k -= tp.NT[2];
            ++j;
        }
        if (j >= tp.NT[1]) {
            j -= tp.NT[1];
            ++i;
        }
    }
    sync();
    // positions (records) are prefetched one particle ahead
    double xn[3] = {0.0, 0.0, 0.0};
    float4 rn = make_float4(0.f, 0.f, 0.f, 0.f);
    if (a + tid < b) {
        const int64_t p0 = a + tid;
        if constexpr (REC) {
            rn = __ldg(A.rec + p0);
        } else {
            xn[0] = A.x[3 * p0];
            xn[1] = A.x[3 * p0 + 1];
            xn[2] = A.x[3 * p0 + 2];
        }
    }
    for (int64_t p = a + tid; p < b; p += NTHR) {
        const double xp[3] = {xn[0], xn[1], xn[2]};
        const float4 rp = rn;
        const int64_t pn = p + NTHR;
        if (pn < b) {
            if constexpr (REC) {
                rn = __ldg(A.rec + pn);
            } else {
                xn[0] = A.x[3 * pn];
                xn[1] = A.x[3 * pn + 1];
                xn[2] = A.x[3 * pn + 2];
            }
        }
        Spline1D<ORDER, float> sp[3];
        int lb[3];
        bool ok;
        if constexpr (REC) ok = locate_record<ORDER>(mp, tp, t, rp, sp, lb);
        else ok = locate<ORDER>(mp, tp, xp, ob, sp, lb);
        if (!ok || lb[0] < i_lo || lb[0] > i_hi) {
            if (A.err) atomicAdd(A.err, 1);
            continue;
        }
        const int base = (lb[0] * tp.NT[1] + lb[1]) * tp.NT[2] + lb[2];
        // APIC.hpp:439-461, contracted one dimension at a time, with the
        // distances relative to the centre knot n0 (dist_q(n) = dist_q(n0)
        // + (n_q - n0) dx):
        //   u_p      = sum_i wx_i sum_j wy_j sum_k wz_k u_ijk
        //   M_q      = sum_ijk w_ijk u_ijk (n_q - n0)
        //   B_p(:,q) = dx M_q + dist_q(n0) u_p
        float up[3] = {0.f, 0.f, 0.f};
        float M[3][3] = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
        const float4* row = tile + base;
#pragma unroll
        for (int i = 0; i < K; ++i) {
            float A0[3], A1[3], A2[3];
#pragma unroll
            for (int j = 0; j < K; ++j) {
                float S0[3], S1[3];
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    const float4 ue = row[k];
                    const float uk[3] = {ue.x, ue.y, ue.z};
#pragma unroll
                    for (int d = 0; d < NU; ++d) {
                        add_moments<ORDER>(k, sp[2].w[k], uk[d], S0[d], S1[d]);
                    }
                }
#pragma unroll
                for (int d = 0; d < NU; ++d) {
                    add_moments<ORDER>(j, sp[1].w[j], S0[d], A0[d], A1[d]);
                    A2[d] = add_term(j, sp[1].w[j], S1[d], A2[d]);
                }
                row += j + 1 < K ? tp.NT[2] : plane - (K - 1) * tp.NT[2];
            }
#pragma unroll
            for (int d = 0; d < NU; ++d) {
                add_moments<ORDER>(i, sp[0].w[i], A0[d], up[d], M[d][0]);
                M[d][1] = add_term(i, sp[0].w[i], A1[d], M[d][1]);
                M[d][2] = add_term(i, sp[0].w[i], A2[d], M[d][2]);
            }
        }
        float B[3][3];
#pragma unroll
        for (int d = 0; d < NU; ++d)
#pragma unroll
            for (int q = 0; q < 3; ++q)
                B[d][q] = fmaf((float)mp.dx[q], M[d][q], sp[q].d[N0] * up[d]);
        if constexpr (STAG) {
            // the gathered component belongs to column stag; the others are 0
            const float u0 = up[0], b0[3] = {B[0][0], B[0][1], B[0][2]};
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const bool mine = d == A.stag;
                up[d] = mine ? u0 : 0.f;
#pragma unroll
                for (int q = 0; q < 3; ++q) B[d][q] = mine ? b0[q] : 0.f;
            }
        }
        // c_p(0, d) = u_p(d); c_p(1 + q, d) = B_p(d, q)  (APIC.hpp:464-471)
        float4* out = reinterpret_cast<float4*>(A.c + 12 * p);
        out[0] = make_float4(up[0], up[1], up[2], B[0][0]);
        out[1] = make_float4(B[1][0], B[2][0], B[0][1], B[1][1]);
        out[2] = make_float4(B[2][1], B[0][2], B[1][2], B[2][2]);
        if constexpr (ADV) {
            const double uo[3] = {(double)up[0], (double)up[1], (double)up[2]};
            advect_particle(A.adv, p, xp, uo, [&](int d, double v) { A.x_out[3 * p + d] = v; });
        }
    }
}

// host helpers (tiled.cu)
bool fused_update_fits(const TileP& tp, int order);
// What a tile is made for: `streams` and `runs` set the strides of the P2G's node tile
// (p2g_item, run_p2g_item); a batch's items are cut by a rule of their own, those of
// `whole` and `runs` not at all (set_parts).
enum class TileUse { other, whole, streams, runs, batch_other, batch_streams };
bool make_tilep(const MeshP& mp, int order, const picasso_bins& bins, int64_t n, TileP* tp,
                TileUse use = TileUse::other);
int64_t item_bound(const TileP& tp);  // parts of all items, at most
int device_smem_optin();
bool packed_x(const PField& x);
bool packed_m(const PField& m);
bool packed_c(const PField& c);
bool valid_lanes(int order, int lanes, bool stag = false);
size_t p2g_warp_bytes(int order, int P, bool stag = false);
// Tiled kernels of a call (tiled.cu); *handled stays false where they do not take it.
// batched: an instance's items as the batched launches cut them (set_parts).
picasso_status apic_p2g_tiled(const MeshP& mp, int order, int ncomp, Form form, int64_t n,
                              const PField& x, const PField& m, const PField& c, const GField& gm,
                              const GField& gmu, const picasso_bins& bins, int* err,
                              cudaStream_t st, bool* handled, const FusedUpdate* fu = nullptr,
                              int stag = -1, const HaloPeers* hp = nullptr, bool batched = false);
picasso_status apic_g2p_tiled(const MeshP& mp, int order, int ncomp, bool f32, int64_t n,
                              const PField& x, const GField& u, const PField& c,
                              const picasso_bins& bins, int* err, const Advect* adv,
                              cudaStream_t st, bool* handled, int stag = -1,
                              const HaloPeers* hp = nullptr);

}  // namespace pb
