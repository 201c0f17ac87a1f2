// FP32 tiled P2G in runs: the P2G of linear splines and of sparse and of large dense
// quadratic sets (run_sums in tiled.cu says where and why; the other sets take the
// streams of p2g_item in tiled.cuh).
//
// A work item's sorted particles are cut into 32 contiguous runs, one per lane.
// Consecutive particles of a run mostly share a stencil, whose sums (4 fields x K^3
// nodes) the lane keeps in registers; particle records arrive through a cp.async ring
// a few particles ahead of use.  When a run's bin changes the lane stages its sums and
// the warp adds the staged values into its FP32 node tile, one staged lane after the
// other: a fixed order without atomics.  The tile then leaves as that of p2g_item.
//
// Bound: the serial merges of a warp at 8 warps per SM (255 registers).  1 per cell,
// linear 2 M particles 0.174 ms, quadratic 0.324 ms (streams: 0.162 and 0.203 ms).
#pragma once

#include "tiled.cuh"

namespace pb {

// Single-warp CTAs per SM the register budget is sized for: 4 x K^3 sums per lane.
constexpr int kRunOccupancy = 8;

template <int ORDER, bool REC>
struct RunCfg {
    static constexpr int K = SplineTraits<ORDER>::K;
    static constexpr int KK = K * K, KKK = K * K * K;
    static constexpr int F = 4;                  // grid fields
    static constexpr int N0 = 1;                 // centre knot of the quadratic stencil
    static constexpr int FS = (KKK + 3) & ~3;    // staged floats per field
    static constexpr int SV = F * FS;            // staged values per lane
    // Staging stride: a multiple of 4 floats whose quarter is odd keeps the 16-byte
    // stores of 8 lanes on distinct banks.
    static constexpr int odd_quarter(int v) { return (v / 4) % 2 == 0 ? v + 4 : v; }
    static constexpr int SS = odd_quarter(SV);
    static constexpr int R = (SV + 31) / 32;     // merge rounds per staged lane
    // merges of one k-plane (the bin moved by one along k): K^2 nodes, packed
    static constexpr int PV = F * KK;
    static constexpr int PS = odd_quarter((PV + 3) & ~3);
    static constexpr int RP = (PV + 31) / 32;
    static constexpr int LANES = 8;              // lanes staged per round of full merges
    // ring per stage: position (3 doubles, or one 16-byte record) | c (12) | m (1)
    static constexpr int XS = REC ? 4 : 6;
    static constexpr int RING_C = XS * 32, RING_M = (XS + 12) * 32, RING = (XS + 13) * 32;
    static constexpr int DEPTH = 4;
    static constexpr int STAGE_OFF = DEPTH * RING;
    static constexpr int STAGE = 32 * PS > LANES * SS ? 32 * PS : LANES * SS;
    static constexpr int TILE_OFF = STAGE_OFF + STAGE;  // F planes of P floats
};

template <int ORDER, bool REC>
__host__ __device__ constexpr int run_warp_floats(int P)
{
    return RunCfg<ORDER, REC>::TILE_OFF + RunCfg<ORDER, REC>::F * P;
}

template <int BYTES>
__device__ __forceinline__ void cp_async(void* dst, const void* src)
{
    if constexpr (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_addr(dst)), "l"(src));
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(smem_addr(dst)), "l"(src),
                     "n"(BYTES));
}

// A lane's sums of its run's current stencil.
template <int ORDER>
struct RunSums {
    using C = RunCfg<ORDER, false>;
    static constexpr int K = C::K;
    float acc[C::F][C::KKK];

    __device__ __forceinline__ void zero()
    {
#pragma unroll
        for (int f = 0; f < C::F; ++f)
#pragma unroll
            for (int n = 0; n < C::KKK; ++n) acc[f][n] = 0.f;
    }

    // Quadratic: cp[3 r + d] = c_p(r, d), in the centre-knot form of p2g_item.
    __device__ __forceinline__ void add_quadratic(const Spline1D<ORDER, float> sp[3], float mass,
                                                  const float cp[12], float D, float Dh)
    {
        float E[C::F], G[C::F][3];
#pragma unroll
        for (int f = 1; f < C::F; ++f) {
            const float bx = cp[2 + f], by = cp[5 + f], bz = cp[8 + f];
            const float bd =
                fmaf(bz, sp[2].d[C::N0], fmaf(by, sp[1].d[C::N0], bx * sp[0].d[C::N0]));
            E[f] = fmaf(D, bd, cp[f - 1]);
            G[f][0] = Dh * bx;
            G[f][1] = Dh * by;
            G[f][2] = Dh * bz;
        }
#pragma unroll
        for (int i = 0; i < K; ++i) {
            const float wi = sp[0].w[i] * mass;
            float pi[C::F];
#pragma unroll
            for (int f = 1; f < C::F; ++f) pi[f] = add_steps(i - C::N0, E[f], G[f][0]);
#pragma unroll
            for (int j = 0; j < K; ++j) {
                const float wij = wi * sp[1].w[j];
                float pij[C::F];
#pragma unroll
                for (int f = 1; f < C::F; ++f) pij[f] = add_steps(j - C::N0, pi[f], G[f][1]);
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    const int n = (i * K + j) * K + k;
                    const float w = wij * sp[2].w[k];
                    acc[0][n] += w;
#pragma unroll
                    for (int f = 1; f < C::F; ++f)
                        acc[f][n] = fmaf(w, add_steps(k - C::N0, pij[f], G[f][2]), acc[f][n]);
                }
            }
        }
    }

    // Linear, gradient form (APIC.hpp:287-318).
    __device__ __forceinline__ void add_linear(const Spline1D<ORDER, float> sp[3], float mass,
                                               const float cp[12])
    {
#pragma unroll
        for (int i = 0; i < K; ++i)
#pragma unroll
            for (int j = 0; j < K; ++j)
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    const int n = (i * K + j) * K + k;
                    const float www = sp[0].w[i] * sp[1].w[j] * sp[2].w[k] * mass;
                    const float gww = sp[0].g[i] * sp[1].w[j] * sp[2].w[k] * mass;
                    const float wgw = sp[0].w[i] * sp[1].g[j] * sp[2].w[k] * mass;
                    const float wwg = sp[0].w[i] * sp[1].w[j] * sp[2].g[k] * mass;
                    acc[0][n] += www;
#pragma unroll
                    for (int f = 1; f < C::F; ++f)
                        acc[f][n] += cp[f - 1] * www + cp[2 + f] * gww + cp[5 + f] * wgw +
                                     cp[8 + f] * wwg;
                }
    }

    // st[f FS + n] <- acc[f][n] with 16-byte stores.
    __device__ __forceinline__ void stage(float* st) const
    {
#pragma unroll
        for (int f = 0; f < C::F; ++f)
#pragma unroll
            for (int q = 0; q < C::FS / 4; ++q) {
                float v[4];
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    v[e] = 4 * q + e < C::KKK ? acc[f][4 * q + e < C::KKK ? 4 * q + e : 0] : 0.f;
                *reinterpret_cast<float4*>(st + f * C::FS + 4 * q) = make_float4(v[0], v[1], v[2], v[3]);
            }
    }

    // The first k-plane (st[f K^2 + row]) with 16-byte stores; the sums then move one
    // node down along k.
    __device__ __forceinline__ void stage_plane(float* st)
    {
#pragma unroll
        for (int q = 0; q < (C::PV + 3) / 4; ++q) {
            float v[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int s = 4 * q + e < C::PV ? 4 * q + e : 0;
                v[e] = 4 * q + e < C::PV ? acc[s / C::KK][(s % C::KK) * K] : 0.f;
            }
            *reinterpret_cast<float4*>(st + 4 * q) = make_float4(v[0], v[1], v[2], v[3]);
        }
#pragma unroll
        for (int f = 0; f < C::F; ++f)
#pragma unroll
            for (int ij = 0; ij < C::KK; ++ij) {
#pragma unroll
                for (int k = 0; k + 1 < K; ++k) acc[f][ij * K + k] = acc[f][ij * K + k + 1];
                acc[f][ij * K + K - 1] = 0.f;
            }
    }
};

// The warp adds staged values into the node tile: lane l adds value l + 32 r of each
// staged slot at tile offset base + off[r] (off < 0: none), slot after slot: slots
// 0 .. slots - 1 (MASK false) or the set bits of `slots`, lowest first (MASK true).
// The next slot's base and values are read before this slot's tile updates, so only
// the tile's read-add-write is on the chain.
template <int NR, int SLOT, bool MASK>
__device__ __forceinline__ void add_staged(unsigned slots, const float* stage, const int* base,
                                           const int (&off)[NR], float* tile, int lane)
{
    int q = MASK ? __ffs(slots) - 1 : 0;
    unsigned rest = MASK ? slots & (slots - 1u) : slots - 1u;  // MASK false: slots left
    int at = base[q];
    float v[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) v[r] = off[r] >= 0 ? stage[q * SLOT + lane + 32 * r] : 0.f;
    for (;;) {
        const int qn = rest ? (MASK ? __ffs(rest) - 1 : q + 1) : q;
        const int atn = base[qn];
        float vn[NR];
#pragma unroll
        for (int r = 0; r < NR; ++r) vn[r] = off[r] >= 0 ? stage[qn * SLOT + lane + 32 * r] : 0.f;
#pragma unroll
        for (int r = 0; r < NR; ++r)
            if (off[r] >= 0) tile[at + off[r]] += v[r];
        __syncwarp();
        if (!rest) break;
        rest = MASK ? rest & (rest - 1u) : rest - 1u;
        q = qn;
        at = atn;
#pragma unroll
        for (int r = 0; r < NR; ++r) v[r] = vn[r];
    }
}

// One P2G work item (tile t, particles [a, b)) by the calling warp, collocated.
// `smem` holds run_warp_floats<ORDER, REC>(P) floats (16-byte aligned), `base` 32 ints
// of shared memory.  REC: spline records instead of the positions.
template <int ORDER, bool REC>
__device__ void run_p2g_item(const P2GArgs& A, int64_t t, int64_t a, int64_t b, float* smem, int* base)
{
    using C = RunCfg<ORDER, REC>;
    constexpr int K = C::K;
    const MeshP& mp = A.mp;
    const TileP& tp = A.tp;
    const int lane = threadIdx.x & 31;
    float* stage = smem + C::STAGE_OFF;
    float* tile = smem + C::TILE_OFF;
    int ob[3], i_lo, i_hi;
    tile_origin(tp, t, ob);
    p2g_rows<ORDER, REC>(A, t, a, b, ob, i_lo, i_hi);
    const int U = (int)((b - a + 31) / 32);
    const int64_t my0 = a + (int64_t)lane * U;
    const int cnt = (int)max((int64_t)0, min(my0 + U, b) - my0);

    for (int i = lane; i < C::F * tp.P; i += 32) tile[i] = 0.f;
    // where value lane + 32 r of a staged lane, and of a staged k-plane, goes
    int off[C::R], poff[C::RP];
#pragma unroll
    for (int r = 0; r < C::R; ++r) {
        const int v = lane + 32 * r, f = v / C::FS, n = v - f * C::FS;
        off[r] = v < C::SV && n < C::KKK
                     ? f * tp.P + n / C::KK * tp.SI + n / K % K * tp.SJ + n % K : -1;
    }
#pragma unroll
    for (int r = 0; r < C::RP; ++r) {
        const int v = lane + 32 * r, f = v / C::KK, ij = v - f * C::KK;
        poff[r] = v < C::PV ? f * tp.P + ij / K * tp.SI + ij % K * tp.SJ : -1;
    }
    const float D = (ORDER >= 2) ? inertial_scaling<ORDER, float>(mp.dx[0]) : 1.f;
    const float Dh = D * (float)mp.dx[0];

    auto slot = [&](int q) { return smem + (q % C::DEPTH) * C::RING; };
    auto issue = [&](int q) {
        if (q < cnt) {
            const int64_t p = my0 + q;
            float* s = slot(q);
            if constexpr (REC) {
                cp_async<16>(s + lane * 4, A.rec + 4 * p);
            } else {
#pragma unroll
                for (int d = 0; d < 3; ++d) cp_async<8>(s + lane * 6 + 2 * d, A.x + 3 * p + d);
            }
#pragma unroll
            for (int v = 0; v < 3; ++v)
                cp_async<16>(s + C::RING_C + lane * 12 + 4 * v, A.c + 12 * p + 4 * v);
            cp_async<4>(s + C::RING_M + lane, A.m + p);
        }
        asm volatile("cp.async.commit_group;\n");
    };
#pragma unroll
    for (int q = 0; q < C::DEPTH - 1; ++q) issue(q);

    RunSums<ORDER> sums;
    sums.zero();
    int cur = -1, cur_base = 0;
    // The lanes of `mask` (whose bin moved by one along k) hand over their first
    // k-plane, all staged at once.
    auto merge_plane = [&](unsigned mask) {
        if ((mask >> lane) & 1u) sums.stage_plane(stage + lane * C::PS);
        base[lane] = cur_base;
        __syncwarp();
        add_staged<C::RP, C::PS, true>(mask, stage, base, poff, tile, lane);
    };
    // The lanes of `mask` hand over all their sums, LANES of them staged at a time.
    auto merge_all = [&](unsigned mask) {
        while (mask) {
            unsigned batch = 0;
#pragma unroll
            for (int q = 0; q < C::LANES; ++q) {
                batch |= mask & (~mask + 1u);
                mask &= mask - 1u;
            }
            if ((batch >> lane) & 1u) {
                const int q = __popc(batch & ((1u << lane) - 1u));
                sums.stage(stage + q * C::SS);
                base[q] = cur_base;
                sums.zero();
            }
            __syncwarp();
            add_staged<C::R, C::SS, false>(__popc(batch), stage, base, off, tile, lane);
        }
    };

    for (int s = 0; s < U; ++s) {
        __syncwarp();  // no lane still reads the slot refilled next
        issue(s + C::DEPTH - 1);
        asm volatile("cp.async.wait_group %0;\n" ::"n"(C::DEPTH - 1) : "memory");  // record s has landed
        __syncwarp();
        Spline1D<ORDER, float> sp[3];
        int lb[3] = {0, 0, 0};
        bool ok = false;
        if (s < cnt) {
            if constexpr (REC) {
                ok = locate_record<ORDER>(mp, tp, t, *reinterpret_cast<const float4*>(slot(s) + lane * 4),
                                          sp, lb);
            } else {
                const double* sx = reinterpret_cast<const double*>(slot(s) + lane * 6);
                const double xp[3] = {sx[0], sx[1], sx[2]};
                ok = locate<ORDER>(mp, tp, xp, ob, sp, lb);
            }
            // a particle out of the item's rows (the particles are not sorted) is
            // skipped like one of another tile
            ok = ok && lb[0] >= i_lo && lb[0] <= i_hi;
            if (!ok && A.err) atomicAdd(A.err, 1);
        }
        const int lbin = ok ? (lb[0] * tp.T[1] + lb[1]) * tp.T[2] + lb[2] : -1;
        const bool chg = ok && cur >= 0 && lbin != cur;
        const bool kstep = chg && lbin == cur + 1 && lb[2] != 0;
        const unsigned pm = __ballot_sync(kFull, kstep);
        const unsigned fm = __ballot_sync(kFull, chg && !kstep);
        if (pm) merge_plane(pm);
        if (fm) merge_all(fm);
        if (ok) {
            if (lbin != cur) {
                cur = lbin;
                cur_base = lb[0] * tp.SI + lb[1] * tp.SJ + lb[2];
            }
            const float* sl = slot(s);
            float cp[12];
#pragma unroll
            for (int v = 0; v < 3; ++v) {
                const float4 w = *reinterpret_cast<const float4*>(sl + C::RING_C + lane * 12 + 4 * v);
                cp[4 * v] = w.x, cp[4 * v + 1] = w.y, cp[4 * v + 2] = w.z, cp[4 * v + 3] = w.w;
            }
            const float mass = sl[C::RING_M + lane];
            if constexpr (ORDER >= 2) sums.add_quadratic(sp, mass, cp, D, Dh);
            else sums.add_linear(sp, mass, cp);
        }
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    const unsigned fm = __ballot_sync(kFull, cur >= 0);
    if (fm) merge_all(fm);
    auto values = [&](int idx, float (&x)[C::F]) {
#pragma unroll
        for (int f = 0; f < C::F; ++f) x[f] = tile[f * tp.P + idx];
    };
    flush_tile<ORDER, C::F>(A, values, fm != 0, i_lo, i_hi, ob, smem, C::TILE_OFF / 8, lane);
    __syncwarp();
}

}  // namespace pb
