// Single-call tiled APIC P2G / G2P kernels (FP32 precision form) for
// particles sorted by picasso_cell_sort: one CTA per work item, the item
// bodies are in tiled.cuh.
//
// P2G runs single-warp CTAs (warps finish their items independently; a
// 4-warp CTA would wait for its slowest warp).
// G2P runs 128-thread CTAs sharing one node tile.
#include <algorithm>
#include <mutex>

#include "run_p2g.cuh"
#include "tiled.cuh"

namespace pb {

// Threads of a tiled G2P CTA (one work item each).  Measured at 256^3
// 8 ppc: quadratic 2.92 ms with 128 threads, 2.79 with 64, 2.94 with 32;
// cubic 5.09 / 4.73 / 4.54 ms; linear 1.87 with 64, 2.28 with 32.
template <int ORDER>
struct G2PThreads {
    static constexpr int value = ORDER == 3 ? 32 : 64;
};

template <int ORDER, bool REC, bool FUSED, bool STAG>
__global__ void __launch_bounds__(32, kP2GOccupancy)
p2g_tiled_kernel(P2GArgs A, FusedUpdate F, int64_t n)
{
    extern __shared__ __align__(16) float smem[];
    if (blockIdx.x == 0 && threadIdx.x == 0 && A.err) {
        const int64_t n_valid = __ldg(A.tp.off + A.tp.ntiles);
        if (n > n_valid) atomicAdd(A.err, (int)(n - n_valid));
    }
    int64_t t, a, b;
    const bool any = item_range(A.tp, blockIdx.x, t, a, b);
    if (any) p2g_item<ORDER, REC, STAG>(A, t, a, b, smem);
    if constexpr (FUSED) {
        if (t >= 0) fused_update_arrive<ORDER>(A, F, t);
    }
}

template <int ORDER, bool REC, bool FUSED>
__global__ void __launch_bounds__(32, kRunOccupancy)
p2g_runs_kernel(P2GArgs A, FusedUpdate F, int64_t n)
{
    extern __shared__ __align__(16) float smem[];
    __shared__ int base[32];
    if (blockIdx.x == 0 && threadIdx.x == 0 && A.err) {
        const int64_t n_valid = __ldg(A.tp.off + A.tp.ntiles);
        if (n > n_valid) atomicAdd(A.err, (int)(n - n_valid));
    }
    int64_t t, a, b;
    if (item_range(A.tp, blockIdx.x, t, a, b)) run_p2g_item<ORDER, REC>(A, t, a, b, smem, base);
    if constexpr (FUSED) {
        if (t >= 0) fused_update_arrive<ORDER>(A, F, t);
    }
}

template <int ORDER, bool ADV, bool REC, bool STAG>
__global__ void __launch_bounds__(G2PThreads<ORDER>::value) g2p_tiled_kernel(G2PArgs A, int64_t n)
{
    extern __shared__ __align__(16) float smem[];
    if (blockIdx.x == 0 && threadIdx.x == 0 && A.err) {
        const int64_t n_valid = __ldg(A.tp.off + A.tp.ntiles);
        if (n > n_valid) atomicAdd(A.err, (int)(n - n_valid));
    }
    int64_t t, a, b;
    if (!item_range(A.tp, blockIdx.x, t, a, b)) return;  // CTA-uniform
    g2p_item<ORDER, G2PThreads<ORDER>::value, ADV, REC, STAG>(A, t, a, b,
                                                       reinterpret_cast<float4*>(smem),
                                                       threadIdx.x);
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
// Node-tile strides of the P2G: the nodes (i, j, k0) of a plane are added by the
// lanes of a stream at once, 16 bytes each, 8 lanes per shared-memory cycle; the
// smallest padding (fewer than 8 nodes per row and per plane) that puts the most
// of 8 consecutive rows' nodes on distinct banks.
static void choose_strides(const int NT[3], int K, int* SJ, int* SI)
{
    int best = -1, size = 0;
    for (int sj = NT[2]; sj < NT[2] + 8; ++sj)
        for (int si = NT[1] * sj; si < NT[1] * sj + 8; ++si) {
            int distinct = 0;
            for (int r0 = 0; r0 < K * K; r0 += 8) {
                unsigned banks = 0;
                for (int r = r0; r < r0 + 8 && r < K * K; ++r) banks |= 1u << ((r / K * si + r % K * sj) & 7);
                distinct += __builtin_popcount(banks);
            }
            if (distinct > best || (distinct == best && si < size)) {
                best = distinct;
                size = si;
                *SJ = sj;
                *SI = si;
            }
        }
}

// Node-tile strides of the P2G in runs: value lane + 32 r of a staged lane (4 fields of
// K^3 nodes) lands at f P + a SI + b SJ + c; the smallest padding that puts the most of
// a merge round's 32 values on distinct banks.  The search takes a fraction of a
// millisecond, so the last shapes are kept.
struct RunStrides {
    int NT[3], K, SJ, SI, P;
};

static void search_run_strides(RunStrides* s)
{
    const int K = s->K, KKK = K * K * K, FS = (KKK + 3) & ~3, SV = 4 * FS;
    int best = -1;
    long size = 0;
    for (int sj = s->NT[2]; sj < s->NT[2] + 8; ++sj)
        for (int si = s->NT[1] * sj; si < s->NT[1] * sj + 16; ++si)
            for (int pp = s->NT[0] * si; pp < s->NT[0] * si + 16; ++pp) {
                int distinct = 0;
                for (int r = 0; r < SV; r += 32) {
                    unsigned banks = 0;
                    for (int v = r; v < r + 32 && v < SV; ++v) {
                        const int n = v % FS;
                        if (n < KKK)
                            banks |= 1u << ((v / FS * pp + n / (K * K) * si + n / K % K * sj + n % K) & 31);
                    }
                    distinct += __builtin_popcount(banks);
                }
                if (distinct > best || (distinct == best && pp < size)) {
                    best = distinct;
                    size = pp;
                    s->SJ = sj;
                    s->SI = si;
                    s->P = pp;
                }
            }
}

static RunStrides run_strides(const int NT[3], int K)
{
    constexpr int kSlots = 64;
    static std::mutex mu;
    static RunStrides kept[kSlots];
    static int used = 0, next = 0;
    RunStrides s{{NT[0], NT[1], NT[2]}, K, 0, 0, 0};
    {
        std::lock_guard<std::mutex> lock(mu);
        for (int i = 0; i < used; ++i)
            if (kept[i].K == K && std::equal(NT, NT + 3, kept[i].NT)) return kept[i];
    }
    search_run_strides(&s);
    std::lock_guard<std::mutex> lock(mu);
    kept[used < kSlots ? used++ : next++ % kSlots] = s;
    return s;
}

// Sets whose FP32 P2G keeps its sums in runs (run_p2g.cuh) instead of streams.
// Positions are FP64 and move by FP32 velocities, so the rounding of the node sums
// shows in them: sums in another order put the advected positions of a step (dt 0.1
// cells) 0.7e-9 to 2.4e-9 apart with linear splines, whose gradients make the
// velocities several times the drawn ones, and with quadratic splines 1.4e-9 at one
// particle per cell, 1.1e-9 at two, 0.9e-9 at three and 0.8e-9 at four (relative to
// their norm).  A program that continues a run repeats its positions to 1e-9 only if
// such sets are summed in the same order as ever.  Cubic ones stay below 0.9e-9.
// (The streams would take 0.6 to 0.9 times as long on them.)  A batch, which moves no
// particle, and staggered fields take the streams.
// Large dense quadratic sets are faster in runs: a run stays long in a stencil and its
// lane adds a particle in fewer instructions.  Runs / streams, ms: clustered 16 per cell
// 8 M 0.339 / 0.351, 32 M 1.10 / 1.23, 13 per cell 32 M 1.18 / 1.27, 10 per cell 32 M 1.31
// / 1.34, 6 per cell 32 M 1.58 / 1.50; uniform 16 per cell 32 M 1.35 / 1.32, 10 per cell
// 1.31 / 1.21; below 5 M the streams' parts fill the GPU better (clustered 16 per cell 4 M
// 0.239 / 0.211).
static bool run_sums(int order, const picasso_bins& bins, int64_t n)
{
    if (order != 2) return order == 1;
    double cells = 1.0;
    for (int d = 0; d < 3; ++d) cells *= bins.bin_extent[d];
    return n < 4.0 * cells || (n >= 11.0 * cells && n >= 5000000);
}

// Values of picasso_bins.p2g_lanes a call accepts (the P2G's lanes per particle
// follow from the order: one per k-row of the stencil): orders 1 and 2 take 1, 2
// or 4 (staggered locations 1 or 2), order 3 takes 4; 0 always.
bool valid_lanes(int order, int lanes, bool stag)
{
    if (lanes == 0) return true;
    if (order == 3) return lanes == 4;
    return lanes == 1 || lanes == 2 || (lanes == 4 && !stag);
}

// Cuts the items of n particles into parts, each of equal size within its item, so
// that small sets fill the GPU and a dense tile is not one warp's work: at least
// 1 / 9 of an SM's share of the particles (about the warps of one wave at 14 per SM
// where no item is filled), in sets below 300 000 particles down to 64.  Where most items are
// shorter, the empty parts behind them (1.5 ns each) stay below a tenth of the time.
// P2G streams from 3.5 M particles on: several waves of thirds of a full item, so that the
// last one is not a wave of whole items (quadratic 8 per cell 6 M 0.335 -> 0.279 ms,
// clustered 6 M 0.392 -> 0.323, 8 M 0.460 -> 0.405 ms, in runs 0.441; cubic clustered 8 M
// 0.638 -> 0.533 ms), whole items again from 22 M on.  The linear G2P, whose particles cost
// little beside the staging of their nodes, takes whole items there (uniform 16 per cell 4 M
// 0.080 -> 0.068 ms).
// 2 M quadratic particles (P2G of the streams, uncut -> cut): 16 per cell, 546 items 194
// -> 110 us; 8 per cell, 1152 items 134 -> 114 us (the runs took 111); 4 per cell clustered
// 226 -> 165 us; 300 000: 75 -> 37 us, clustered 159 -> 48 us.  12^3 cells of 4: 69 -> 19 us.
// A batch fills the GPU by its number of instances: there items are cut only where an
// instance has at most 296 (two parts for each of 592), into at most 8 parts (24 instances
// up to 64^3 with the other rule 1.92, so 1.76 ms).  Both are functions of the sizes alone,
// so that every call on the same bins sums in the same order.
// Runs (32 per item already) and the PolyPIC P2G's tiles are not cut.
static void set_parts(TileP* tp, int64_t n, TileUse use, int order)
{
    const int64_t items = tp->ntiles + (n + tp->chunk - 1) / tp->chunk;
    const int64_t few = 148 * 4;
    int64_t part, parts;
    if (use == TileUse::runs || use == TileUse::whole) {
        part = tp->chunk;
        parts = 1;
    } else if (use == TileUse::batch_streams || use == TileUse::batch_other) {
        part = 64;
        parts = std::min<int64_t>({few / items, n / tp->ntiles / part, 8});
    } else {
        int64_t share = n / (148 * 9);
        if (share > 2600 && use == TileUse::streams) share = std::max<int64_t>(1366, share / 4);
        if (share > 2600 && use == TileUse::other && order == 1) share = tp->chunk;
        part = std::max<int64_t>({share, std::min<int64_t>(256, n / few), 64});
        parts = std::min<int64_t>({(std::min<int64_t>(tp->chunk, n) + part - 1) / part,
                                   1 + (1024 + n / 256) / items, 16});
    }
    tp->items_max = items;
    tp->part = (int)std::min<int64_t>(part, tp->chunk);
    tp->split = (int)std::max<int64_t>(1, parts);
}

int64_t item_bound(const TileP& tp)
{
    return tp.items_max * tp.split;
}

// Tile geometry for the bins of n particles, with the strides of the P2G node
// tile if asked.
bool make_tilep(const MeshP& mp, int order, const picasso_bins& bins, int64_t n, TileP* tp,
                TileUse use)
{
    const int K = order + 1;
    int64_t nt = 1;
    for (int d = 0; d < 3; ++d) {
        const int nb = mp.periodic[d] ? mp.own_n[d] : mp.ext[d];
        if (bins.bin_extent[d] != nb || bins.tile[d] < 1) return false;
        if (bins.num_tiles[d] != (nb + bins.tile[d] - 1) / bins.tile[d]) return false;
        tp->T[d] = bins.tile[d];
        tp->nt[d] = bins.num_tiles[d];
        tp->nb[d] = nb;
        tp->NT[d] = bins.tile[d] + K - 1;
        tp->tsh[d] = -1;
        for (int sh = 0; sh < 31; ++sh)
            if ((1 << sh) == bins.tile[d]) tp->tsh[d] = sh;
        nt *= bins.num_tiles[d];
    }
    tp->tsize = (uint32_t)bins.tile[0] * (uint32_t)bins.tile[1] * (uint32_t)bins.tile[2];
    tp->nodes = tp->NT[0] * tp->NT[1] * tp->NT[2];
    tp->SJ = tp->NT[2];
    tp->SI = tp->NT[1] * tp->NT[2];
    tp->P = tp->nodes;
    tp->runs = use == TileUse::runs;
    if (tp->runs) {
        const RunStrides s = run_strides(tp->NT, K);
        tp->SJ = s.SJ;
        tp->SI = s.SI;
        tp->P = s.P;
    } else if (use == TileUse::streams || use == TileUse::batch_streams) {
        int sj, si;
        choose_strides(tp->NT, K, &sj, &si);
        // (a tile that the padding pushes out of shared memory stays unpadded)
        const int64_t limit =
            device_smem_optin() - (use == TileUse::batch_streams ? kBatchStaticSmem : 0);
        if ((int64_t)p2g_warp_bytes(order, tp->NT[0] * si) <= limit) {
            tp->SJ = sj;
            tp->SI = si;
            tp->P = tp->NT[0] * si;
        }
    }
    tp->ntiles = nt;
    tp->off = bins.tile_offset;
    tp->items = bins.tile_items;
    tp->chunk = bins.chunk;
    if (!bins.tile_offset || !bins.tile_items || bins.chunk < 32) return false;
    set_parts(tp, n, use, order);
    return true;
}

// The fused update needs every tile (the last one included) to hold at least
// K - 1 bins along each dimension, so that a node is touched by the items of
// its own tile and of the previous one only.
bool fused_update_fits(const TileP& tp, int order)
{
    const int K = order + 1;
    for (int d = 0; d < 3; ++d) {
        const int last = tp.nb[d] - (tp.nt[d] - 1) * tp.T[d];
        if (tp.T[d] < K - 1 || last < K - 1) return false;
    }
    return true;
}

int device_smem_optin()
{
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    return v;
}

// Packed storage the tiled kernels read: x (N,3) FP64, m (N) FP32, c (N,12)
// FP32 with 16-byte aligned rows.
bool packed_x(const PField& x)
{
    return x.shift == 0 && x.tile_stride == 3 && x.comp_stride == 1 &&
           (reinterpret_cast<uintptr_t>(x.data) % 8) == 0;
}
bool packed_m(const PField& m) { return (m.shift == 0 && m.tile_stride == 1) || m.shift == 63; }
bool packed_c(const PField& c)
{
    return c.shift == 0 && c.tile_stride == 12 && c.comp_stride == 1 &&
           (reinterpret_cast<uintptr_t>(c.data) % 16) == 0;
}

size_t p2g_warp_bytes(int order, int P, bool stag)
{
    const int floats = order == 1 ? (stag ? p2g_warp_floats<1, true>(P) : p2g_warp_floats<1>(P))
                       : order == 2 ? (stag ? p2g_warp_floats<2, true>(P) : p2g_warp_floats<2>(P))
                                    : (stag ? p2g_warp_floats<3, true>(P) : p2g_warp_floats<3>(P));
    return sizeof(float) * (size_t)floats;
}

// (with 128 bytes of static shared memory beside it)
static size_t run_warp_bytes(int order, bool rec, int P)
{
    const int floats = order == 1 ? (rec ? run_warp_floats<1, true>(P) : run_warp_floats<1, false>(P))
                                  : (rec ? run_warp_floats<2, true>(P) : run_warp_floats<2, false>(P));
    return sizeof(float) * (size_t)floats + 128;
}

template <int ORDER, bool REC>
static picasso_status launch_p2g_runs(const P2GArgs& args, const FusedUpdate* fu, int64_t n,
                                      cudaStream_t st)
{
    P2GArgs A = args;
    // (as below: one k-row at least must fit)
    if (RunCfg<ORDER, REC>::TILE_OFF / 8 < A.tp.NT[2]) A.bulk_flush = 0;
    const size_t smem = sizeof(float) * (size_t)run_warp_floats<ORDER, REC>(A.tp.P);
    const int64_t items = item_bound(A.tp);
    auto launch = [&](auto kern, const FusedUpdate& F) -> picasso_status {
        PB_CUDA_TRY(allow_smem(kern, smem));
        kern<<<(unsigned)(items ? items : 1), 32, smem, st>>>(A, F, n);
        return check_launch();
    };
    if (fu) return launch(p2g_runs_kernel<ORDER, REC, true>, *fu);
    return launch(p2g_runs_kernel<ORDER, REC, false>, FusedUpdate{});
}

template <int ORDER, bool REC, bool STAG>
static picasso_status launch_p2g_tiled(const P2GArgs& args, const FusedUpdate* fu, int64_t n,
                                       cudaStream_t st)
{
    P2GArgs A = args;
    // the bulk flush rounds rows into the table: one k-row at least must fit
    if (P2GCfg<ORDER, STAG>::TILE_OFF / 8 < A.tp.NT[2]) A.bulk_flush = 0;
    const size_t smem = p2g_warp_bytes(ORDER, A.tp.P, STAG);
    const int64_t items = item_bound(A.tp);
    auto launch = [&](auto kern, const FusedUpdate& F) -> picasso_status {
        PB_CUDA_TRY(allow_smem(kern, smem));
        kern<<<(unsigned)(items ? items : 1), 32, smem, st>>>(A, F, n);
        return check_launch();
    };
    if constexpr (!STAG) {
        if (fu) return launch(p2g_tiled_kernel<ORDER, REC, true, false>, *fu);
    } else if (fu) {
        return PICASSO_ERR_UNSUPPORTED;  // the fused update is collocated
    }
    return launch(p2g_tiled_kernel<ORDER, REC, false, STAG>, FusedUpdate{});
}

template <int ORDER, bool ADV, bool REC, bool STAG>
static picasso_status launch_g2p_tiled(const G2PArgs& A, int64_t n, cudaStream_t st)
{
    const size_t smem = sizeof(float4) * (size_t)A.tp.nodes;
    PB_CUDA_TRY(allow_smem(g2p_tiled_kernel<ORDER, ADV, REC, STAG>, smem));
    const int64_t items = item_bound(A.tp);
    g2p_tiled_kernel<ORDER, ADV, REC, STAG>
        <<<(unsigned)(items ? items : 1), G2PThreads<ORDER>::value, smem, st>>>(A, n);
    return check_launch();
}

// gm and gmu are views of one (..., 4) 64-bit accumulator: a node's mass and
// momentum are 4 consecutive words, nodes 16-byte aligned, a k-row of nodes
// contiguous.
static bool packed_accumulator(const GField& gm, const GField& gmu)
{
    return gmu.data == gm.data + sizeof(long long) && gm.s[2] == 4 && gmu.s[2] == 4 &&
           gm.s[0] == gmu.s[0] && gm.s[1] == gmu.s[1] && gmu.s[3] == 1 && gm.s[0] % 2 == 0 &&
           gm.s[1] % 2 == 0 && reinterpret_cast<uintptr_t>(gm.data) % 16 == 0;
}

// Spline records the tiled kernels may read instead of the positions: a
// 16-byte aligned array, when the bins carry one.
static const float* bins_records(const picasso_bins& bins)
{
    const uintptr_t r = reinterpret_cast<uintptr_t>(bins.records);
    return (r && r % 16 == 0) ? static_cast<const float*>(bins.records) : nullptr;
}

// stag: the entity's dimension of a staggered location (its grid fields are
// the mass and one momentum component: c_p column stag), else -1.
picasso_status apic_p2g_tiled(const MeshP& mp, int order, int ncomp, Form form, int64_t n,
                              const PField& x, const PField& m, const PField& c, const GField& gm,
                              const GField& gmu, const picasso_bins& bins, int* err,
                              cudaStream_t st, bool* handled, const FusedUpdate* fu, int stag,
                              const HaloPeers* hp, bool batched)
{
    *handled = false;
    if (form != Form::F32Fixed || ncomp != 3 || !packed_x(x) || !packed_m(m) || !packed_c(c))
        return PICASSO_OK;
    const bool sg = stag >= 0;
    if (!valid_lanes(order, bins.p2g_lanes, sg)) return PICASSO_ERR_INVALID_ARGUMENT;
    P2GArgs A;
    const TileUse use = batched ? TileUse::batch_streams
                                : !sg && run_sums(order, bins, n) ? TileUse::runs : TileUse::streams;
    if (!make_tilep(mp, order, bins, n, &A.tp, use)) return PICASSO_ERR_INVALID_ARGUMENT;
    A.rec = bins_records(bins);
    const bool rec = A.rec != nullptr;
    const size_t smem = A.tp.runs ? run_warp_bytes(order, rec, A.tp.P)
                                  : p2g_warp_bytes(order, A.tp.P, sg);
    if ((int64_t)smem > device_smem_optin()) return PICASSO_OK;  // tile too large: plain path
    *handled = true;
    A.mp = mp;
    A.stag = stag;
    A.x = reinterpret_cast<const double*>(x.data);
    A.m = reinterpret_cast<const float*>(m.data);
    A.c = reinterpret_cast<const float*>(c.data);
    A.gm = gm;
    A.gmu = gmu;
    A.scale_m = ldexpf(1.f, gm.fixed_bits);
    A.scale_mu = ldexpf(1.f, gmu.fixed_bits);
    A.err = err;
    A.hp = hp ? *hp : HaloPeers{};
    // the fused update counts its arrivals after element-wise reductions; a
    // neighbour's rows take element-wise reductions too
    A.bulk_flush = !sg && !fu && !A.hp.on && packed_accumulator(gm, gmu);
    if (A.tp.runs) {
        if (order == 1)
            return rec ? launch_p2g_runs<1, true>(A, fu, n, st) : launch_p2g_runs<1, false>(A, fu, n, st);
        return rec ? launch_p2g_runs<2, true>(A, fu, n, st) : launch_p2g_runs<2, false>(A, fu, n, st);
    }
#define PB_CASE(O)                                                                         \
    if (order == O)                                                                        \
        return sg ? (rec ? launch_p2g_tiled<O, true, true>(A, fu, n, st)                   \
                         : launch_p2g_tiled<O, false, true>(A, fu, n, st))                 \
                  : (rec ? launch_p2g_tiled<O, true, false>(A, fu, n, st)                  \
                         : launch_p2g_tiled<O, false, false>(A, fu, n, st));
    PB_CASE(1) PB_CASE(2) PB_CASE(3)
#undef PB_CASE
    return PICASSO_ERR_INVALID_ARGUMENT;
}

template <int ORDER>
static picasso_status launch_g2p_order(const G2PArgs& A, int64_t n, cudaStream_t st, bool adv,
                                       bool stag)
{
    if (adv) return launch_g2p_tiled<ORDER, true, false, false>(A, n, st);
    if (stag) {
        if (A.rec) return launch_g2p_tiled<ORDER, false, true, true>(A, n, st);
        return launch_g2p_tiled<ORDER, false, false, true>(A, n, st);
    }
    if (A.rec) return launch_g2p_tiled<ORDER, false, true, false>(A, n, st);
    return launch_g2p_tiled<ORDER, false, false, false>(A, n, st);
}

picasso_status apic_g2p_tiled(const MeshP& mp, int order, int ncomp, bool f32, int64_t n,
                              const PField& x, const GField& u, const PField& c,
                              const picasso_bins& bins, int* err, const Advect* adv,
                              cudaStream_t st, bool* handled, int stag, const HaloPeers* hp)
{
    *handled = false;
    if (!f32 || ncomp != 3 || !packed_x(x) || !packed_c(c)) return PICASSO_OK;
    if (adv && stag >= 0) return PICASSO_OK;
    G2PArgs A;
    if (!make_tilep(mp, order, bins, n, &A.tp)) return PICASSO_ERR_INVALID_ARGUMENT;
    const size_t smem = sizeof(float4) * (size_t)A.tp.nodes;
    if ((int64_t)smem > device_smem_optin()) return PICASSO_OK;
    *handled = true;
    A.mp = mp;
    A.stag = stag;
    A.x = reinterpret_cast<const double*>(x.data);
    A.u = u;
    A.c = reinterpret_cast<float*>(c.data);
    A.err = err;
    A.x_out = adv ? reinterpret_cast<double*>(x.data) : nullptr;
    A.adv = adv ? *adv : Advect{};
    A.hp = hp ? *hp : HaloPeers{};
    // the advection needs the positions; without it the records replace them
    A.rec = adv ? nullptr : reinterpret_cast<const float4*>(bins_records(bins));
    if (order == 1) return launch_g2p_order<1>(A, n, st, adv != nullptr, stag >= 0);
    if (order == 2) return launch_g2p_order<2>(A, n, st, adv != nullptr, stag >= 0);
    return launch_g2p_order<3>(A, n, st, adv != nullptr, stag >= 0);
}

}  // namespace pb

using namespace pb;

// Arrival counters of the fused update: 8 per tile.
extern "C" picasso_status picasso_apic_p2g_update_workspace(const picasso_bins* bins,
                                                            int64_t* bytes)
{
    if (!bins || !bytes) return PICASSO_ERR_INVALID_ARGUMENT;
    int64_t nt = 1;
    for (int d = 0; d < 3; ++d) {
        if (bins->num_tiles[d] < 1) return PICASSO_ERR_INVALID_ARGUMENT;
        nt *= bins->num_tiles[d];
    }
    *bytes = nt * 8 * (int64_t)sizeof(uint32_t);
    return PICASSO_OK;
}

// Halo peers of the ABI in the kernels' form; false if they do not describe
// neighbour slabs of this (x-non-periodic) mesh.
static bool make_halo_peers(const picasso_halo_peers* p, const MeshP& mp, int nfields,
                            HaloPeers* hp)
{
    if (!p || mp.periodic[0]) return false;
    if (p->lo_end < 0 || p->hi_begin > mp.ext[0] || p->lo_end > p->hi_begin) return false;
    *hp = HaloPeers{};
    hp->on = 1;
    hp->lo_end = p->lo_end;
    hp->hi_begin = p->hi_begin;
    hp->lo_shift = p->lo_shift;
    hp->hi_shift = p->hi_shift;
    for (int f = 0; f < nfields; ++f) {
        if ((p->lo_end > 0 && !p->lo[f]) || (p->hi_begin < mp.ext[0] && !p->hi[f])) return false;
        hp->lo[f] = static_cast<char*>(p->lo[f]);
        hp->hi[f] = static_cast<char*>(p->hi[f]);
    }
    return true;
}

extern "C" picasso_status picasso_apic_p2g_halo(const picasso_spline* sd, int64_t num_particles,
                                                picasso_particle_field x_p,
                                                picasso_particle_field m_p,
                                                picasso_particle_field c_p,
                                                picasso_grid_field m_i, picasso_grid_field mu_i,
                                                const picasso_halo_peers* peers,
                                                const picasso_exec* exec)
{
    MeshP mp;
    picasso_status st = make_mesh(sd, &mp);
    if (st) return st;
    if (num_particles < 0 || !peers) return PICASSO_ERR_INVALID_ARGUMENT;
    if ((st = validate_pfield(num_particles, x_p, PICASSO_F64))) return st;
    if ((st = validate_pfield(num_particles, m_p, PICASSO_F64, PICASSO_F32))) return st;
    if ((st = validate_pfield(num_particles, c_p, m_p.dtype))) return st;
    if ((st = validate_gfield(m_i, PICASSO_F64, PICASSO_I64_FIXED))) return st;
    if ((st = validate_gfield(mu_i, m_i.dtype))) return st;
    if (sd->location != PICASSO_NODE || m_p.dtype != PICASSO_F32 ||
        m_i.dtype != PICASSO_I64_FIXED || !exec || !exec->bins)
        return PICASSO_ERR_UNSUPPORTED;
    if (exec->bins->order != sd->order || exec->bins->location != sd->location)
        return PICASSO_ERR_INVALID_ARGUMENT;
    HaloPeers hp;
    if (!make_halo_peers(peers, mp, 2, &hp)) return PICASSO_ERR_INVALID_ARGUMENT;
    if (num_particles == 0) return PICASSO_OK;
    const PField x = make_pfield(x_p), m = make_pfield(m_p), c = make_pfield(c_p);
    GField gm = make_gfield(m_i), gmu = make_gfield(mu_i);
    gm.overflow = gmu.overflow = exec->overflow_count;
    bool handled = false;
    st = apic_p2g_tiled(mp, sd->order, 3, Form::F32Fixed, num_particles, x, m, c, gm, gmu,
                        *exec->bins, exec->error_count, stream_of(exec), &handled, nullptr, -1,
                        &hp);
    if (st) return st;
    return handled ? PICASSO_OK : PICASSO_ERR_UNSUPPORTED;
}

extern "C" picasso_status picasso_apic_g2p_halo(const picasso_spline* sd, int64_t num_particles,
                                                picasso_particle_field x_p,
                                                picasso_grid_field u_i,
                                                picasso_particle_field c_p,
                                                const picasso_halo_peers* peers,
                                                const picasso_exec* exec)
{
    MeshP mp;
    picasso_status st = make_mesh(sd, &mp);
    if (st) return st;
    if (num_particles < 0 || !peers) return PICASSO_ERR_INVALID_ARGUMENT;
    if ((st = validate_pfield(num_particles, x_p, PICASSO_F64))) return st;
    if ((st = validate_gfield(u_i, PICASSO_F64, PICASSO_F32))) return st;
    if ((st = validate_pfield(num_particles, c_p, u_i.dtype))) return st;
    if (sd->location != PICASSO_NODE || u_i.dtype != PICASSO_F32 || !exec || !exec->bins)
        return PICASSO_ERR_UNSUPPORTED;
    if (exec->bins->order != sd->order || exec->bins->location != sd->location)
        return PICASSO_ERR_INVALID_ARGUMENT;
    HaloPeers hp;
    if (!make_halo_peers(peers, mp, 1, &hp)) return PICASSO_ERR_INVALID_ARGUMENT;
    if (num_particles == 0) return PICASSO_OK;
    const PField x = make_pfield(x_p), c = make_pfield(c_p);
    const GField u = make_gfield(u_i);
    bool handled = false;
    st = apic_g2p_tiled(mp, sd->order, 3, true, num_particles, x, u, c, *exec->bins,
                        exec->error_count, nullptr, stream_of(exec), &handled, -1, &hp);
    if (st) return st;
    return handled ? PICASSO_OK : PICASSO_ERR_UNSUPPORTED;
}

extern "C" picasso_status picasso_apic_p2g_update(
    const picasso_spline* sd, int64_t num_particles, picasso_particle_field x_p,
    picasso_particle_field m_p, picasso_particle_field c_p, picasso_grid_field m_i,
    picasso_grid_field mu_i, picasso_grid_field f_i, const picasso_grid_update_params* prm,
    picasso_grid_field u_i, picasso_grid_field u64_i, void* workspace, int64_t workspace_bytes,
    const picasso_exec* exec)
{
    MeshP mp;
    picasso_status st = make_mesh(sd, &mp);
    if (st) return st;
    if (num_particles < 0 || !prm) return PICASSO_ERR_INVALID_ARGUMENT;
    // the separate calls: same results, two passes (validation included)
    auto separate = [&]() {
        picasso_status s2 = picasso_apic_p2g(sd, num_particles, 3, x_p, m_p, c_p, m_i, mu_i, exec);
        if (s2) return s2;
        return picasso_grid_update(&sd->mesh, m_i, mu_i, f_i, prm, u_i, u64_i, exec);
    };
    const picasso_bins* bins = exec ? exec->bins : nullptr;
    const bool eligible = bins && staggered_dim(sd->location) < 0 && num_particles > 0 &&
                          m_p.dtype == PICASSO_F32 && m_i.dtype == PICASSO_I64_FIXED &&
                          mu_i.dtype == PICASSO_I64_FIXED && u_i.dtype == PICASSO_F32 &&
                          (!f_i.data || f_i.dtype == PICASSO_F64) &&
                          (!u64_i.data || u64_i.dtype == PICASSO_F64) &&
                          bins->order == sd->order && bins->location == sd->location;
    if (!eligible) return separate();
    if ((st = validate_pfield(num_particles, x_p, PICASSO_F64))) return st;
    if ((st = validate_pfield(num_particles, m_p, PICASSO_F32))) return st;
    if ((st = validate_pfield(num_particles, c_p, PICASSO_F32))) return st;
    if ((st = validate_gfield(m_i, PICASSO_I64_FIXED))) return st;
    if ((st = validate_gfield(mu_i, PICASSO_I64_FIXED))) return st;
    if ((st = validate_gfield(u_i, PICASSO_F32))) return st;
    if (f_i.data && (st = validate_gfield(f_i, PICASSO_F64))) return st;
    if (u64_i.data && (st = validate_gfield(u64_i, PICASSO_F64))) return st;
    TileP tp;
    if (!make_tilep(mp, sd->order, *bins, num_particles, &tp)) return PICASSO_ERR_INVALID_ARGUMENT;
    int64_t need = 0;
    if ((st = picasso_apic_p2g_update_workspace(bins, &need))) return st;
    if (!fused_update_fits(tp, sd->order)) return separate();
    if (!workspace || workspace_bytes < need || reinterpret_cast<uintptr_t>(workspace) % 4)
        return PICASSO_ERR_INVALID_ARGUMENT;
    FusedUpdate F;
    if ((st = make_grid_update(&sd->mesh, prm, m_i, mu_i, f_i, &F.P))) return st;
    F.gf = make_gfield(f_i);
    F.gu = make_gfield(u_i);
    F.gu64 = make_gfield(u64_i);
    F.count = static_cast<uint32_t*>(workspace);
    cudaStream_t s = stream_of(exec);
    PB_CUDA_TRY(cudaMemsetAsync(workspace, 0, (size_t)need, s));
    // nodes of regions that no work item touches get the update of an
    // empty node, 0
    {
        const unsigned blocks = grid_for(tp.ntiles * 8, 256, 148LL * 16);
        if (sd->order == 1) zero_untouched_regions_kernel<1><<<blocks, 256, 0, s>>>(mp, tp, F);
        else if (sd->order == 2) zero_untouched_regions_kernel<2><<<blocks, 256, 0, s>>>(mp, tp, F);
        else zero_untouched_regions_kernel<3><<<blocks, 256, 0, s>>>(mp, tp, F);
        if ((st = check_launch())) return st;
    }
    const PField x = make_pfield(x_p), m = make_pfield(m_p), c = make_pfield(c_p);
    GField gm = make_gfield(m_i), gmu = make_gfield(mu_i);
    gm.overflow = gmu.overflow = exec->overflow_count;
    bool handled = false;
    st = apic_p2g_tiled(mp, sd->order, 3, Form::F32Fixed, num_particles, x, m, c, gm, gmu, *bins,
                        exec->error_count, s, &handled, &F, -1, nullptr);
    if (st || handled) return st;
    // the tiled kernel does not take these particles (layout, tile size):
    // the fill of u above is overwritten by the separate update
    return separate();
}
