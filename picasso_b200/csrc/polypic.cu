// PolyPIC particle-to-grid (streams of particles, a lane per k-row of the stencil)
// and grid-to-particle transfers (one thread per particle).  Linear (8 modes)
// follows Picasso_PolyPIC.hpp; quadratic (27 modes) has no reference
// implementation and is the 3-D tensor-product extension of the reference's 2-D
// derivation (doc/polypic/polypic_2d_quadratic.nb): per dimension the
// weight-orthogonal modes
//   s0 = 1, s1 = r, s2 = r^2 - h^2/4 - alpha r,
//   alpha = p (h^2 - 4 p^2) / h^2, p = particle offset from the centre knot,
// and the G2P coefficients are the weighted least-squares projections
//   c_r = sum_i w_i s_r(r_i) u_i / sum_i w_i s_r(r_i)^2
// (for linear splines these reduce to w and dw/dx, PolyPIC.hpp:269-284).
#include "common.cuh"
#include "g2p_f64.cuh"
#include "tiled.cuh"
#include "transfer.cuh"

namespace pb {

// Mode r <-> per-dimension degree.  Modes 0..7 are the reference's linear
// modes {1, x, y, z, xy, xz, yz, xyz} (PolyPIC.hpp:109-116); 8..26 the
// remaining degree <= 2 tensor products, lexicographic in (a, b, c).  The
// degrees of dimension d are packed two bits per mode so that the lookup
// folds to a constant inside unrolled loops.
__host__ __device__ __forceinline__ constexpr int mode_deg(int r, int d)
{
    return (int)(((d == 0 ? 0x2aaaa554004504ull : d == 1 ? 0x2a540a92a45110ull
                                                         : 0x2492492a4a5440ull) >>
                  (2 * r)) & 3ull);
}

__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }

// (Here and in inverse3 every rounding is written out: the kernels of the fixed-point
// P2G have to agree in every bit, and a sum of two products can be fused in two ways.)
template <class R>
__device__ __forceinline__ R quad_alpha(R p, R h)
{
    const R hh = mul_rn(h, h);
    return mul_rn(p, fma(R(-4) * p, p, hh)) / hh;
}

// a[i] for a register array and a run-time i (a select chain, no local memory).
template <int K, class T>
__device__ __forceinline__ T pick(const T (&a)[K], int i)
{
    T v = a[0];
#pragma unroll
    for (int q = 1; q < K; ++q) v = (i == q) ? a[q] : v;
    return v;
}

template <class R>
__device__ __forceinline__ R mode1d(int deg, R r, R h, R alpha)
{
    return deg == 0 ? R(1) : (deg == 1 ? r : r * r - R(0.25) * h * h - alpha * r);
}

// 3x3 inverse by cofactors times 1/det (BatchedLinearAlgebra.hpp:4337-4350,
// 4626-4686); row-major.
template <class R>
__device__ __forceinline__ void inverse3(const R a[9], R inv[9])
{
    auto minor = [&](int p, int q, int r, int s) { return fma(a[p], a[q], -mul_rn(a[r], a[s])); };
    const R c0 = minor(4, 8, 5, 7), c1 = minor(5, 6, 3, 8), c2 = minor(3, 7, 4, 6);
    const R r = R(1) / fma(a[0], c0, fma(a[1], c1, mul_rn(a[2], c2)));
    inv[0] = c0 * r;
    inv[1] = minor(2, 7, 1, 8) * r;
    inv[2] = minor(1, 5, 2, 4) * r;
    inv[3] = c1 * r;
    inv[4] = minor(0, 8, 2, 6) * r;
    inv[5] = minor(2, 3, 0, 5) * r;
    inv[6] = c2 * r;
    inv[7] = minor(1, 6, 0, 7) * r;
    inv[8] = minor(0, 4, 1, 3) * r;
}

// The P2G's spline: eval_spline, in FP64 with the weights of g2p_spline.
template <int ORDER, class R>
__device__ __forceinline__ void pp_spline(double x, double lo, double dx, double rdx,
                                          Spline1D<ORDER, R>& sp)
{
    if constexpr (std::is_same<R, double>::value) {
        double dist0;
        g2p_spline<ORDER>(x, lo, dx, rdx, sp.s0, sp.w, dist0);
#pragma unroll
        for (int n = 0; n < SplineTraits<ORDER>::K; ++n)
            sp.d[n] = __dsub_rn(fma((double)(sp.s0 + n), dx, lo), x);
    } else {
        eval_spline<ORDER>(x, lo, dx, rdx, sp);
    }
}

// ---------------------------------------------------------------------------
// P2G: PolyPIC.hpp:41-130 (collocated) and :140-229 (staggered)
// ---------------------------------------------------------------------------
// A warp takes a contiguous segment of the particles, cut into S streams (3 for
// quadratic, 8 for linear splines) that it sweeps side by side.  Its lanes first
// stage the next particles of every stream in shared memory -- one lane per
// particle evaluates the spline, the backtracking matrix A^-1 and the mode shifts;
// the mode coefficients are copied in the order of their degrees (a, b, c) -- and
// then, step by step, K^2 lanes per stream, one for every k-row of the stencil,
// evaluate the stream's next particle at the row's K nodes,
//   w m sum_abc f0_a(xi_0) f1_b(xi_1) f2_c(xi_2) c_abc,  xi = A^-1 d,
// one dimension after the other, and add it to sums in registers: FP64, or 64-bit
// fixed point with every contribution rounded.  Only when the stream's stencil
// moves are the finished nodes (one k-plane for a move along k, else all) added
// to the grid.  The particles may come in any order; sorted ones move rarely.
// The fixed-point sums are integers: the grid does not depend on the particles'
// order, nor on how they are cut into segments and streams.
//
// With the bins of cell-sorted particles, one that is not in the tile it was sorted
// into is counted instead, as the G2P does (where polypic_tiles takes the bins).
//
// Bound: quadratic, the shared-memory wavefronts of the coefficients (81 values are
// read once per lane group and particle: 64 % of the pipe in FP32, 70 % in FP64)
// next to the FMAs of the sums (about 100 per node with 3 components) and, in fixed
// point, 16 instructions per node for the four roundings (57 % of the issue slots);
// linear, the instructions around the few FMAs, 57 per particle (57 % of the issue
// slots), and 18 L1 wavefronts (69 %).  Against one thread per particle
// with a shared integer tile (FP32) or grid atomics per node (FP64), cell-sorted
// particles: quadratic FP32 96^3 cells 8 per cell 2.50 -> 1.89 ms, FP64 48^3 0.73 ->
// 0.44 ms, linear FP32 101 x 67 x 83 0.278 -> 0.240 ms.  Quadratic warps hold 10
// (FP64: 6) particles per stream in the table and half of them in each of the two
// coefficient chunks; other splits of the shared memory between table and chunks
// took 1 to 9 % longer.
template <int ORDER, int NCU, class R>
struct PPStreams {
    static constexpr int K = SplineTraits<ORDER>::K;
    static constexpr int KK = K * K;
    static constexpr int D = ORDER + 1;                    // modes per dimension
    static constexpr int S = 32 / KK;                      // streams
    // Evaluated particles per stream (table slots), and of those the ones whose
    // coefficients are in shared memory at a time (two chunks, the next one on its
    // way while one is used).
    static constexpr int B = ORDER == 2 ? (sizeof(R) == 8 ? 6 : 10) : 32 / S;
    static constexpr int H = ORDER == 2 ? B / 2 : B;
    static_assert(B % H == 0, "whole chunks");
    static constexpr int P = S * B;
    static constexpr int AB = (D * D * NCU + 3) & ~3;      // coefficients of degree a, padded
    static constexpr int CN = D * AB;
    // Entry of a particle: A^-1, alpha, d_z, (pad), w_z, (pad), d_x, d_y, w_x w_y m.
    // 36 values: the 16-byte accesses of 8 lanes fall on distinct banks.
    static constexpr int E_ALPHA = 9, E_DZ = 12, E_WZ = 16, E_DX = 20, E_DY = 20 + K, E_W = 20 + 2 * K;
    static constexpr int ENTRY = 36;
    static_assert(E_W + KK <= ENTRY, "a particle's entry");
    // A stream's entries and coefficients, with linear splines 16 bytes apart: the
    // 8 streams' reads, 4 lanes of one address each, then fall on distinct banks
    // (without: 4 and 8 on one, 0.276 instead of 0.240 ms).
    static constexpr int GAP = ORDER == 1 ? 16 / (int)sizeof(R) : 0;
    static constexpr int SE = B * ENTRY + GAP, SC = H * CN + GAP;
    static constexpr int CHUNK = S * SC;  // coefficients of a chunk
    static constexpr size_t kBytes = sizeof(R) * (2 * CHUNK + S * SE) + sizeof(int4) * P;  // per warp
};

// Consecutive values of shared memory from a 16-byte aligned address.
template <int N, class R>
__device__ __forceinline__ void read_shared(const R* p, R (&v)[N])
{
    constexpr int W = 16 / sizeof(R);
    static_assert(N % W == 0, "whole 16-byte words");
#pragma unroll
    for (int q = 0; q < N / W; ++q) {
        if constexpr (sizeof(R) == 4) {
            const float4 w = reinterpret_cast<const float4*>(p)[q];
            v[4 * q] = w.x, v[4 * q + 1] = w.y, v[4 * q + 2] = w.z, v[4 * q + 3] = w.w;
        } else {
            const double2 w = reinterpret_cast<const double2*>(p)[q];
            v[2 * q] = w.x, v[2 * q + 1] = w.y;
        }
    }
}

// NC: components of u_p and c_p; STAG: a staggered location, column col of a
// 3-component field (col >= 0, PolyPIC.hpp:181) transferred.  PT: particle storage;
// R: arithmetic; FIXED: 64-bit fixed-point grids (else FP64).
constexpr int kPPWarps = 4;

template <int ORDER, int NC, bool STAG, class PT, class R, bool FIXED>
__global__ void __launch_bounds__(32 * kPPWarps, sizeof(R) == 8 ? 2 : 3)
polypic_p2g_kernel(MeshP mp, TileP tp, int64_t n, int64_t seg, PField x, PField m, PField u, PField c,
                   GField gmu, GField gm, R dt, int col, R scale_mu, R scale_m, int* err)
{
    constexpr int NCU = STAG ? 1 : NC;
    using C = PPStreams<ORDER, NCU, R>;
    using A = typename std::conditional<FIXED, unsigned long long, double>::type;
    constexpr int K = C::K, KK = C::KK, D = C::D, S = C::S, B = C::B, NF = 1 + NCU;
    extern __shared__ __align__(16) unsigned char pp_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    R* cs = reinterpret_cast<R*>(pp_smem + warp * C::kBytes);
    R* table = cs + 2 * C::CHUNK;
    int4* meta = reinterpret_cast<int4*>(table + S * C::SE);
    const int64_t a = ((int64_t)blockIdx.x * kPPWarps + warp) * seg;
    if (a >= n) return;
    const int64_t b = min(a + seg, n);
    const int len = (int)(b - a), U = (len + S - 1) / S;  // particles, per stream
    const int ncp = STAG ? (col >= 0 ? NC : 1) : NC;

    // the lane as evaluator: slot es of stream eg
    const int eg = lane / B, es = lane - eg * B;
    const int64_t p_first = a + (int64_t)eg * U;
    const int ecnt = eg < S ? (int)max((int64_t)0, min(p_first + U, b) - p_first) : 0;
    // the lane as k-row (ri, rj) of stream g
    const bool act = lane < S * KK;
    const int g = act ? lane / KK : 0, row = act ? lane - g * KK : 0;
    const int ri = row / K, rj = row - ri * K;

    // where the lane's values of a particle's record go among the coefficients by
    // degree (bytes)
    constexpr int NVAL = D * D * D * NCU, VPL = (NVAL + 31) / 32;
    unsigned to[VPL];
#pragma unroll
    for (int v = 0; v < VPL; ++v) {
        const int e = lane + 32 * v, r = e / NCU, comp = e - r * NCU;
        to[v] = (unsigned)sizeof(R) *
                (mode_deg(r, 0) * C::AB + (mode_deg(r, 1) * D + mode_deg(r, 2)) * NCU + comp);
    }
    const bool packed = !STAG && c.shift == 0 && c.tile_stride == NVAL && c.comp_stride == 1;

    int lim[3], off[3];  // wrap of a stencil index: [0, lim) then + off
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        lim[d] = mp.periodic[d] ? mp.own_n[d] : 0x7FFFFFFF;
        off[d] = mp.periodic[d] ? mp.own_lo[d] : 0;
    }
    A acc[NF][K];
#pragma unroll
    for (int f = 0; f < NF; ++f)
#pragma unroll
        for (int k = 0; k < K; ++k) acc[f][k] = A(0);
    int cur[3] = {-1, -1, -1};  // stencil start of the sums
    // the sums of the first `count` nodes of the lane's row to the grid
    auto add_nodes = [&](int count) {
        const bool inside = cur[0] + K <= lim[0] && cur[1] + K <= lim[1] && cur[2] + K <= lim[2];
        int q[3] = {cur[0] + ri, cur[1] + rj, cur[2]};
        if (!inside) {
#pragma unroll
            for (int d = 0; d < 2; ++d)
                while (q[d] >= lim[d]) q[d] -= lim[d];
        }
        A* pm = gm.ptr<A>(q[0] + off[0], q[1] + off[1], off[2], 0);
        A* pmu = gmu.ptr<A>(q[0] + off[0], q[1] + off[1], off[2], 0);
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (k >= count) break;
            int qk = q[2] + k;
            while (qk >= lim[2]) qk -= lim[2];
            atomicAdd(pm + (int64_t)qk * gm.s[2], acc[0][k]);
#pragma unroll
            for (int f = 1; f < NF; ++f)
                atomicAdd(pmu + (int64_t)qk * gmu.s[2] + (f - 1) * gmu.s[3], acc[f][k]);
        }
    };
    bool in_range = true;  // of fixed point, the step's contributions
    auto add_to = [&](A& sum, R q) {  // q: scaled to the fixed point
        if constexpr (FIXED) {
            if constexpr (sizeof(R) == 4) {
                in_range = in_range && fabsf(q) < kFixedLimitF;
                sum += (unsigned long long)__float2ll_rn(q);
            } else {
                in_range = in_range && fabs(q) < kFixedLimitD;
                sum += (unsigned long long)__double2ll_rn(q);
            }
        } else {
            sum += q;
        }
    };

    // Copies of the mode coefficients of chunk `ci` (particles ci H .. of every
    // stream) into its buffer, by degree.
    auto fetch = [&](int ci) {
        const int s0 = ci * C::H;
        R* buf = cs + (ci & 1) * C::CHUNK;
        unsigned dst = smem_addr(buf);
        const int here = min(C::H, U - s0);
        auto copy = [](unsigned at, const PT* from) {
            asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(at), "l"(from),
                         "n"(sizeof(R)));
        };
        if (packed) {  // a record's values are consecutive, as are the records
            const PT* src = reinterpret_cast<const PT*>(c.data) + (a + s0) * NVAL + lane;
            int left = len - s0;  // particles from the stream's next one on
#pragma unroll 1
            for (int q = 0; q < S; ++q, left -= U, src += (int64_t)U * NVAL,
                     dst += (unsigned)sizeof(R) * C::SC) {
#pragma unroll
                for (int pl = 0; pl < C::H; ++pl) {
                    if (pl >= here || pl >= left) break;
#pragma unroll
                    for (int v = 0; v < VPL; ++v)
                        if (lane + 32 * v < NVAL)
                            copy(dst + (unsigned)sizeof(R) * pl * C::CN + to[v],
                                 src + pl * NVAL + 32 * v);
                }
            }
        } else {
#pragma unroll 1
            for (int q = 0; q < S; ++q) {
                const int64_t first = a + (int64_t)q * U + s0;
#pragma unroll 1
                for (int pl = 0; pl < here && first + pl < b; ++pl) {
                    const PT* src = reinterpret_cast<const PT*>(c.data) + c.index(first + pl, 0);
#pragma unroll
                    for (int v = 0; v < VPL; ++v) {
                        const int e = lane + 32 * v, r = e / NCU, comp = e - r * NCU;
                        if (e < NVAL)
                            copy(dst + (unsigned)sizeof(R) * (q * C::SC + pl * C::CN) + to[v],
                                 src + (int64_t)(r * ncp + (STAG ? max(col, 0) : comp)) * c.comp_stride);
                    }
                }
            }
        }
        asm volatile("cp.async.commit_group;\n");
    };
    static_assert(sizeof(PT) == sizeof(R), "copied as they are");

    fetch(0);
    for (int s0 = 0; s0 < U; s0 += B) {
        // (the table's readers have passed the syncwarp after their last chunk)
        if (s0 + B + es < ecnt) {  // the next table's particles, into L2
            asm volatile("prefetch.global.L2 [%0];\n" ::"l"(reinterpret_cast<const double*>(x.data) +
                                                            x.index(p_first + s0 + B + es, 0)));
        }
        if (lane < C::P) {
            int4 at = make_int4(-1, -1, -1, 0);
            R* e = table + eg * C::SE + es * C::ENTRY;
            if (s0 + es < ecnt) {
                const int64_t p = p_first + s0 + es;
                Spline1D<ORDER, R> sp[3];
                int st[3];
                bool ok = true;
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    pp_spline<ORDER>(x.get<double>(p, d), mp.lo[d], mp.dx[d], mp.rdx[d], sp[d]);
                    ok = stencil_start<K>(mp, d, sp[d].s0, st[d]) && ok;
                }
                int64_t t_lo = 0, t_hi = n;  // particles sorted into its tile
                if (tp.off && ok) {
                    int64_t t = 0;
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        const int bin = bin_of(mp, tp, d, sp[d].s0);
                        t = t * tp.nt[d] + (tp.tsh[d] >= 0 ? bin >> tp.tsh[d] : bin / tp.T[d]);
                    }
                    t_lo = __ldg(tp.off + t);
                    t_hi = __ldg(tp.off + t + 1);
                }
                if (ok) {
                    const R mass = (R)m.get<PT>(p, 0);
                    // affine material motion operator and its inverse
                    // (PolyPIC.hpp:81-87)
                    R am[9], ai[9];
#pragma unroll
                    for (int q = 0; q < 3; ++q)
#pragma unroll
                        for (int r = 0; r < 3; ++r)
                            am[3 * q + r] =
                                fma(dt, (R)u.get<PT>(p, (1 + q) * 3 + r), R(q == r ? 1 : 0));
                    inverse3(am, ai);
#pragma unroll
                    for (int q = 0; q < 9; ++q) e[q] = ai[q];
#pragma unroll
                    for (int d = 0; d < 3; ++d)
                        e[C::E_ALPHA + d] = ORDER == 2 ? quad_alpha(-sp[d].d[1], (R)mp.dx[d]) : R(0);
#pragma unroll
                    for (int k = 0; k < K; ++k) {
                        e[C::E_DZ + k] = sp[2].d[k];
                        e[C::E_WZ + k] = sp[2].w[k];
                        e[C::E_DX + k] = sp[0].d[k];
                        e[C::E_DY + k] = sp[1].d[k];
                    }
#pragma unroll
                    for (int i = 0; i < K; ++i)
#pragma unroll
                        for (int j = 0; j < K; ++j)
                            e[C::E_W + i * K + j] = mass * sp[0].w[i] * sp[1].w[j];
                }
                if (ok && p >= t_lo && p < t_hi) at = make_int4(st[0], st[1], st[2], 0);
                else if (err) atomicAdd(err, 1);
            }
            if (at.x < 0) {  // adds nothing, moves nothing
#pragma unroll
                for (int q = 0; q < C::ENTRY; ++q) e[q] = R(0);
            }
            meta[lane] = at;
        }
        for (int h = 0; h < B / C::H && s0 + h * C::H < U; ++h) {
        const int ci = s0 / C::H + h;
        fetch(ci + 1);
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");  // this chunk has landed
        __syncwarp();  // ... for every lane, and the table is written
        const int steps = min(C::H, U - (s0 + h * C::H));
        const R* chunk = cs + (ci & 1) * C::CHUNK + g * C::SC;
#pragma unroll 1
        for (int q = 0; q < steps; ++q) {
            const int slot = g * B + h * C::H + q;
            int4 at = meta[slot];
            if (!act) at.x = -1;
            const bool live = at.x >= 0;
            const bool same2 = at.x == cur[0] && at.y == cur[1];
            if (live && !(same2 && at.z == cur[2])) {
                const bool step = same2 && at.z == cur[2] + 1;
                if (cur[0] >= 0) {
                    add_nodes(step ? 1 : K);
#pragma unroll
                    for (int f = 0; f < NF; ++f)
#pragma unroll
                        for (int k = 0; k < K; ++k)
                            acc[f][k] = step && k + 1 < K ? acc[f][k + 1 < K ? k + 1 : k] : A(0);
                }
                cur[0] = at.x;
                cur[1] = at.y;
                cur[2] = at.z;
            }
            __syncwarp();
            if (!live) continue;
            const R* e = table + g * C::SE + (h * C::H + q) * C::ENTRY;
            R ia[12], dz[4], wz[4];  // A^-1 and alpha, d_z, w_z
            read_shared(e, ia);
            read_shared(e + C::E_DZ, dz);
            read_shared(e + C::E_WZ, wz);
            const R di = e[C::E_DX + ri], dj = e[C::E_DY + rj], wab = e[C::E_W + row];
            // modes of the row's nodes (f[.][.][0] is 1): xi = A^-1 d (the
            // backtracked distance, PolyPIC.hpp:90-106), and for degree 2
            // xi^2 - h^2/4 - alpha xi
            R f1[3][K], f2[3][K];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const R base = fma(ia[3 * d + 1], dj, ia[3 * d] * di);
                const R h2 = R(0.25) * (R)mp.dx[d] * (R)mp.dx[d];
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    f1[d][k] = fma(ia[3 * d + 2], dz[k], base);
                    f2[d][k] = ORDER == 2 ? fma(f1[d][k], f1[d][k] - ia[C::E_ALPHA + d], -h2) : R(0);
                }
            }
            // sum_a f0_a sum_b f1_b sum_c f2_c c_abc of every component and node
            R sa[NCU][K];
            const R* cp = chunk + q * C::CN;
#pragma unroll
            for (int da = 0; da < D; ++da) {
                R cc[C::AB];
                read_shared(cp + da * C::AB, cc);
#pragma unroll
                for (int n_ = 0; n_ < NCU; ++n_)
#pragma unroll
                    for (int k = 0; k < K; ++k) {
                        R sb = R(0);
#pragma unroll
                        for (int db = 0; db < D; ++db) {
                            R sc = fma(f1[2][k], cc[(db * D + 1) * NCU + n_], cc[db * D * NCU + n_]);
                            if (ORDER == 2) sc = fma(f2[2][k], cc[(db * D + D - 1) * NCU + n_], sc);
                            sb = db == 0 ? sc : fma(db == 1 ? f1[1][k] : f2[1][k], sc, sb);
                        }
                        sa[n_][k] = da == 0 ? sb : fma(da == 1 ? f1[0][k] : f2[0][k], sb, sa[n_][k]);
                    }
            }
            // (the scales are powers of two: the weights take them exactly)
            const R wm = FIXED ? wab * scale_m : wab, wmu = FIXED ? wab * scale_mu : wab;
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const R w = wmu * wz[k];
                add_to(acc[0][k], wm * wz[k]);
#pragma unroll
                for (int n_ = 0; n_ < NCU; ++n_) add_to(acc[1 + n_][k], w * sa[n_][k]);
            }
            if (FIXED && !in_range) {  // count the contributions out of range
                in_range = true;
                if (gm.overflow) {
#pragma unroll
                    for (int k = 0; k < K; ++k) {
                        to_fixed(gm, wm * wz[k]);
#pragma unroll
                        for (int n_ = 0; n_ < NCU; ++n_) to_fixed(gmu, wmu * wz[k] * sa[n_][k]);
                    }
                }
            }
        }
        __syncwarp();  // the chunk's buffer may be refilled
        }
    }
    asm volatile("cp.async.wait_group 0;\n");
    if (act && cur[0] >= 0) add_nodes(K);
}

// Modes per particle record (c_p rows): 8 linear, 27 quadratic.
template <int ORDER>
struct PPModes {
    static constexpr int value = ORDER == 1 ? 8 : 27;
};

// Shared-memory records of a warp's 32 consecutive particles (packed c_p of
// NV values each, at an odd stride so that the 32 lanes' records start on
// distinct banks): the warp writes every particle's record with coalesced
// stores instead of NV strided stores per thread.
template <class PT, int NV>
struct WarpRecords {
    static constexpr int NVP = NV | 1;
    PT* buf;
    static constexpr size_t kBytesPerWarp = sizeof(PT) * 32 * NVP;
    __device__ __forceinline__ PT& at(int lane, int v) const { return buf[lane * NVP + v]; }
    // records of the particles in `mask` (bit q: particle p0 + q) to packed
    // storage
    __device__ __forceinline__ void store(PT* dst, int cnt, unsigned mask, int lane) const
    {
        __syncwarp();
        for (int e = lane; e < cnt * NV; e += 32) {
            const int q = e / NV;
            if ((mask >> q) & 1u) dst[e] = buf[q * NVP + (e - q * NV)];
        }
        __syncwarp();
    }
};

// Spline and stencil indices of a particle on the whole local mesh (periodic
// wrap, bounds check): the placement of the plain kernels.  STREAM: pp_spline's.
template <int ORDER, class R, bool STREAM = false>
struct MeshPlace {
    const MeshP& mp;
    __device__ __forceinline__ bool operator()(const double xp[3], Spline1D<ORDER, R> sp[3],
                                               int idx[3][SplineTraits<ORDER>::K]) const
    {
        bool ok = true;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            if constexpr (STREAM) pp_spline<ORDER>(xp[d], mp.lo[d], mp.dx[d], mp.rdx[d], sp[d]);
            else eval_spline<ORDER>(xp[d], mp.lo[d], mp.dx[d], mp.rdx[d], sp[d]);
            ok = ok && resolve_stencil<SplineTraits<ORDER>::K>(mp, d, sp[d].s0, idx[d]);
        }
        return ok;
    }
};

// One particle.  place(xp, sp, idx) evaluates the spline and the stencil's
// grid indices (false: skip the particle); acc(f, i, j, k, v) adds v to grid
// field f (0 mass, 1 + d momentum component d); mode(v) returns c_p value v
// (element v of the particle's record).  STREAM: every value in the operations of the
// streams above, in their order, and times 2^fixed_bits of its field (scale_mu,
// scale_m), so that a fixed-point grid has the same bits whichever kernel filled it.
template <int ORDER, int NC, bool STAG, bool STREAM, class PT, class R, class Place, class Acc,
          class Mode>
__device__ __forceinline__ void polypic_p2g_particle(const MeshP& mp, int64_t p, const PField& x,
                                                     const PField& m, const PField& u, R dt,
                                                     int col, R scale_mu, R scale_m, int* err,
                                                     Place&& place, Acc&& acc, Mode&& mode)
{
    constexpr int K = SplineTraits<ORDER>::K;
    {
        Spline1D<ORDER, R> sp[3];
        int idx[3][K];
        const double xp[3] = {x.get<double>(p, 0), x.get<double>(p, 1), x.get<double>(p, 2)};
        if (!place(xp, sp, idx)) {
            if (err) atomicAdd(err, 1);
            return;
        }
        const R mass = (R)m.get<PT>(p, 0);
        // affine material motion operator and its inverse (PolyPIC.hpp:81-87)
        R am[9], ai[9];
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b)
                am[3 * a + b] = fma(dt, (R)u.get<PT>(p, (1 + a) * 3 + b), R(a == b ? 1 : 0));
        inverse3(am, ai);
        R alpha[3] = {R(0), R(0), R(0)};
        R h[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            h[d] = (R)mp.dx[d];
            if (ORDER == 2) alpha[d] = quad_alpha(-sp[d].d[1], h[d]);
        }
        // modes of the transferred field: all NC columns, or column `col`
        constexpr int NCU = STAG ? 1 : NC;
        constexpr int D = ORDER + 1;  // modes per dimension: degrees 0 .. ORDER
        const int ncp = STAG ? (col >= 0 ? NC : 1) : NC;
        // The components are transferred in passes of CB (27 FP64 modes: one
        // at a time, so that a pass holds 27 mode values rather than 81 in
        // registers).
        // The basis sum sum_r c_r b_r(xi) is contracted one dimension at a
        // time: sum_a f0_a sum_b f1_b sum_c f2_c c_(abc).
        constexpr int CB = (sizeof(R) == 8 && ORDER == 2) ? 1 : NCU;
#pragma unroll 1
        for (int d0 = 0; d0 < NCU; d0 += CB) {
            R cp[D][D][D][CB];
            // loop over the modes: their degrees fold to constants
#pragma unroll
            for (int r = 0; r < D * D * D; ++r)
#pragma unroll
                for (int e = 0; e < CB; ++e)
                    cp[mode_deg(r, 0)][mode_deg(r, 1)][mode_deg(r, 2)][e] =
                        (R)mode(r * ncp + (STAG ? col : d0 + e));
            // quadratic: i-planes one after the other, not unrolled (bounds the
            // live range of the 9-node plane bodies, which spill in FP64, and
            // the code size, whose instruction-cache misses stalled the FP32
            // kernel)
#pragma unroll(ORDER == 2 ? 1 : K)
            for (int i = 0; i < K; ++i) {
                const R wxi = pick<K>(sp[0].w, i), dxi = pick<K>(sp[0].d, i);
                const int gi = pick<K>(idx[0], i);
#pragma unroll
                for (int j = 0; j < K; ++j)
#pragma unroll
                    for (int k = 0; k < K; ++k) {
                        const R wab = mass * wxi * sp[1].w[j];
                        const R wm = STREAM ? wab * scale_m * sp[2].w[k] : wab * sp[2].w[k];
                        const R wmu = STREAM ? wab * scale_mu * sp[2].w[k] : wm;
                        const R dist[3] = {dxi, sp[1].d[j], sp[2].d[k]};
                        // backtracked distance xi = A^-1 d (PolyPIC.hpp:90-106) and
                        // its modes
                        R f[3][D];
#pragma unroll
                        for (int q = 0; q < 3; ++q) {
                            f[q][0] = R(1);
                            if constexpr (STREAM) {
                                f[q][1] = fma(ai[3 * q + 2], dist[2],
                                              fma(ai[3 * q + 1], dist[1], ai[3 * q] * dist[0]));
                                if (ORDER == 2)
                                    f[q][D - 1] = fma(f[q][1], f[q][1] - alpha[q],
                                                      -(R(0.25) * h[q] * h[q]));
                            } else {
                                R t = R(0);
#pragma unroll
                                for (int v = 0; v < 3; ++v) t += ai[3 * q + v] * dist[v];
#pragma unroll
                                for (int g = 1; g < D; ++g)
                                    f[q][g] = ORDER == 1 ? t : mode1d(g, t, h[q], alpha[q]);
                            }
                        }
#pragma unroll
                        for (int e = 0; e < CB; ++e) {
                            R sa = R(0);
#pragma unroll
                            for (int a = 0; a < D; ++a) {
                                R sb = R(0);
#pragma unroll
                                for (int b = 0; b < D; ++b) {
                                    R sc = STREAM ? cp[a][b][0][e] : R(0);
#pragma unroll
                                    for (int cc = STREAM ? 1 : 0; cc < D; ++cc) {
                                        if (STREAM) sc = fma(f[2][cc], cp[a][b][cc][e], sc);
                                        else sc += f[2][cc] * cp[a][b][cc][e];
                                    }
                                    if (STREAM) sb = b == 0 ? sc : fma(f[1][b], sc, sb);
                                    else sb += f[1][b] * sc;
                                }
                                if (STREAM) sa = a == 0 ? sb : fma(f[0][a], sb, sa);
                                else sa += f[0][a] * sb;
                            }
                            acc(1 + d0 + e, gi, idx[1][j], idx[2][k], wmu * sa);
                        }
                        if (d0 == 0) acc(0, gi, idx[1][j], idx[2][k], wm);
                    }
            }
        }
    }
}

// P2G of particles in no known order: one thread per particle, every contribution
// added to the grid by itself, bound by the L2's additions (108 per quadratic particle,
// 180 G/s).  In random order a stream of the kernel above moves its stencil with nearly
// every particle and adds as much, on top of its tables; in the order of a cell sort
// the streams win (pp_kernel).
template <int ORDER, int NC, bool STAG, class R, bool FIXED>
__global__ void __launch_bounds__(128)
polypic_p2g_plain_kernel(MeshP mp, int64_t n, PField x, PField m, PField u, PField c, GField gmu,
                         GField gm, R dt, int col, R scale_mu, R scale_m, int* err)
{
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const MeshPlace<ORDER, R, FIXED> place{mp};
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += stride)
        polypic_p2g_particle<ORDER, NC, STAG, FIXED, R, R>(
            mp, p, x, m, u, dt, col, scale_mu, scale_m, err, place,
            [&](int f, int i, int j, int k, R v) {
                if constexpr (FIXED)
                    atomicAdd(f == 0 ? gm.ptr<unsigned long long>(i, j, k, 0)
                                     : gmu.ptr<unsigned long long>(i, j, k, f - 1),
                              (unsigned long long)to_fixed(f == 0 ? gm : gmu, v));
                else
                    atomicAdd(f == 0 ? gm.ptr<double>(i, j, k, 0) : gmu.ptr<double>(i, j, k, f - 1), v);
            },
            [&](int v) { return c.get<R>(p, v); });
}

// ---------------------------------------------------------------------------
// G2P: PolyPIC.hpp:236-293 (collocated) and :300-358 (staggered)
// ---------------------------------------------------------------------------
// One particle; emit(v, value) receives c_p value v (element v of the
// particle's record).  False if the particle was skipped (stencil outside a
// non-periodic mesh): then nothing is emitted.
// place(x, splines, indices) locates the particle; grid(i, j, k, c) returns
// component c of u at stencil indices (i, j, k).
template <int ORDER, int NC, bool STAG, class PT, class R, class Place, class Grid, class Emit>
__device__ __forceinline__ bool polypic_g2p_particle(const MeshP& mp, int64_t p, const PField& x,
                                                     int col, int* err, Place&& place,
                                                     Grid&& grid, Emit&& emit)
{
    constexpr int K = SplineTraits<ORDER>::K;
    constexpr int NCU = STAG ? 1 : NC;
    {
        Spline1D<ORDER, R> sp[3];
        int idx[3][K];
        const double xp[3] = {x.get<double>(p, 0), x.get<double>(p, 1), x.get<double>(p, 2)};
        if (!place(xp, sp, idx)) {
            if (err) atomicAdd(err, 1);
            return false;
        }
        // per-dimension factors G[d][degree][knot]
        R G[3][3][K];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
#pragma unroll
            for (int q = 0; q < K; ++q) {
                G[d][0][q] = sp[d].w[q];
                G[d][1][q] = sp[d].g[q];
                G[d][2][q] = R(0);
            }
            if (ORDER == 2) {
                // closed forms of w s_g(r) / sum_n w s_g(r)^2: G1 = 4 w r / h^2,
                // G2 = {1/(2h^2), -1/h^2, 1/(2h^2)} (the degree-2 quotient is
                // a 0/0 limit at cell faces)
                const R h = (R)mp.dx[d];
                const R rh2 = R(1) / (h * h);
#pragma unroll
                for (int q = 0; q < K; ++q) G[d][1][q] = R(4) * sp[d].w[q] * sp[d].d[q] * rh2;
                G[d][2][0] = R(0.5) * rh2;
                G[d][2][1] = -rh2;
                G[d][2][2] = R(0.5) * rh2;
            }
        }
        // c_(abc) = sum_i G0[a][i] sum_j G1[b][j] sum_k G2[c][k] u_ijk, one
        // i-plane at a time, the components in passes of CB (27 FP64 modes:
        // one component per pass)
        constexpr int D = ORDER + 1;
        constexpr int CB = (sizeof(R) == 8 && ORDER == 2) ? 1 : NCU;
        const int ncp = STAG ? (col >= 0 ? NC : 1) : NC;
#pragma unroll
        for (int d0 = 0; d0 < NCU; d0 += CB) {
            R cp[D][D][D][CB];
#pragma unroll
            for (int a = 0; a < D; ++a)
#pragma unroll
                for (int b = 0; b < D; ++b)
#pragma unroll
                    for (int cc = 0; cc < D; ++cc)
#pragma unroll
                        for (int e = 0; e < CB; ++e) cp[a][b][cc][e] = R(0);
#pragma unroll
            for (int i = 0; i < K; ++i) {
                R t2[D][D][CB];  // [b][c] of this i-plane
#pragma unroll
                for (int b = 0; b < D; ++b)
#pragma unroll
                    for (int cc = 0; cc < D; ++cc)
#pragma unroll
                        for (int e = 0; e < CB; ++e) t2[b][cc][e] = R(0);
#pragma unroll
                for (int j = 0; j < K; ++j) {
                    R ue[K][CB];
#pragma unroll
                    for (int k = 0; k < K; ++k)
#pragma unroll
                        for (int e = 0; e < CB; ++e)
                            ue[k][e] = grid(idx[0][i], idx[1][j], idx[2][k], d0 + e);
#pragma unroll
                    for (int cc = 0; cc < D; ++cc)
#pragma unroll
                        for (int e = 0; e < CB; ++e) {
                            R t1 = R(0);
#pragma unroll
                            for (int k = 0; k < K; ++k) t1 += G[2][cc][k] * ue[k][e];
#pragma unroll
                            for (int b = 0; b < D; ++b) t2[b][cc][e] += G[1][b][j] * t1;
                        }
                }
#pragma unroll
                for (int a = 0; a < D; ++a)
#pragma unroll
                    for (int b = 0; b < D; ++b)
#pragma unroll
                        for (int cc = 0; cc < D; ++cc)
#pragma unroll
                            for (int e = 0; e < CB; ++e)
                                cp[a][b][cc][e] += G[0][a][i] * t2[b][cc][e];
            }
#pragma unroll
            for (int r = 0; r < D * D * D; ++r)
#pragma unroll
                for (int e = 0; e < CB; ++e)
                    emit(r * ncp + (STAG ? col : d0 + e),
                         (PT)cp[mode_deg(r, 0)][mode_deg(r, 1)][mode_deg(r, 2)][e]);
        }
    }
    return true;
}

// WS: c_p is packed (the record of particle p at element p * NV) and written
// through WarpRecords; the lanes of a warp take consecutive particles and
// iterate together.
template <int ORDER, int NC, bool STAG, class GT, class PT, class R, bool WS>
__global__ void __launch_bounds__(128)
polypic_g2p_kernel(MeshP mp, int64_t n, PField x, GField u, PField c, int col, int* err)
{
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const MeshPlace<ORDER, R> place{mp};
    auto grid = [&](int i, int j, int k, int cc) { return (R)__ldg(u.ptr<GT>(i, j, k, cc)); };
    if constexpr (!WS) {
        for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += stride)
            polypic_g2p_particle<ORDER, NC, STAG, PT, R>(
                mp, p, x, col, err, place, grid, [&](int v, PT val) { c.set<PT>(p, v, val); });
    } else {
        constexpr int NV = PPModes<ORDER>::value * NC;
        extern __shared__ __align__(16) unsigned char pp_smem[];
        const int lane = threadIdx.x & 31;
        const WarpRecords<PT, NV> rec{reinterpret_cast<PT*>(pp_smem) +
                                      (threadIdx.x >> 5) * 32 * WarpRecords<PT, NV>::NVP};
        PT* cbase = reinterpret_cast<PT*>(c.data);
        for (int64_t p0 = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31); p0 < n;
             p0 += stride) {
            const int cnt = (int)min((int64_t)32, n - p0);
            bool wrote = false;
            if (lane < cnt)
                wrote = polypic_g2p_particle<ORDER, NC, STAG, PT, R>(
                    mp, p0 + lane, x, col, err, place, grid,
                    [&](int v, PT val) { rec.at(lane, v) = val; });
            rec.store(cbase + p0 * NV, cnt, __ballot_sync(0xFFFFFFFFu, wrote), lane);
        }
    }
}

// c_p stored packed: the record of particle p (all modes and components) at
// element p * NV, 16-byte aligned.
template <int ORDER, int NC, class PT>
static bool packed_record(const PField& c)
{
    constexpr int NV = PPModes<ORDER>::value * NC;
    return c.shift == 0 && c.tile_stride == NV && c.comp_stride == 1 &&
           reinterpret_cast<uintptr_t>(c.data) % 16 == 0;
}

// ---------------------------------------------------------------------------
// Tiled FP32-form kernels (cell-sorted particles, one 128-thread CTA per work
// item of the bins)
// ---------------------------------------------------------------------------
// Placement inside a tile: the spline of the plain FP32 form and the stencil
// in tile-local node indices; false if the particle is not in this tile.
template <int ORDER>
struct TilePlace {
    const MeshP& mp;
    const TileP& tp;
    const int* ob;
    __device__ __forceinline__ bool operator()(const double xp[3], Spline1D<ORDER, float> sp[3],
                                               int idx[3][SplineTraits<ORDER>::K]) const
    {
        int lb[3];
        if (!locate<ORDER>(mp, tp, xp, ob, sp, lb)) return false;
#pragma unroll
        for (int d = 0; d < 3; ++d)
#pragma unroll
            for (int q = 0; q < SplineTraits<ORDER>::K; ++q) idx[d][q] = lb[d] + q;
        return true;
    }
};

__device__ __forceinline__ void count_unsorted(const TileP& tp, int64_t n, int* err)
{
    // particles sorted past the last tile (outside the mesh) belong to no item
    if (blockIdx.x == 0 && threadIdx.x == 0 && err) {
        const int64_t n_valid = __ldg(tp.off + tp.ntiles);
        if (n > n_valid) atomicAdd(err, (int)(n - n_valid));
    }
}

// P2G of sparse cell-sorted sets: the contributions of an item, rounded to fixed point,
// are summed in a shared-memory node tile with 32-bit integer atomics, either on three
// slices of each value (q = hi 2^32 + mid 2^16 + lo with mid, lo in [0, 2^16): the lo
// and mid sums of at most 65536 contributions are exact, the hi sum is exact modulo
// 2^32) or on two words (the low word's carries, read from the atomics' old values,
// added to the high word), so that the recombined 64-bit total is the sum modulo 2^64;
// then the tile is added to the grid, with one grid atomic per touched node and field.
template <int ORDER, int NC>
__global__ void __launch_bounds__(128, ORDER == 2 ? 3 : 1)
polypic_p2g_tiled_kernel(MeshP mp, TileP tp, int64_t n, PField x, PField m, PField u, PField c,
                         GField gmu, GField gm, float dt, float scale_mu, float scale_m, int* err)
{
    extern __shared__ __align__(16) unsigned int pp_tacc[];  // 2 or 3 slices x (1 + NC) x nodes
    count_unsorted(tp, n, err);
    int64_t t, a, b;
    if (!item_range(tp, blockIdx.x, t, a, b)) return;  // CTA-uniform
    // Linear: two words (128^3 8 per cell 2.11 -> 1.52 ms); quadratic, where a run per
    // thread leaves few conflicts: three slices without returned values (the returning
    // atomic measured 6.20 -> 7.27 ms there).
    constexpr bool TWO = ORDER == 1;
    const int nodes = tp.nodes, slice = (1 + NC) * nodes;
    for (int e = threadIdx.x; e < (TWO ? 2 : 3) * slice; e += blockDim.x) pp_tacc[e] = 0u;
    __syncthreads();
    int ob[3];
    tile_origin(tp, t, ob);
    const TilePlace<ORDER> place{mp, tp, ob};
    // Quadratic: each thread sweeps its own contiguous run of the item, so that the lanes
    // of a warp sit in different cells.  Linear (8 nodes, little arithmetic) keeps
    // consecutive particles per warp for coalesced loads.
    const int64_t U = ORDER == 2 ? (b - a + blockDim.x - 1) / blockDim.x : 1;
    const int64_t r0 = a + (int64_t)threadIdx.x * U;
    const int64_t r1 = ORDER == 2 ? min(r0 + U, b) : b;
    const int64_t step = ORDER == 2 ? 1 : blockDim.x;
    for (int64_t p = r0; p < r1; p += step)
        polypic_p2g_particle<ORDER, NC, false, true, float, float>(
            mp, p, x, m, u, dt, -1, scale_mu, scale_m, err, place,
            [&](int f, int i, int j, int k, float v) {
                const unsigned long long q = (unsigned long long)to_fixed(f == 0 ? gm : gmu, v);
                const int e = f * nodes + (i * tp.NT[1] + j) * tp.NT[2] + k;
                if constexpr (TWO) {
                    const unsigned lo = (unsigned)q;
                    const unsigned old = atomicAdd(&pp_tacc[e], lo);
                    const unsigned hi = (unsigned)(q >> 32) + (old + lo < old ? 1u : 0u);
                    if (hi) atomicAdd(&pp_tacc[slice + e], hi);
                } else {
                    atomicAdd(&pp_tacc[e], (unsigned)(q & 0xFFFF));
                    atomicAdd(&pp_tacc[slice + e], (unsigned)((q >> 16) & 0xFFFF));
                    atomicAdd(&pp_tacc[2 * slice + e], (unsigned)(q >> 32));
                }
            },
            [&](int v) { return c.get<float>(p, v); });
    __syncthreads();
    for (int e = threadIdx.x; e < nodes; e += blockDim.x) {
        const int k = e % tp.NT[2], j = (e / tp.NT[2]) % tp.NT[1], i = e / (tp.NT[1] * tp.NT[2]);
        const int gi = node_global(mp, tp, 0, ob[0], i);
        const int gj = node_global(mp, tp, 1, ob[1], j);
        const int gk = node_global(mp, tp, 2, ob[2], k);
#pragma unroll
        for (int f = 0; f <= NC; ++f) {
            const int q = f * nodes + e;
            const unsigned long long v =
                TWO ? ((unsigned long long)pp_tacc[slice + q] << 32) + (unsigned long long)pp_tacc[q]
                    : ((unsigned long long)pp_tacc[2 * slice + q] << 32) +
                          ((unsigned long long)pp_tacc[slice + q] << 16) +
                          (unsigned long long)pp_tacc[q];
            if (v)
                atomicAdd(f == 0 ? gm.ptr<unsigned long long>(gi, gj, gk, 0)
                                 : gmu.ptr<unsigned long long>(gi, gj, gk, f - 1),
                          v);
        }
    }
}

template <int ORDER, int NC>
static picasso_status launch_pp_p2g_tiled(const MeshP& mp, const TileP& tp, int64_t n,
                                          const PField& x, const PField& m, const PField& u,
                                          const PField& c, const GField& gmu, const GField& gm,
                                          double dt, int* err, cudaStream_t st)
{
    const size_t smem = (ORDER == 1 ? 2 : 3) * sizeof(unsigned) * (1 + NC) * (size_t)tp.nodes;
    auto kern = polypic_p2g_tiled_kernel<ORDER, NC>;
    PB_CUDA_TRY(allow_smem(kern, smem));
    kern<<<(unsigned)item_bound(tp), 128, smem, st>>>(mp, tp, n, x, m, u, c, gmu, gm, (float)dt,
                                                      ldexpf(1.f, gmu.fixed_bits),
                                                      ldexpf(1.f, gm.fixed_bits), err);
    return check_launch();
}

// G2P: the tile's node velocities are staged once per item in shared memory;
// packed c_p records leave through WarpRecords.
template <int ORDER, int NC, bool WS>
__global__ void __launch_bounds__(128)
polypic_g2p_tiled_kernel(MeshP mp, TileP tp, int64_t n, PField x, GField u, PField c, int* err)
{
    extern __shared__ __align__(16) unsigned char pp_smem[];
    float4* tile = reinterpret_cast<float4*>(pp_smem);
    count_unsorted(tp, n, err);
    int64_t t, a, b;
    if (!item_range(tp, blockIdx.x, t, a, b)) return;  // CTA-uniform
    int ob[3];
    tile_origin(tp, t, ob);
    for (int e = threadIdx.x; e < tp.nodes; e += blockDim.x) {
        const int k = e % tp.NT[2], j = (e / tp.NT[2]) % tp.NT[1], i = e / (tp.NT[1] * tp.NT[2]);
        const int gi = node_global(mp, tp, 0, ob[0], i);
        const int gj = node_global(mp, tp, 1, ob[1], j);
        const int gk = node_global(mp, tp, 2, ob[2], k);
        const bool inside = (mp.periodic[0] || gi < mp.ext[0]) &&
                            (mp.periodic[1] || gj < mp.ext[1]) &&
                            (mp.periodic[2] || gk < mp.ext[2]);
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (inside) {
            v.x = __ldg(u.ptr<float>(gi, gj, gk, 0));
            if (NC > 1) v.y = __ldg(u.ptr<float>(gi, gj, gk, 1));
            if (NC > 2) v.z = __ldg(u.ptr<float>(gi, gj, gk, 2));
        }
        tile[e] = v;
    }
    __syncthreads();
    const TilePlace<ORDER> place{mp, tp, ob};
    auto grid = [&](int i, int j, int k, int cc) {
        const float4 v = tile[(i * tp.NT[1] + j) * tp.NT[2] + k];
        return cc == 0 ? v.x : (cc == 1 ? v.y : v.z);
    };
    if constexpr (!WS) {
        for (int64_t p = a + threadIdx.x; p < b; p += blockDim.x)
            polypic_g2p_particle<ORDER, NC, false, float, float>(
                mp, p, x, -1, err, place, grid, [&](int v, float val) { c.set<float>(p, v, val); });
    } else {
        constexpr int NV = PPModes<ORDER>::value * NC;
        const int lane = threadIdx.x & 31;
        const WarpRecords<float, NV> rec{
            reinterpret_cast<float*>(pp_smem + ((sizeof(float4) * tp.nodes + 15) & ~size_t(15))) +
            (threadIdx.x >> 5) * 32 * WarpRecords<float, NV>::NVP};
        float* cbase = reinterpret_cast<float*>(c.data);
        for (int64_t p0 = a + (threadIdx.x & ~31); p0 < b; p0 += blockDim.x) {
            const int cnt = (int)min((int64_t)32, b - p0);
            bool wrote = false;
            if (lane < cnt)
                wrote = polypic_g2p_particle<ORDER, NC, false, float, float>(
                    mp, p0 + lane, x, -1, err, place, grid,
                    [&](int v, float val) { rec.at(lane, v) = val; });
            rec.store(cbase + p0 * NV, cnt, __ballot_sync(0xFFFFFFFFu, wrote), lane);
        }
    }
}

template <int ORDER, int NC>
static picasso_status launch_pp_g2p_tiled(const MeshP& mp, const TileP& tp, int64_t n,
                                          const PField& x, const GField& u, const PField& c,
                                          int* err, cudaStream_t st)
{
    constexpr int NV = PPModes<ORDER>::value * NC;
    const bool ws = packed_record<ORDER, NC, float>(c);
    const size_t smem = ((sizeof(float4) * tp.nodes + 15) & ~size_t(15)) +
                        (ws ? 4 * WarpRecords<float, NV>::kBytesPerWarp : 0);
    const int64_t items = item_bound(tp);
    if (ws) {
        auto kern = polypic_g2p_tiled_kernel<ORDER, NC, true>;
        PB_CUDA_TRY(allow_smem(kern, smem));
        kern<<<(unsigned)items, 128, smem, st>>>(mp, tp, n, x, u, c, err);
    } else {
        auto kern = polypic_g2p_tiled_kernel<ORDER, NC, false>;
        PB_CUDA_TRY(allow_smem(kern, smem));
        kern<<<(unsigned)items, 128, smem, st>>>(mp, tp, n, x, u, c, err);
    }
    return check_launch();
}

// ---------------------------------------------------------------------------
// dispatch
// ---------------------------------------------------------------------------
// Launches `kernel` with warp-staged records (dynamic shared memory of four
// warps' records) or without.
template <class PT, int NV, class Kern, class... Args>
static void launch_staged(Kern kernel, bool ws, unsigned blocks, cudaStream_t st, Args... args)
{
    const size_t smem = ws ? 4 * WarpRecords<PT, NV>::kBytesPerWarp : 0;
    if (ws) allow_smem(kernel, smem);
    kernel<<<blocks, 128, smem, st>>>(args...);
}

// The three P2G kernels: particles in no known order go one per thread; the bins tell
// that the particles are in the order of their stencils, where streams win unless there
// is about one particle per stencil.  1 M particles, ms:
//   without bins, streams / particles: random order FP32 linear 0.178 / 0.169, clustered
//   0.274 / 0.240, quadratic clustered 0.930 / 0.881; fixed point of FP64 particles
//   linear 0.217 / 0.199, quadratic 0.785 / 0.587 (only particles that happen to be in
//   cell order would gain: FP32 linear 8 per cell 0.076 / 0.215);
//   sorted FP32, streams / tile: linear 1 per cell 0.145 / 0.124, 2 per cell 0.097 /
//   0.110; quadratic 1 per cell 0.452 / 0.406, 2 per cell 0.330 / 0.354, but 0.1 M of 1
//   per cell 0.045 / 0.049;
//   sorted FP64, streams / particles: linear 1 per cell 0.187 / 0.183, 3 per cell 0.151
//   / 0.205; fixed point 1 per cell linear 0.185 / 0.178, quadratic 0.604 / 0.594, but
//   clustered 0.159 / 0.560 and 0.577 / 1.69.
enum class PPKernel { streams, particles, tile };

static PPKernel pp_kernel(int form, int order, int64_t n, const picasso_bins* bins, bool tiled)
{
    if (!bins) return PPKernel::particles;
    double cells = 1.0;
    for (int d = 0; d < 3; ++d) cells *= bins->bin_extent[d];
    if (form == 0 && order == 1 && n < 2.0 * cells) return PPKernel::particles;
    if (tiled && n < 1.5 * cells && (order == 1 || n >= 500000)) return PPKernel::tile;
    return PPKernel::streams;
}

// Particles per warp: up to 8 tables (a run's end at a segment's costs as much as
// a stencil), as few as leave the warps in the same number of whole waves: with a rule
// by the particles alone 1 M linear FP32 particles were 2.2 waves of 8 tables, now 3 of
// 6 (3 per cell 0.100 -> 0.095 ms; 0.4 M 0.055 -> 0.039 ms; quadratic 0.4 M 0.145 ->
// 0.131 ms).
template <int ORDER, int NC, bool STAG, class PT, class R, bool FIXED>
static picasso_status launch_pp_p2g_form(const MeshP& mp, const TileP& tp, int64_t n, const PField& x,
                                         const PField& m, const PField& u, const PField& c,
                                         const GField& gmu, const GField& gm, R dt, int col, R smu,
                                         R sm, int* err, cudaStream_t st)
{
    using C = PPStreams<ORDER, STAG ? 1 : NC, R>;
    auto kern = polypic_p2g_kernel<ORDER, NC, STAG, PT, R, FIXED>;
    const size_t smem = kPPWarps * C::kBytes;
    PB_CUDA_TRY(allow_smem(kern, smem));
    static const int ctas_per_sm = [&] {
        int v = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, kern, 32 * kPPWarps, smem);
        return v > 0 ? v : 1;
    }();
    const int64_t slots = (int64_t)148 * kPPWarps * ctas_per_sm * C::P;
    const int64_t waves = (n + 8 * slots - 1) / (8 * slots);
    const int64_t tables = (n + waves * slots - 1) / (waves * slots);
    const int64_t seg = tables * C::P;
    const int64_t ctas = (n + seg * kPPWarps - 1) / (seg * kPPWarps);
    kern<<<(unsigned)ctas, 32 * kPPWarps, smem, st>>>(mp, tp, n, seg, x, m, u, c, gmu, gm, dt, col, smu, sm,
                                                      err);
    return check_launch();
}

template <int ORDER, int NC, bool STAG, class R, bool FIXED>
static picasso_status launch_pp_p2g_plain(const MeshP& mp, int64_t n, const PField& x, const PField& m,
                                          const PField& u, const PField& c, const GField& gmu,
                                          const GField& gm, double dt, int col, int* err,
                                          cudaStream_t st)
{
    polypic_p2g_plain_kernel<ORDER, NC, STAG, R, FIXED>
        <<<grid_for(n, 128, 148LL * 128), 128, 0, st>>>(
            mp, n, x, m, u, c, gmu, gm, (R)dt, col, (R)ldexp(1.0, gmu.fixed_bits),
            (R)ldexp(1.0, gm.fixed_bits), err);
    return check_launch();
}

template <int ORDER, int NC, bool STAG>
static picasso_status launch_pp_p2g(int form, PPKernel kernel, const MeshP& mp, const TileP& tp,
                                    int64_t n, const PField& x, const PField& m, const PField& u,
                                    const PField& c, const GField& gmu, const GField& gm, double dt,
                                    int col, int* err, cudaStream_t st)
{
    if (kernel == PPKernel::particles) {
        if (form == 0)
            return launch_pp_p2g_plain<ORDER, NC, STAG, double, false>(mp, n, x, m, u, c, gmu, gm, dt,
                                                                       col, err, st);
        if (form == 1)
            return launch_pp_p2g_plain<ORDER, NC, STAG, float, true>(mp, n, x, m, u, c, gmu, gm, dt,
                                                                     col, err, st);
        return launch_pp_p2g_plain<ORDER, NC, STAG, double, true>(mp, n, x, m, u, c, gmu, gm, dt, col,
                                                                  err, st);
    }
    if constexpr (!STAG) {
        if (kernel == PPKernel::tile)
            return launch_pp_p2g_tiled<ORDER, NC>(mp, tp, n, x, m, u, c, gmu, gm, dt, err, st);
    }
    if (form == 0)
        return launch_pp_p2g_form<ORDER, NC, STAG, double, double, false>(
            mp, tp, n, x, m, u, c, gmu, gm, dt, col, 0.0, 0.0, err, st);
    if (form == 1)
        return launch_pp_p2g_form<ORDER, NC, STAG, float, float, true>(
            mp, tp, n, x, m, u, c, gmu, gm, (float)dt, col, ldexpf(1.0f, gmu.fixed_bits),
            ldexpf(1.0f, gm.fixed_bits), err, st);
    return launch_pp_p2g_form<ORDER, NC, STAG, double, double, true>(
        mp, tp, n, x, m, u, c, gmu, gm, dt, col, ldexp(1.0, gmu.fixed_bits), ldexp(1.0, gm.fixed_bits),
        err, st);
}

template <int ORDER, int NC, bool STAG, class T>
static void launch_pp_g2p_form(const MeshP& mp, int64_t n, const PField& x, const GField& u,
                               const PField& c, int col, int* err, cudaStream_t st)
{
    constexpr int NV = PPModes<ORDER>::value * NC;
    const unsigned blocks = grid_for(n, 128, 148LL * 128);
    if (!STAG && packed_record<ORDER, NC, T>(c))
        launch_staged<T, NV>(polypic_g2p_kernel<ORDER, NC, STAG, T, T, T, true>, true, blocks, st,
                             mp, n, x, u, c, col, err);
    else
        launch_staged<T, NV>(polypic_g2p_kernel<ORDER, NC, STAG, T, T, T, false>, false, blocks,
                             st, mp, n, x, u, c, col, err);
}

template <int ORDER, int NC, bool STAG>
static void launch_pp_g2p(bool f32, const MeshP& mp, int64_t n, const PField& x, const GField& u,
                          const PField& c, int col, int* err, cudaStream_t st)
{
    if (f32) launch_pp_g2p_form<ORDER, NC, STAG, float>(mp, n, x, u, c, col, err, st);
    else launch_pp_g2p_form<ORDER, NC, STAG, double>(mp, n, x, u, c, col, err, st);
}

#define PB_PP_NC_SWITCH(ncomp, ...)                                   \
    switch (ncomp) {                                                  \
        case 1: { constexpr int NC_ = 1; __VA_ARGS__; } break;        \
        case 2: { constexpr int NC_ = 2; __VA_ARGS__; } break;        \
        default: { constexpr int NC_ = 3; __VA_ARGS__; } break;       \
    }

}  // namespace pb

using namespace pb;

static picasso_status polypic_common(const picasso_spline* sd, int64_t n, int32_t ncomp,
                                     MeshP* mp, int* stag, int* col)
{
    picasso_status st = make_mesh(sd, mp);
    if (st) return st;
    if (n < 0 || ncomp < 1 || ncomp > 3) return PICASSO_ERR_INVALID_ARGUMENT;
    if (sd->order == 3) return PICASSO_ERR_UNSUPPORTED;
    *stag = staggered_dim(sd->location);
    if (*stag >= 0 && sd->order != 1) return PICASSO_ERR_UNSUPPORTED;
    // staggered: a 3-component field works on column `dim`, a scalar field
    // on column 0 (PolyPIC.hpp:181, :325)
    *col = (*stag >= 0) ? (ncomp == 3 ? *stag : 0) : -1;
    return PICASSO_OK;
}

// Tiled path for sorted particles (picasso_exec.bins): FP32 form, collocated
// locations; the bins must match the spline.  *tiled stays false when not
// eligible or when the node tile of `node_bytes` per node does not fit in
// shared memory: then particles that have left the tile they were sorted into
// are transferred like the others, else they are counted.
static picasso_status polypic_tiles(const picasso_spline* sd, const picasso_exec* exec, int64_t n,
                                    bool eligible, const MeshP& mp, int node_bytes, TileUse use,
                                    bool* tiled, TileP* tp)
{
    *tiled = false;
    if (!exec || !exec->bins) return PICASSO_OK;
    if (exec->bins->order != sd->order || exec->bins->location != sd->location)
        return PICASSO_ERR_INVALID_ARGUMENT;
    if (!eligible) return PICASSO_OK;
    if (!make_tilep(mp, sd->order, *exec->bins, n, tp, use)) return PICASSO_ERR_INVALID_ARGUMENT;
    // records of four warps on top of the node tile in the G2P (at most)
    const int64_t extra = 4 * 32 * 82 * 4;
    if ((int64_t)node_bytes * tp->nodes + extra > device_smem_optin()) return PICASSO_OK;
    *tiled = true;
    return PICASSO_OK;
}

extern "C" picasso_status picasso_polypic_p2g(const picasso_spline* sd, int64_t num_particles,
                                              int32_t ncomp, picasso_particle_field x_p,
                                              picasso_particle_field m_p,
                                              picasso_particle_field u_p,
                                              picasso_particle_field c_p,
                                              picasso_grid_field mu_i, picasso_grid_field m_i,
                                              double dt, const picasso_exec* exec)
{
    MeshP mp;
    int stag, col;
    picasso_status st = polypic_common(sd, num_particles, ncomp, &mp, &stag, &col);
    if (st) return st;
    if ((st = validate_pfield(num_particles, x_p, PICASSO_F64))) return st;
    if ((st = validate_pfield(num_particles, m_p, PICASSO_F64, PICASSO_F32))) return st;
    if ((st = validate_pfield(num_particles, u_p, m_p.dtype))) return st;
    if ((st = validate_pfield(num_particles, c_p, m_p.dtype))) return st;
    if ((st = validate_gfield(m_i, PICASSO_F64, PICASSO_I64_FIXED))) return st;
    if ((st = validate_gfield(mu_i, m_i.dtype))) return st;
    int form;
    if (m_p.dtype == PICASSO_F64 && m_i.dtype == PICASSO_F64) form = 0;
    else if (m_p.dtype == PICASSO_F32 && m_i.dtype == PICASSO_I64_FIXED) form = 1;
    else if (m_p.dtype == PICASSO_F64 && m_i.dtype == PICASSO_I64_FIXED) form = 2;
    else return PICASSO_ERR_UNSUPPORTED;
    if (num_particles == 0) return PICASSO_OK;
    cudaStream_t s = stream_of(exec);
    int* err = exec ? exec->error_count : nullptr;
    PField x = make_pfield(x_p), m = make_pfield(m_p), u = make_pfield(u_p), c = make_pfield(c_p);
    GField gmu = make_gfield(mu_i), gm = make_gfield(m_i);
    gmu.overflow = gm.overflow = exec ? exec->overflow_count : nullptr;
    bool tiled = false;
    TileP tp;
    // (the tile kernel's 32-bit sums are exact for work items of at most 65536 particles)
    const bool p2g_ok = form == 1 && stag < 0 && exec && exec->bins && exec->bins->chunk <= 65536;
    if ((st = polypic_tiles(sd, exec, num_particles, p2g_ok, mp, 12 * (1 + ncomp), TileUse::whole,
                            &tiled, &tp)))
        return st;
    if (!tiled) tp.off = nullptr;
    const PPKernel kernel =
        pp_kernel(form, sd->order, num_particles, exec ? exec->bins : nullptr, tiled);
    if (sd->order == 1) {
        if (stag >= 0) {
            PB_PP_NC_SWITCH(ncomp, return launch_pp_p2g<1, NC_, true>(form, kernel, mp, tp, num_particles,
                                                                      x, m, u, c, gmu, gm, dt, col,
                                                                      err, s));
        } else {
            PB_PP_NC_SWITCH(ncomp, return launch_pp_p2g<1, NC_, false>(form, kernel, mp, tp,
                                                                       num_particles, x, m, u, c, gmu,
                                                                       gm, dt, col, err, s));
        }
    }
    PB_PP_NC_SWITCH(ncomp, return launch_pp_p2g<2, NC_, false>(form, kernel, mp, tp, num_particles, x, m, u, c,
                                                               gmu, gm, dt, col, err, s));
    return PICASSO_OK;
}

extern "C" picasso_status picasso_polypic_g2p(const picasso_spline* sd, int64_t num_particles,
                                              int32_t ncomp, picasso_particle_field x_p,
                                              picasso_grid_field u_i, picasso_particle_field c_p,
                                              const picasso_exec* exec)
{
    MeshP mp;
    int stag, col;
    picasso_status st = polypic_common(sd, num_particles, ncomp, &mp, &stag, &col);
    if (st) return st;
    if ((st = validate_pfield(num_particles, x_p, PICASSO_F64))) return st;
    if ((st = validate_gfield(u_i, PICASSO_F64, PICASSO_F32))) return st;
    if ((st = validate_pfield(num_particles, c_p, u_i.dtype))) return st;
    if (num_particles == 0) return PICASSO_OK;
    const bool f32 = u_i.dtype == PICASSO_F32;
    cudaStream_t s = stream_of(exec);
    int* err = exec ? exec->error_count : nullptr;
    PField x = make_pfield(x_p), c = make_pfield(c_p);
    GField u = make_gfield(u_i);
    bool tiled = false;
    TileP tp;
    if ((st = polypic_tiles(sd, exec, num_particles, f32 && stag < 0, mp, 16, TileUse::other, &tiled, &tp))) return st;
    if (tiled) {
        if (sd->order == 1) {
            PB_PP_NC_SWITCH(ncomp, return launch_pp_g2p_tiled<1, NC_>(mp, tp, num_particles, x, u,
                                                                      c, err, s));
        } else {
            PB_PP_NC_SWITCH(ncomp, return launch_pp_g2p_tiled<2, NC_>(mp, tp, num_particles, x, u,
                                                                      c, err, s));
        }
    }
    if (sd->order == 1) {
        if (stag >= 0) {
            PB_PP_NC_SWITCH(ncomp, launch_pp_g2p<1, NC_, true>(f32, mp, num_particles, x, u, c, col,
                                                                err, s));
        } else {
            PB_PP_NC_SWITCH(ncomp, launch_pp_g2p<1, NC_, false>(f32, mp, num_particles, x, u, c, col,
                                                                 err, s));
        }
    } else {
        PB_PP_NC_SWITCH(ncomp, launch_pp_g2p<2, NC_, false>(f32, mp, num_particles, x, u, c, col,
                                                             err, s));
    }
    return check_launch();
}
