// APIC particle-to-grid and grid-to-particle transfers of the plain form of
// Picasso_APIC.hpp, for particles in any order: FP64 by warps (warp_p2g.cuh,
// g2p_f64.cuh; the latter with a node tile for binned particles), the fixed-point
// P2G and FP32 G2P by one thread per particle (plain.cuh).  The shared-memory
// tiled FP32 kernels for binned particles are in tiled.cu.
#include "g2p_f64.cuh"
#include "plain.cuh"
#include "warp_p2g.cuh"

namespace pb {

// ---------------------------------------------------------------------------
// kernels: one thread per particle, grid-stride
// ---------------------------------------------------------------------------
template <int ORDER, int NC, bool STAG, class R>
__global__ void __launch_bounds__(256)
apic_p2g_kernel(MeshP mp, int64_t n, PField x, PField m, PField c, GField gm, GField gmu,
                int stag, R scale_m, R scale_mu, int* err)
{
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += stride)
        apic_p2g_particle<ORDER, NC, STAG, R>(mp, p, x, m, c, gm, gmu, stag, scale_m, scale_mu,
                                              err);
}

template <int ORDER, int NC, bool STAG, bool ADV>
__global__ void __launch_bounds__(256)
apic_g2p_kernel(MeshP mp, int64_t n, PField x, GField u, PField c, int stag, int* err, Advect adv)
{
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += stride)
        apic_g2p_particle<ORDER, NC, STAG, ADV>(mp, p, x, u, c, stag, err, &adv);
}

// FP64 G2P: grid-stride over 32 particles per warp.  Cubic: 3 CTAs, without spills, and
// the particles as they come: 192 loads of 8 bytes hide their latency by themselves, and
// 4 CTAs or ordering the lanes only cost (0.1 M clustered in random order 0.051 -> 0.035
// ms, 4 M 1.53 -> 1.41 ms; in cell order 4 M 0.394 -> 0.406 ms).  Scalar fields, whose
// results are one sector per particle, neither: linear 1 M in cell order 0.026 -> 0.020
// ms (one thread per particle 0.021).
template <int ORDER, int NC, bool STAG, bool ADV, bool UNIT>
__global__ void __launch_bounds__(128, ORDER == 3 ? 3 : 4)
apic_g2p_f64_kernel(MeshP mp, int64_t n, PField x, GField u, PField c, int stag, int* err,
                    Advect adv, bool packed)
{
    using R = WarpRows<STAG ? 3 : NC, ADV>;
    __shared__ double rows[4][R::DOUBLES];
    const int warp = threadIdx.x >> 5;
    double* mine = packed ? rows[warp] : nullptr;
    const int64_t stride = (int64_t)gridDim.x * 128;
    for (int64_t p0 = (int64_t)blockIdx.x * 128 + warp * 32; p0 < n; p0 += stride)
        apic_g2p_warp<ORDER, NC, STAG, false, ADV, UNIT, ORDER == 3 || (NC == 1 && !STAG)>(
            mp, p0, (int)min((int64_t)32, n - p0), x, u, c, stag, err, &adv, mine);
}

// FP64 G2P of cell-sorted particles: one CTA per work item of the bins.  The
// particles past the last item (out of the mesh at the sort) are taken from
// global memory by all CTAs.
template <int ORDER, bool ADV>
__global__ void __launch_bounds__(128, 4)
apic_g2p_tiled_f64_kernel(MeshP mp, TileP tp, int64_t n, PField x, GField u, PField c, int* err,
                          Advect adv, bool packed)
{
    using R = WarpRows<3, ADV>;
    extern __shared__ __align__(16) double g2p_nodes[];  // 3 per tile node
    __shared__ double rows[4][R::DOUBLES];
    const int tid = threadIdx.x, warp = tid >> 5;
    int64_t t, a, b;
    if (item_range(tp, blockIdx.x, t, a, b)) {
        b = min(b, n);
        if (a < b)
            g2p_item_f64<ORDER, 128, false, ADV>(mp, tp, t, a, b, x, u, c, err, &adv, g2p_nodes,
                                                 packed ? rows[0] : nullptr, tid);
    }
    // (32 particles per warp; their rows go through the warp's buffer)
    for (int64_t p0 = __ldg(tp.off + tp.ntiles) + (int64_t)blockIdx.x * 128 + warp * 32; p0 < n;
         p0 += (int64_t)gridDim.x * 128) {
        const int64_t p = p0 + (tid & 31);
        bool ok = p < n;
        double xp[3] = {0.0, 0.0, 0.0}, up[3], B[3][3];
        if (ok) {
#pragma unroll
            for (int d = 0; d < 3; ++d) xp[d] = x.get<double>(p, d);
            ok = g2p_stray<ORDER, false>(mp, xp, u, up, B);
            if (!ok && err) atomicAdd(err, 1);
        }
        g2p_store<3, false, ADV>(p0, tid & 31, ok, xp, up, B, x, c, -1, &adv,
                                 packed ? rows[warp] : nullptr);
    }
}

// FP64 P2G: 4-warp CTAs, each warp one segment of `seg` consecutive particles.
constexpr int kWarpP2GWarps = 4;

template <int ORDER, int NC, bool STAG>
__global__ void __launch_bounds__(32 * kWarpP2GWarps, ORDER == 3 ? 3 : 4)
apic_p2g_warp_kernel(MeshP mp, int64_t n, int64_t seg, PField x, PField m, PField c, bool wide,
                     GField gm, GField gmu, int stag, int* err)
{
    using W = WarpP2G<ORDER, NC, STAG>;
    __shared__ __align__(16) double sm[kWarpP2GWarps][W::DOUBLES];
    const int warp = threadIdx.x >> 5;
    const int64_t a = ((int64_t)blockIdx.x * kWarpP2GWarps + warp) * seg;
    if (a < n)
        apic_p2g_warp<ORDER, NC, STAG>(mp, a, min(a + seg, n), x, m, c, wide, gm, gmu, stag, err,
                                       sm[warp]);
}

// Particles per warp: 256 (long enough that the flush at a segment's end is a
// small part, 108 grid additions per quadratic segment), less -- at least 8, or
// with one momentum component, whose lanes may add a particle each, 32 -- when the
// particles would not give every SM 16 warps.
static int64_t warp_segment(int64_t n, int64_t least)
{
    const int64_t seg = (n / (148 * 16) + 7) / 8 * 8;
    return seg < least ? least : (seg > 32 ? (seg > 256 ? 256 : seg / 32 * 32) : seg);
}

// ---------------------------------------------------------------------------
// dispatch
// ---------------------------------------------------------------------------
template <int ORDER, int NC, bool STAG>
static void launch_p2g(Form form, const MeshP& mp, int64_t n, const PField& x, const PField& m,
                       const PField& c, const GField& gm, const GField& gmu, int stag, int* err,
                       cudaStream_t st)
{
    const int threads = 256;
    const unsigned blocks = grid_for(n, threads);
    if (form == Form::F64) {
        const int64_t seg = warp_segment(n, STAG || NC == 1 ? 32 : 8);
        const int64_t ctas = (n + seg * kWarpP2GWarps - 1) / (seg * kWarpP2GWarps);
        apic_p2g_warp_kernel<ORDER, NC, STAG><<<(unsigned)ctas, 32 * kWarpP2GWarps, 0, st>>>(
            mp, n, seg, x, m, c, wide_rows<STAG ? 3 : NC>(c), gm, gmu, stag, err);
    } else if (form == Form::F32Fixed) {
        apic_p2g_kernel<ORDER, NC, STAG, float><<<blocks, threads, 0, st>>>(
            mp, n, x, m, c, gm, gmu, stag, ldexpf(1.0f, gm.fixed_bits),
            ldexpf(1.0f, gmu.fixed_bits), err);
    } else {
        apic_p2g_kernel<ORDER, NC, STAG, double><<<blocks, threads, 0, st>>>(
            mp, n, x, m, c, gm, gmu, stag, ldexp(1.0, gm.fixed_bits),
            ldexp(1.0, gmu.fixed_bits), err);
    }
}

// adv != nullptr (collocated, 3 components only): G2P then the position update.
template <int ORDER, int NC, bool STAG>
static void launch_g2p(bool f32, const MeshP& mp, int64_t n, const PField& x, const GField& u,
                       const PField& c, int stag, int* err, const Advect* adv, cudaStream_t st)
{
    const Advect a = adv ? *adv : Advect{};
    if (!f32) {
        const unsigned blocks = grid_for(n, 128, 148LL * 64);
        const bool packed =
            (NC > 1 || STAG) && packed_rows_f64(x, c, 4 * (STAG ? 3 : NC), adv != nullptr);
        auto launch = [&](auto kern) {
            kern<<<blocks, 128, 0, st>>>(mp, n, x, u, c, stag, err, a, packed);
        };
        if constexpr (STAG || NC == 1) {  // one component: nothing to be adjacent
            launch(apic_g2p_f64_kernel<ORDER, NC, STAG, false, true>);
        } else {
            const bool unit = u.s[3] == 1;
            if constexpr (NC == 3) {
                if (adv) {
                    if (unit) launch(apic_g2p_f64_kernel<ORDER, NC, STAG, true, true>);
                    else launch(apic_g2p_f64_kernel<ORDER, NC, STAG, true, false>);
                    return;
                }
            }
            if (unit) launch(apic_g2p_f64_kernel<ORDER, NC, STAG, false, true>);
            else launch(apic_g2p_f64_kernel<ORDER, NC, STAG, false, false>);
        }
        return;
    }
    const int threads = 256;
    const unsigned blocks = grid_for(n, threads);
    if constexpr (NC == 3 && !STAG) {
        if (adv) {
            apic_g2p_kernel<ORDER, NC, STAG, true>
                <<<blocks, threads, 0, st>>>(mp, n, x, u, c, stag, err, a);
            return;
        }
    }
    apic_g2p_kernel<ORDER, NC, STAG, false><<<blocks, threads, 0, st>>>(
        mp, n, x, u, c, stag, err, a);
}

// FP64 G2P with bins (3 collocated components); *handled stays false where gathering
// from global memory is faster: g2p_tiles_pay, and sets that leave the tiles' CTAs about
// a wave (tile / global memory, sorted, 8 per cell, ms: quadratic 0.15 M 0.019 / 0.013,
// 0.5 M 0.035 / 0.031, 1 M 0.063 / 0.066, 2 M 0.104 / 0.120; cubic 0.5 M 0.052 / 0.054,
// 1 M 0.084 / 0.107).
template <int ORDER>
static picasso_status launch_g2p_tiled_f64(const MeshP& mp, const TileP& tp, int64_t n,
                                           const PField& x, const GField& u, const PField& c,
                                           int* err, const Advect* adv, cudaStream_t st,
                                           bool* handled)
{
    const size_t smem = 3 * sizeof(double) * (size_t)tp.nodes;
    const size_t rows = 4 * sizeof(double) * (size_t)(adv ? WarpRows<3, true>::DOUBLES
                                                          : WarpRows<3, false>::DOUBLES);
    if ((int64_t)(smem + rows) > device_smem_optin()) return PICASSO_OK;
    if (n < (ORDER == 3 ? 1000000 : 1500000) || !g2p_tiles_pay(tp, ORDER, n)) return PICASSO_OK;
    *handled = true;
    const bool packed = packed_rows_f64(x, c, 12, adv != nullptr);
    const int64_t items = item_bound(tp);
    auto launch = [&](auto kern) -> picasso_status {
        PB_CUDA_TRY(allow_smem(kern, smem));
        kern<<<(unsigned)items, 128, smem, st>>>(mp, tp, n, x, u, c, err, adv ? *adv : Advect{}, packed);
        return check_launch();
    };
    if (adv) return launch(apic_g2p_tiled_f64_kernel<ORDER, true>);
    return launch(apic_g2p_tiled_f64_kernel<ORDER, false>);
}

#define PB_ORDER_SWITCH(order, ...)               \
    switch (order) {                              \
        case 1: { constexpr int O_ = 1; __VA_ARGS__; } break; \
        case 2: { constexpr int O_ = 2; __VA_ARGS__; } break; \
        default: { constexpr int O_ = 3; __VA_ARGS__; } break; \
    }

picasso_status apic_p2g_plain(const MeshP& mp, int order, int stag, int ncomp, Form form,
                              int64_t n, const PField& x, const PField& m, const PField& c,
                              const GField& gm, const GField& gmu, int* err, cudaStream_t st)
{
    if (stag >= 0) {
        PB_ORDER_SWITCH(order, launch_p2g<O_, 3, true>(form, mp, n, x, m, c, gm, gmu, stag, err, st));
    } else if (ncomp == 1) {
        PB_ORDER_SWITCH(order, launch_p2g<O_, 1, false>(form, mp, n, x, m, c, gm, gmu, -1, err, st));
    } else if (ncomp == 2) {
        PB_ORDER_SWITCH(order, launch_p2g<O_, 2, false>(form, mp, n, x, m, c, gm, gmu, -1, err, st));
    } else {
        PB_ORDER_SWITCH(order, launch_p2g<O_, 3, false>(form, mp, n, x, m, c, gm, gmu, -1, err, st));
    }
    return check_launch();
}

picasso_status apic_g2p_plain(const MeshP& mp, int order, int stag, int ncomp, bool f32,
                              int64_t n, const PField& x, const GField& u, const PField& c,
                              int* err, const Advect* adv, cudaStream_t st)
{
    if (stag >= 0) {
        PB_ORDER_SWITCH(order, launch_g2p<O_, 3, true>(f32, mp, n, x, u, c, stag, err, nullptr, st));
    } else if (ncomp == 1) {
        PB_ORDER_SWITCH(order, launch_g2p<O_, 1, false>(f32, mp, n, x, u, c, -1, err, nullptr, st));
    } else if (ncomp == 2) {
        PB_ORDER_SWITCH(order, launch_g2p<O_, 2, false>(f32, mp, n, x, u, c, -1, err, nullptr, st));
    } else {
        PB_ORDER_SWITCH(order, launch_g2p<O_, 3, false>(f32, mp, n, x, u, c, -1, err, adv, st));
    }
    return check_launch();
}

}  // namespace pb

using namespace pb;

extern "C" picasso_status picasso_apic_p2g(const picasso_spline* sd, int64_t num_particles,
                                           int32_t ncomp, picasso_particle_field x_p,
                                           picasso_particle_field m_p, picasso_particle_field c_p,
                                           picasso_grid_field m_i, picasso_grid_field mu_i,
                                           const picasso_exec* exec)
{
    MeshP mp;
    picasso_status st = make_mesh(sd, &mp);
    if (st) return st;
    if (num_particles < 0) return PICASSO_ERR_INVALID_ARGUMENT;
    const int stag = staggered_dim(sd->location);
    if (stag >= 0 ? ncomp != 3 : (ncomp < 1 || ncomp > 3)) return PICASSO_ERR_INVALID_ARGUMENT;
    if ((st = validate_pfield(num_particles, x_p, PICASSO_F64))) return st;
    if ((st = validate_pfield(num_particles, m_p, PICASSO_F64, PICASSO_F32))) return st;
    if ((st = validate_pfield(num_particles, c_p, m_p.dtype))) return st;
    if ((st = validate_gfield(m_i, PICASSO_F64, PICASSO_I64_FIXED))) return st;
    if ((st = validate_gfield(mu_i, m_i.dtype))) return st;
    Form form;
    if (m_p.dtype == PICASSO_F64 && m_i.dtype == PICASSO_F64) form = Form::F64;
    else if (m_p.dtype == PICASSO_F32 && m_i.dtype == PICASSO_I64_FIXED) form = Form::F32Fixed;
    else if (m_p.dtype == PICASSO_F64 && m_i.dtype == PICASSO_I64_FIXED) form = Form::F64Fixed;
    else return PICASSO_ERR_UNSUPPORTED;
    if (num_particles == 0) return PICASSO_OK;
    cudaStream_t s = stream_of(exec);
    int* err = exec ? exec->error_count : nullptr;
    PField x = make_pfield(x_p), m = make_pfield(m_p), c = make_pfield(c_p);
    GField gm = make_gfield(m_i), gmu = make_gfield(mu_i);
    gm.overflow = gmu.overflow = exec ? exec->overflow_count : nullptr;
    if (exec && exec->bins) {
        // bins describe particles sorted for this spline
        if (exec->bins->order != sd->order || exec->bins->location != sd->location)
            return PICASSO_ERR_INVALID_ARGUMENT;
        bool handled = false;
        st = apic_p2g_tiled(mp, sd->order, ncomp, form, num_particles, x, m, c, gm, gmu,
                            *exec->bins, err, s, &handled, nullptr, stag);
        if (st || handled) return st;
    }
    return apic_p2g_plain(mp, sd->order, stag, ncomp, form, num_particles, x, m, c, gm, gmu,
                          err, s);
}

// G2P, and with dt != nullptr the position update x += dt u_p after it.
// dt != nullptr: G2P with advection; key_out != nullptr: it also writes the
// sort key of every moved particle for bins of the given tile shape.
static picasso_status apic_g2p_entry(const picasso_spline* sd, int64_t num_particles,
                                     int32_t ncomp, picasso_particle_field x_p,
                                     picasso_grid_field u_i, picasso_particle_field c_p,
                                     const double* dt, const picasso_exec* exec,
                                     const int32_t* key_tile = nullptr,
                                     uint32_t* key_out = nullptr)
{
    MeshP mp;
    picasso_status st = make_mesh(sd, &mp);
    if (st) return st;
    if (num_particles < 0) return PICASSO_ERR_INVALID_ARGUMENT;
    const int stag = staggered_dim(sd->location);
    if (stag >= 0 ? ncomp != 3 : (ncomp < 1 || ncomp > 3)) return PICASSO_ERR_INVALID_ARGUMENT;
    if (dt && (stag >= 0 || ncomp != 3)) return PICASSO_ERR_INVALID_ARGUMENT;
    if ((st = validate_pfield(num_particles, x_p, PICASSO_F64))) return st;
    if ((st = validate_gfield(u_i, PICASSO_F64, PICASSO_F32))) return st;
    if ((st = validate_pfield(num_particles, c_p, u_i.dtype))) return st;
    BinP bins;
    if (key_tile) {
        int64_t ntiles = 0;
        if ((st = make_binp(sd, key_tile, &bins, &ntiles))) return st;
        if (num_particles > 0 && !key_out) return PICASSO_ERR_INVALID_ARGUMENT;
    }
    if (num_particles == 0) return PICASSO_OK;
    const bool f32 = u_i.dtype == PICASSO_F32;
    cudaStream_t s = stream_of(exec);
    int* err = exec ? exec->error_count : nullptr;
    PField x = make_pfield(x_p), c = make_pfield(c_p);
    GField u = make_gfield(u_i);
    Advect adv;
    if (dt) adv = make_advect(sd->mesh, *dt);
    if (dt && key_tile) {
        adv.key_out = key_out;
        adv.bins = bins;
    }
    const Advect* ap = dt ? &adv : nullptr;
    if (exec && exec->bins) {
        if (exec->bins->order != sd->order || exec->bins->location != sd->location)
            return PICASSO_ERR_INVALID_ARGUMENT;
        bool handled = false;
        st = apic_g2p_tiled(mp, sd->order, ncomp, f32, num_particles, x, u, c, *exec->bins, err,
                            ap, s, &handled, stag);
        if (st || handled) return st;
        TileP tp;
        if (!f32 && stag < 0 && ncomp == 3 && make_tilep(mp, sd->order, *exec->bins, num_particles, &tp)) {
            PB_ORDER_SWITCH(sd->order, st = launch_g2p_tiled_f64<O_>(mp, tp, num_particles, x, u, c,
                                                                     err, ap, s, &handled));
            if (st || handled) return st;
        }
    }
    return apic_g2p_plain(mp, sd->order, stag, ncomp, f32, num_particles, x, u, c, err, ap, s);
}

extern "C" picasso_status picasso_apic_g2p(const picasso_spline* sd, int64_t num_particles,
                                           int32_t ncomp, picasso_particle_field x_p,
                                           picasso_grid_field u_i, picasso_particle_field c_p,
                                           const picasso_exec* exec)
{
    return apic_g2p_entry(sd, num_particles, ncomp, x_p, u_i, c_p, nullptr, exec);
}

extern "C" picasso_status picasso_apic_g2p_advect(const picasso_spline* sd,
                                                  int64_t num_particles,
                                                  picasso_particle_field x_p,
                                                  picasso_grid_field u_i,
                                                  picasso_particle_field c_p, double dt,
                                                  const picasso_exec* exec)
{
    return apic_g2p_entry(sd, num_particles, 3, x_p, u_i, c_p, &dt, exec);
}

extern "C" picasso_status picasso_apic_g2p_advect_keys(const picasso_spline* sd,
                                                       int64_t num_particles,
                                                       picasso_particle_field x_p,
                                                       picasso_grid_field u_i,
                                                       picasso_particle_field c_p, double dt,
                                                       const int32_t tile[3], uint32_t* key_out,
                                                       const picasso_exec* exec)
{
    if (!tile) return PICASSO_ERR_INVALID_ARGUMENT;
    return apic_g2p_entry(sd, num_particles, 3, x_p, u_i, c_p, &dt, exec, tile, key_out);
}
