// Spline dispatch by arithmetic type and APIC constants shared by the plain
// and tiled transfer kernels.
#pragma once

#include <type_traits>

#include "common.cuh"

namespace pb {

// Storage / arithmetic form of a P2G call: all FP64 with FP64 atomics; FP32
// particles with 64-bit fixed-point grid; FP64 particles with fixed-point grid.
enum class Form { F64, F32Fixed, F64Fixed };

// FP64 arithmetic follows the oracle's expressions; reduced precision forms
// the weights from the in-cell fraction (see spline_eval_frac).
template <int ORDER, class R>
__device__ __forceinline__ void eval_spline(double x, double lo, double dx, double rdx,
                                            Spline1D<ORDER, R>& sp)
{
    if constexpr (std::is_same<R, double>::value)
        spline_eval_f64<ORDER>(x, lo, dx, rdx, sp);
    else
        spline_eval_frac<ORDER, R>(x, lo, dx, rdx, sp);
}

// APIC inertial tensor scaling D_p^-1 (Picasso_APIC.hpp:33-47): 4/dx^2 for
// quadratic, 3/dx^2 for cubic splines, from the first dimension's cell size.
template <int ORDER, class R>
__device__ __forceinline__ R inertial_scaling(double dx0)
{
    return (R)((ORDER == 2 ? 4.0 : 3.0) / (dx0 * dx0));
}

// Exponent and leading bits of |v|: kNotFinite and above for infinities and NaN.
__device__ __forceinline__ unsigned high_bits(double v)
{
    return (unsigned)__double2hiint(v) << 1;
}
constexpr unsigned kNotFinite = 0xFFE00000u;

// First stencil node of a particle along d, counted from the owned box in a
// periodic dimension; false if the stencil leaves a non-periodic mesh.
template <int K>
__device__ __forceinline__ bool stencil_start(const MeshP& mp, int d, int s0, int& r)
{
    if (!mp.periodic[d]) {
        r = s0;
        return s0 >= 0 && s0 <= mp.ext[d] - K;
    }
    const int n = mp.own_n[d];
    r = s0 - mp.own_lo[d];
    if (r < 0) r += n;         // one period covers every particle inside or
    else if (r >= n) r -= n;   // next to the owned box
    if ((unsigned)r >= (unsigned)n) {
        r %= n;
        if (r < 0) r += n;
    }
    return true;
}

// Bitonic sort of a warp's (stencil, lane) pairs: bits 0-4 of the result are the
// lane whose stencil has this lane's rank; lanes that are not live come last.
// (Stencils 2^27 apart in the linear index may compare equal: callers only use
// the order to bring equal stencils together.)
__device__ __forceinline__ unsigned warp_sort_by_stencil(bool live, unsigned linear)
{
    const unsigned lane = threadIdx.x & 31;
    unsigned key = live ? (linear << 5) | lane : 0xFFFFFFE0u | lane;
#pragma unroll
    for (unsigned size = 2; size <= 32; size *= 2)
#pragma unroll
        for (unsigned st = size / 2; st > 0; st /= 2) {
            const unsigned other = __shfl_xor_sync(0xFFFFFFFFu, key, st);
            const bool up = (lane & size) == 0 || size == 32;
            key = ((lane & st) == 0) == up ? min(key, other) : max(key, other);
        }
    return key;
}

// Select element `sel` of a small register array without dynamic indexing.
template <int N, class R>
__device__ __forceinline__ R select(const R (&v)[N], int sel)
{
    R r = v[0];
#pragma unroll
    for (int q = 1; q < N; ++q)
        if (q == sel) r = v[q];
    return r;
}

}  // namespace pb
