// aa32.cuh -- node arithmetic of the FP32 in-place (AA) step shared by the launch-per-step kernels
// (flow_f32.cu) and the resident ones (flow_f32_resident.cu): the same operations in both, so the
// states they produce have the same bits.
#pragma once

#include "collide32.cuh"
#include "common.cuh"
#include "flow.h"
#include "lbgpu.h"

#include <cfloat>

namespace lbg {

// Moments (with F/2 when fm) and collision (forced when fc) of one node's 19 deviations.
template <int FMASK>
__device__ __forceinline__ void aa_relax(float (&f)[Q], const FlowArgs32 &a, int fm, int fc)
{
    float drho = 0.0f, jx = 0.0f, jy = 0.0f, jz = 0.0f;
    static_for<0, Q>([&](auto L) {
        constexpr int l = decltype(L)::value;
        constexpr Vel c = vel(l);
        drho += f[l];
        if constexpr (c.x > 0) jx += f[l];
        if constexpr (c.x < 0) jx -= f[l];
        if constexpr (c.y > 0) jy += f[l];
        if constexpr (c.y < 0) jy -= f[l];
        if constexpr (c.z > 0) jz += f[l];
        if constexpr (c.z < 0) jz -= f[l];
    });
    if (FMASK && fm) {
        jx = __fadd_rn(jx, __fmul_rn(0.5f, a.F[0]));
        jy = __fadd_rn(jy, __fmul_rn(0.5f, a.F[1]));
        jz = __fadd_rn(jz, __fmul_rn(0.5f, a.F[2]));
    }
    collide_dev<FMASK>(f, drho, jx, jy, jz, a, fc != 0);
}

// j of 19 FP32 deviations as doubles, each sum formed exactly in 64-bit integers and rounded once: a
// deviation is its 24-bit significand shifted to a grid 33 bits below the largest one's (57 bits,
// and the ten terms of a sum stay below 2^61); what lies below the grid is finer than the last bit
// of a double of the largest deviation's size, so the sum is at least as accurate as FP64 additions
// one by one.  Those would occupy the FP64 pipe, 19 SM cycles per warp instruction (16 per
// conversion): 18 conversions and 30 additions, about 860 cycles per 32 nodes, against about 100 of
// integer work here.
__device__ __forceinline__ void exact_flux(const float (&f)[Q], double &jx, double &jy, double &jz)
{
    int emax = 1;
#pragma unroll
    for (int l = 1; l < Q; ++l) emax = max(emax, (int)((__float_as_uint(f[l]) >> 23) & 255u));
    long long X = 0, Y = 0, Z = 0;
    static_for<1, Q>([&](auto L) {
        constexpr int l = decltype(L)::value;
        constexpr Vel c = vel(l);
        const unsigned b = __float_as_uint(f[l]);
        const int e = (int)((b >> 23) & 255u);
        const unsigned m = (b & 0x7fffffu) | (e ? 0x800000u : 0u);   // a denormal has no leading 1
        const int up = 33 - (emax - max(e, 1));                      // <= 33
        const long long v = up >= 0 ? (long long)((unsigned long long)m << up) : (long long)(m >> min(-up, 31));
        const long long d = (int)b < 0 ? -v : v;
        if constexpr (c.x > 0) X += d;
        if constexpr (c.x < 0) X -= d;
        if constexpr (c.y > 0) Y += d;
        if constexpr (c.y < 0) Y -= d;
        if constexpr (c.z > 0) Z += d;
        if constexpr (c.z < 0) Z -= d;
    });
    // one unit of the sums is 2^(emax - 33 - 150) (emax = 255: a non-finite deviation, reported
    // by the caller); the scaling adds to the exponent of the (normal) double
    auto scaled = [&](long long v) {
        const double r = (double)v;
        return v == 0 ? 0.0 : __hiloint2double(__double2hiint(r) + (emax - 183) * (1 << 20), __double2loint(r));
    };
    jx = scaled(X);
    jy = scaled(Y);
    jz = scaled(Z);
}

// n < 0 and non-finite bits of one node's deviations (FlowArgs32::neg_below).
__device__ __forceinline__ unsigned check_dev19(const float (&f)[Q], const FlowArgs32 &a)
{
    bool neg = false, nonfinite = false;
    static_for<0, Q>([&](auto L) {
        constexpr int l = decltype(L)::value;
        neg |= f[l] < a.neg_below[wclass(l)];
        nonfinite |= !(fabsf(f[l]) <= FLT_MAX);
    });
    return (neg ? (unsigned)LBGPU_ERR_NEGATIVE_POPULATION : 0u) | (nonfinite ? (unsigned)LBGPU_ERR_NONFINITE : 0u) |
           a.bad_rho0;
}

// |j - j_old|'s largest component as the bits of a non-negative double, whose order is that of
// their bits; a NaN difference (of a non-finite first state) counts as infinite.
__device__ __forceinline__ unsigned long long flux_change_bits(double dx, double dy, double dz)
{
    const unsigned long long b =
        (unsigned long long)__double_as_longlong(max_nonneg(max_nonneg(fabs(dx), fabs(dy)), fabs(dz)));
    return b > 0x7ff0000000000000ull ? 0x7ff0000000000000ull : b;
}

// The decision of the FP32 reference loop for the state S_t of step t = c.t (equilibration.f90:
// 339-489): l2err history, convergence at l2err <= target_error and t > 2, f_ext from the next
// collision on at the first convergence, exit at the second, the step cap.  Unlike the FP64 fused
// step no step is repeated: the decision is taken before S_t is collided (or, where it was
// collided ahead of the decision, that collision is undone).  st: status bits of the check;
// phase: AA phase of S_t.
__device__ __forceinline__ void decide32(FlowCtl &c, unsigned long long err_bits, unsigned st, int phase, double *hist)
{
    const double l2 = __longlong_as_double((long long)err_bits);
    const int t = c.t;
    bool finish = false;
    if (st & (LBGPU_ERR_NEGATIVE_POPULATION | LBGPU_ERR_NONFINITE)) {
        finish = true;
    } else {
        if (hist && t - 1 < c.hist_cap) hist[t - 1] = l2;
        c.last_l2err = l2;
        if (l2 <= c.target_error && t > 2) {
            if (!c.conv_without) {
                c.conv_without = 1;
                c.aa_fc = 1;          // f_ext acts from the collision of step t+1 on
            } else {
                c.conv_with = 1;
                finish = true;
            }
        }
    }
    c.exit_force_moment = c.check_fm;
    c.exit_step = t;
    c.exit_phase = phase;
    c.aa_fm = c.check_fm;         // moment force of S_t
    c.check_fm = c.aa_fc;         // S_{t+1} = collide(S_t) with aa_fc: its moments carry it
    c.t = t + 1;
    c.status |= st;
    if (!finish && c.max_steps > 0 && t >= c.max_steps) {
        finish = true;
        c.status |= (unsigned)LBGPU_ERR_STEP_CAP;
    }
    if (finish) c.done = 1;
}

}  // namespace lbg
