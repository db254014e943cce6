// flow64.cuh -- node arithmetic of the FP64 flow (strict and fused), for translation units compiled
// with -fmad=false: shared by the kernels that launch once per step (flow_f64.cu) and the resident
// ones (flow_f64_resident.cu), so that their states have the same bits.
#pragma once

#include <type_traits>

#include "common.cuh"
#include "flow.h"
#include "lbgpu.h"

namespace lbg {

// (cx*x + cy*y) + cz*z with the zero-velocity terms left out (c = +-1 terms are exact).
template <int CX, int CY, int CZ>
__device__ __forceinline__ double dotc(double x, double y, double z)
{
    const double tx = CX > 0 ? x : -x, ty = CY > 0 ? y : -y, tz = CZ > 0 ? z : -z;
    if constexpr (CX != 0 && CY != 0 && CZ != 0) return (tx + ty) + tz;
    else if constexpr (CX != 0 && CY != 0) return tx + ty;
    else if constexpr (CX != 0 && CZ != 0) return tx + tz;
    else if constexpr (CY != 0 && CZ != 0) return ty + tz;
    else if constexpr (CX != 0) return tx;
    else if constexpr (CY != 0) return ty;
    else if constexpr (CZ != 0) return tz;
    else return 0.0;
}

template <int SIGN>
__device__ __forceinline__ double addsgn(double s, double t)
{
    if constexpr (SIGN > 0) return s + t;
    else if constexpr (SIGN < 0) return s - t;
    else return s;
}

// the quarter of the velocities that collides velocity l where four warps share a node
__host__ __device__ constexpr int role_of(int l)
{
    return l < 7 ? 0 : (vel(l).z == 0 ? 1 : (vel(l).y == 0 ? 2 : 3));
}

// module_collision.f90:77-108 for one fluid node, all 19 velocities.
// FMASK: which components of the force are non-zero (bit 0 x, 1 y, 2 z); 0 = no force.
// UCF: the force is the launch-uniform f_ext and c_l.F is taken from a.cf.
// FORM, by the relaxation time: FORM_TAU1, tau = 1 (c1 = 0, c2 = 1, c3 = 1/2), the reference's
// default; FORM_POW2, c1 = 1 - 1/tau a power of two in magnitude (tau = 0.8, 2/3, 4/3, 2, ..), so
// that c1 n is exact; FORM_ANY.
//
// The step is bound by the FP64 pipe (one warp instruction per 19 cycles of an SM), so what counts
// is the number of FP64 instructions.  Every rounding of the reference is kept, but a product that
// is exact needs no rounding of its own: scaling by a power of two is exact, and a fused
// multiply-add of an exact product rounds where the reference's separate addition does.  With the
// reference's weights a2 = 1/4, 1/8 and 2 a2 = 1/2, 1/4 (axis, diagonal), so
//   x + a2 S              = fma(a2, S, x)
//   (2 a2 cu) cF + x      = fma(2 a2, cu cF, x)      cu cF formed once per pair (both change sign)
// and a1 and 2 a2 of a diagonal link are half of an axis link's, so T of a diagonal link is half
// of the same expression with the axis constants (c3 T = (c3/2) (2 T)).  With FORM_POW2 also
//   c1 n + c2 neq         = fma(c1, n, c2 neq)
// and with FORM_TAU1 that without c2 and x + c3 T = fma(c3, T, x).
// (Exact unless a value falls below the smallest normal double.)  The step of a porous medium
// issues 334 FP64 instructions per node in the term-by-term form and 405 us for 0.52 M fluid nodes
// (tau 0.8, loop); 287 and 319 us so far; with the sums and divisions in integers (moments19_units,
// velocity) 231 and 261 us, with FORM_POW2 212 and 237 us, 88 % of the pipe.
// ROLE: every velocity (-1), or a quarter of them: 0 the rest and axis velocities, 1 / 2 / 3 the
// diagonals of the xy / xz / yz planes (role_of).
template <int FMASK, bool UCF, int FORM, int ROLE = -1>
__device__ __forceinline__ void collide_node(double (&n)[Q], const double rho, const double jx,
                                             const double jy, const double jz, const double ux,
                                             const double uy, const double uz, const double fx,
                                             const double fy, const double fz,
                                             const FlowArgs64 &a)
{
    const LbConst64 &K = a.K;
    const double Pxx = jx * ux, Pxy = jx * uy, Pxz = jx * uz;
    const double Pyx = jy * ux, Pyy = jy * uy, Pyz = jy * uz;
    const double Pzx = jz * ux, Pzy = jz * uy, Pzz = jz * uz;
    const double Dx1 = Pxx * K.k1, Dx0 = Pxx * K.k0;
    const double Dy1 = Pyy * K.k1, Dy0 = Pyy * K.k0;
    const double Dz1 = Pzz * K.k1, Dz0 = Pzz * K.k0;
    const double ar[3] = {K.a0[0] * rho, K.a0[1] * rho, K.a0[2] * rho};
    // (c_a - u_a) * f_a for c_a = 0, +1, -1
    double gx0 = 0, gxp = 0, gxm = 0, gy0 = 0, gyp = 0, gym = 0, gz0 = 0, gzp = 0, gzm = 0;
    if constexpr (FMASK & 1) { gx0 = (-ux) * fx; gxp = (1.0 - ux) * fx; gxm = (-1.0 - ux) * fx; }
    if constexpr (FMASK & 2) { gy0 = (-uy) * fy; gyp = (1.0 - uy) * fy; gym = (-1.0 - uy) * fy; }
    if constexpr (FMASK & 4) { gz0 = (-uz) * fz; gzp = (1.0 - uz) * fz; gzm = (-1.0 - uz) * fz; }
    // a2 term: jx*ux*(cx^2-cs^2) + jx*uy*cx*cy + ... + jz*uz*(cz^2-cs^2), even in c
    auto a2_sum = [&](auto CX, auto CY, auto CZ) {
        constexpr int cx = decltype(CX)::value, cy = decltype(CY)::value, cz = decltype(CZ)::value;
        double S = cx != 0 ? Dx1 : Dx0;
        S = addsgn<cx * cy>(S, Pxy);
        S = addsgn<cx * cz>(S, Pxz);
        S = addsgn<cy * cx>(S, Pyx);
        S = S + (cy != 0 ? Dy1 : Dy0);
        S = addsgn<cy * cz>(S, Pyz);
        S = addsgn<cz * cx>(S, Pzx);
        S = addsgn<cz * cy>(S, Pzy);
        return S + (cz != 0 ? Dz1 : Dz0);
    };
    // c1 n + c2 neq + c3 T of direction l, T = a1*((cx-ux)*fx + (cy-uy)*fy + (cz-uz)*fz)
    // + 2*a2*(c.u)*(c.f), cucf = (c.u)*(c.f)
    auto relax = [&](auto L, double neq, double cucf) {
        constexpr int l = decltype(L)::value;
        constexpr Vel c = vel(l);
        constexpr int w = wclass(l);
        double r = FORM == FORM_TAU1   ? __fma_rn(K.c1, n[l], neq)
                   : FORM == FORM_POW2 ? __fma_rn(K.c1, n[l], K.c2 * neq)
                                       : K.c1 * n[l] + K.c2 * neq;
        if constexpr (FMASK != 0) {
            double t1 = 0.0;
            if constexpr (FMASK & 1) t1 = c.x > 0 ? gxp : (c.x < 0 ? gxm : gx0);
            if constexpr (FMASK & 2) {
                const double g = c.y > 0 ? gyp : (c.y < 0 ? gym : gy0);
                if constexpr (FMASK & 1) t1 = t1 + g;
                else t1 = g;
            }
            if constexpr (FMASK & 4) {
                const double g = c.z > 0 ? gzp : (c.z < 0 ? gzm : gz0);
                if constexpr (FMASK & 3) t1 = t1 + g;
                else t1 = g;
            }
            // T (rest, axis), 2 T (diagonal); a1 of the rest velocity is 1
            double T = l == 0 ? t1 : K.a1[1] * t1;
            constexpr bool hasT2 = ((FMASK & 1) && c.x != 0) || ((FMASK & 2) && c.y != 0) ||
                                   ((FMASK & 4) && c.z != 0);
            if constexpr (hasT2) T = __fma_rn(K.two_a2[1], cucf, T);
            const double k3 = w == 2 ? K.c3h : K.c3;
            r = FORM == FORM_TAU1 ? __fma_rn(k3, T, r) : r + k3 * T;
        }
        n[l] = r;
    };
    if constexpr (ROLE <= 0) relax(std::integral_constant<int, 0>{},
          ar[0] + K.a2[0] * a2_sum(std::integral_constant<int, 0>{}, std::integral_constant<int, 0>{},
                                   std::integral_constant<int, 0>{}),
          0.0);
    static_for<0, 9>([&](auto P) {
        constexpr int l = pair_l(decltype(P)::value);
        if constexpr (ROLE >= 0 && ROLE != role_of(l)) return;
        constexpr int li = inv(l);
        constexpr Vel c = vel(l);
        constexpr int w = wclass(l);
        const double S = a2_sum(std::integral_constant<int, c.x>{}, std::integral_constant<int, c.y>{},
                                std::integral_constant<int, c.z>{});
        const double a1cj = K.a1[w] * dotc<c.x, c.y, c.z>(jx, jy, jz);
        double cucf = 0.0;
        if constexpr (FMASK != 0) {
            double cfl;
            if constexpr (UCF) cfl = a.cf[l];
            else cfl = dotc<(FMASK & 1) ? c.x : 0, (FMASK & 2) ? c.y : 0, (FMASK & 4) ? c.z : 0>(fx, fy, fz);
            cucf = dotc<c.x, c.y, c.z>(ux, uy, uz) * cfl;
        }
        relax(std::integral_constant<int, l>{}, __fma_rn(K.a2[w], S, ar[w] + a1cj), cucf);
        relax(std::integral_constant<int, li>{}, __fma_rn(K.a2[w], S, ar[w] - a1cj), cucf);
    });
}

// The same for a force switched on or off at run time, in the form of the box's relaxation time.
template <int FMASK, bool UCF, int ROLE = -1>
__device__ __forceinline__ void collide_strict_u(double (&n)[Q], const double rho, const double jx, const double jy,
                                                 const double jz, const double ux, const double uy, const double uz,
                                                 const double fx, const double fy, const double fz,
                                                 const FlowArgs64 &a, const bool force)
{
    auto collide = [&](auto F) {
        constexpr int form = decltype(F)::value;
        if (force) collide_node<FMASK, UCF, form, ROLE>(n, rho, jx, jy, jz, ux, uy, uz, fx, fy, fz, a);
        else collide_node<0, true, form, ROLE>(n, rho, jx, jy, jz, ux, uy, uz, 0.0, 0.0, 0.0, a);
    };
    if (a.K.form == FORM_TAU1) collide(std::integral_constant<int, FORM_TAU1>{});
    else if (a.K.form == FORM_POW2) collide(std::integral_constant<int, FORM_POW2>{});
    else collide(std::integral_constant<int, FORM_ANY>{});
}

// j / rho with the rounding of an IEEE division, on the integer pipes: a division is some ten
// dependent FP64 instructions of 19 SM cycles a warp, this some 15 cycles, and the three of a node
// share one reciprocal.  Long division of the mantissas: with r = 2^125 / R (R, J the mantissas at bit
// 62) the quotient's first 54 bits M = floor are those of J r / 2^64 or one off, the remainder
// J 2^k - M R (exact modulo 2^64) puts M right, and M's last bit with the remainder rounds to nearest
// even.  Arguments outside 2^-500 .. 2^500 in magnitude (0 apart), or a rho <= 0, are divided in FP64:
// within, the quotient is a normal number, as its exponent put together here must be.
__device__ __forceinline__ bool div_range(double x)
{
    const unsigned e = ((unsigned)__double2hiint(x) >> 20) & 0x7ffu;
    return e - 523u < 1000u;
}

__device__ __forceinline__ bool is_zero(double x)
{
    return ((unsigned)__double2hiint(x) << 1 | (unsigned)__double2loint(x)) == 0u;
}

__device__ __forceinline__ unsigned long long mantissa53(double x)
{
    return ((unsigned long long)(((unsigned)__double2hiint(x) & 0xfffffu) | 0x100000u) << 32) | (unsigned)__double2loint(x);
}

// 2^125 / R: the reciprocal of R's leading 24 bits in FP32, then two Newton-Raphson steps
// r <- r + r (1 - R r), each of which doubles the bits that are right (to 44, then to some 59)
__device__ __forceinline__ unsigned long long recip125(unsigned long long R)
{
    const unsigned q = __float_as_uint(__frcp_rn((float)(unsigned)(R >> 39)));
    unsigned long long r = (unsigned long long)((q & 0x7fffffu) | 0x800000u) << ((q >> 23) - 64u);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const long long e = (long long)((1ull << 61) - __umul64hi(R, r));
        r += (unsigned long long)__mul64hi((long long)(r >> 1), e << 4);
    }
    return r;
}

__device__ __forceinline__ double div_recip(double j, double rho, unsigned long long r)
{
    const unsigned long long Rm = mantissa53(rho), Jm = mantissa53(j);
    const unsigned hj = (unsigned)__double2hiint(j), hr = (unsigned)__double2hiint(rho);
    const bool below = Jm < Rm;
    unsigned long long M = __umul64hi(Jm << 10, r) >> (below ? 7 : 8);
    long long rem = (long long)((Jm << (below ? 54 : 53)) - M * Rm);
    if (rem < 0) {
        --M;
        rem += (long long)Rm;
    } else if (rem >= (long long)Rm) {
        ++M;
        rem -= (long long)Rm;
    }
    const unsigned lo = (unsigned)M, up = lo & 1u & (unsigned)(rem != 0 || (lo & 2u));
    const unsigned e = 1022u + ((hj >> 20) & 0x7ffu) - (hr >> 20) - (below ? 1u : 0u);
    const unsigned long long bits = ((unsigned long long)(e << 20 | (hj & 0x80000000u)) << 32) + ((M >> 1) + up);
    return is_zero(j) ? j : __longlong_as_double((long long)bits);
}

// one quotient, for the threads that share a node
__device__ __forceinline__ double divide(double j, double rho)
{
    if (__double2hiint(rho) >= 0 && div_range(rho) && (div_range(j) || is_zero(j)))
        return div_recip(j, rho, recip125(mantissa53(rho) << 10));
    return j / rho;
}

__device__ __forceinline__ void velocity(double jx, double jy, double jz, double rho, double &ux, double &uy, double &uz)
{
    auto fits = [](double j) { return div_range(j) || is_zero(j); };
    if (__double2hiint(rho) >= 0 && div_range(rho) && fits(jx) && fits(jy) && fits(jz)) {
        const unsigned long long r = recip125(mantissa53(rho) << 10);
        ux = div_recip(jx, rho, r);
        uy = div_recip(jy, rho, r);
        uz = div_recip(jz, rho, r);
    } else {
        ux = jx / rho;
        uy = jy / rho;
        uz = jz / rho;
    }
}

template <int FMASK, bool UCF>
__device__ __forceinline__ void collide_strict(double (&n)[Q], const double rho, const double jx, const double jy,
                                               const double jz, const double fx, const double fy, const double fz,
                                               const FlowArgs64 &a, const bool force)
{
    double ux, uy, uz;
    velocity(jx, jy, jz, rho, ux, uy, uz);
    collide_strict_u<FMASK, UCF>(n, rho, jx, jy, jz, ux, uy, uz, fx, fy, fz, a, force);
}

// LBGPU_FP64_FUSED: density and flux from the pair sums and differences of opposite velocities
// (n_l + n_inv l, n_l - n_inv l): fewer FP64 additions than the term-by-term sums of moments19.
__device__ __forceinline__ void moments19_pairs(const double (&n)[Q], double fhx, double fhy, double fhz,
                                                double &rho, double &jx, double &jy, double &jz)
{
    double r = n[0], X = fhx, Y = fhy, Z = fhz;
    static_for<0, 9>([&](auto P) {
        constexpr int l = pair_l(decltype(P)::value);
        constexpr int li = inv(l);
        constexpr Vel c = vel(l);
        r = r + (n[l] + n[li]);
        const double d = n[l] - n[li];
        X = addsgn<c.x>(X, d);
        Y = addsgn<c.y>(Y, d);
        Z = addsgn<c.z>(Z, d);
    });
    rho = r;
    jx = X;
    jy = Y;
    jz = Z;
}

// LBGPU_FP64_FUSED: the same BGK + Guo collision regrouped per pair of opposite velocities
// (l, inv l), where c.j, c.u and c.F change sign and nothing else does:
//   n_l   <- c1 n_l   + (E + O),   n_inv <- c1 n_inv + (E - O)
//   E = c2 [a0 rho + a2 ((c.j)(c.u) - cs^2 j.u)] + c3 [2 a2 (c.u)(c.F) - a1 u.F]
//   O = c2 a1 (c.j) + c3 a1 (c.F)
// evaluated with fused multiply-adds and one reciprocal of rho: about half the FP64 operations
// of the operation-for-operation form, which bounds this kernel on GB300's FP64 pipe.  UCF: the
// uniform f_ext, with c3 a1 (c.F) and c3 2 a2 (c.F) taken per pair from a.kF / a.kT.
template <int FMASK, bool UCF>
__device__ __forceinline__ void collide_node_fused(double (&n)[Q], const double rho, const double jx,
                                                   const double jy, const double jz, const double fx,
                                                   const double fy, const double fz,
                                                   const FlowArgs64 &a)
{
    const LbConst64 &K = a.K;
    const double ir = 1.0 / rho;
    const double ux = jx * ir, uy = jy * ir, uz = jz * ir;
    const double ju = __fma_rn(jx, ux, __fma_rn(jy, uy, jz * uz));
    double base[3];
#pragma unroll
    for (int w = 0; w < 3; ++w) base[w] = __fma_rn(K.c2a0[w], rho, -(K.c2a2cs2[w] * ju));
    if constexpr (FMASK != 0) {
        const double uF = __fma_rn(ux, fx, __fma_rn(uy, fy, uz * fz));
#pragma unroll
        for (int w = 0; w < 3; ++w) base[w] = __fma_rn(-K.c3a1[w], uF, base[w]);
    }
    n[0] = __fma_rn(K.c1, n[0], base[0]);
    static_for<0, 9>([&](auto P) {
        constexpr int p = decltype(P)::value;
        constexpr int l = pair_l(p);
        constexpr int li = inv(l);
        constexpr Vel c = vel(l);
        constexpr int w = wclass(l);
        const double cj = dotc<c.x, c.y, c.z>(jx, jy, jz);
        const double cu = dotc<c.x, c.y, c.z>(ux, uy, uz);
        double A = __fma_rn(K.c2a2[w], cj * cu, base[w]);
        double B = K.c2a1[w] * cj;
        if constexpr (FMASK != 0) {
            double kT, kF;
            if constexpr (UCF) {
                kT = a.kT[p];
                kF = a.kF[p];
            } else {
                const double cF = dotc<c.x, c.y, c.z>(fx, fy, fz);
                kT = (K.c3 * K.two_a2[w]) * cF;
                kF = K.c3a1[w] * cF;
            }
            A = __fma_rn(kT, cu, A);
            B = B + kF;
        }
        n[l] = __fma_rn(K.c1, n[l], A + B);
        n[li] = __fma_rn(K.c1, n[li], A - B);
    });
}

// ---- LBGPU_FP64_FUSED in 64-bit fixed point
//
// The FP64 pipe issues one warp instruction per 19 cycles of an SM, a 64-bit integer addition takes
// 0.3 and the high half of a 64 x 64-bit product 4.4, and the integer pipes are otherwise idle here.
// So the fused step of an ordinary node runs in fixed point: its populations become integers on a
// grid 60 bits below the largest one's binade (exact while they are within 2^7 of it, to nearest
// below), moments are exact integer sums, and each result is rounded once to a
// double.  j and what is made of it carry 3 more bits, so that the rounding down of a product's high
// half leaves no bias worth a tenth of a unit (a bias in j, unlike a random error, adds up like a
// force).  With c at the scale of a diagonal link (a0 = 1/36, a1 = 1/12, a2 = 1/8;
// an axis link has twice each, the rest velocity 12 times a0), per pair of opposite velocities:
//   H = c2 j/8 + c3 F/4,  b = (c2 j + c3 F)/12,  Q = sum_a u_a H_a,  base = c2 rho/36 - Q/3
//   n'(l, inv l) = [c1 s/2 + base + (c.u)(c.H)] +- [c1 d/2 + c.b],   s, d = n_l +- n_inv
// the same regrouping as collide_node_fused's.  (c.u)(c.H) of the two pairs of a plane comes from
// one product and the squares; the rest population takes what the others leave of rho.  The rounded
// constants of the FP64 form do not quite sum to 1 (at tau = 1 as the weights in the reference's
// code: 1/3 + 6/18 + 12/36 = 1 - 2^-54), so a step changes a node's mass by a fixed share of it: the
// rest population takes that too (fix_loss; 4e-13 of rho after 7000 steps, and the tracer sums
// depend on rho).  The axis pairs take what the diagonals leave of the flux, which a collision keeps
// apart from the force: rounded pair by pair instead, each a sixteenth of a unit too high on average,
// j's error against binary128 in a porous medium of 96^3 after 120 steps at tau 0.8 was 4.5e-13 of its
// norm across the force, where the FP64 form has 1.5e-13.  Nodes outside the fixed-point range -- a
// negative or non-finite
// population, the largest one below 2^-895, rho from 8 times the largest one's binade up, |j| from
// a quarter of it up, a force from a sixteenth of it up -- take the FP64 form.
// Porous medium of 128^3 (1.26 M fluid nodes), tau 0.8: 400 -> 135 us a step (57 us of HBM traffic;
// now bound by the integer pipes): 165 as first built, 140 in blocks of 128 threads, 134 with the
// short shifts of the common case and since the axis pairs take the rest of the flux (the loop's step 195).  Error of jx / jy / jz against binary128, force along x, each of its norm: porous medium of
// 96^3, tau 0.8, 120 steps 1.2e-14 / 2.9e-14 / 3.5e-14 where the FP64 form has 5.9e-14 / 1.4e-13 /
// 1.5e-13; 64^3, tau 0.62, 400 steps 0.6e-14 / 1.4e-14 / 1.6e-14 and 3.2e-14 / 7.8e-14 / 8.7e-14.

__device__ __forceinline__ long long mulhi(long long a, long long b) { return __mul64hi(a, b); }

// value of v units of 2^(emax - 1082), rounded to nearest even
__device__ __forceinline__ double fixed_to_double(long long v, int emax)
{
    const int hi = (int)(v >> 32);
    const int sh = 11 - __clz(hi);   // drops v to 53 bits
    if (hi <= 0 || sh < 1) {         // negative or small: by conversion, its exponent shifted
        if (v == 0) return 0.0;
        const double r = (double)v;
        return __hiloint2double(__double2hiint(r) + (emax - 1082) * (1 << 20), __double2loint(r));
    }
    const unsigned lo = (unsigned)v, half = 1u << (sh - 1);
    const unsigned long long m = ((unsigned long long)v + (half - 1u) + ((lo >> sh) & 1u)) >> (sh & 15);   // sh is 1 .. 10
    // the leading 1 of m adds one to the exponent field
    return __longlong_as_double((long long)(m + ((unsigned long long)(unsigned)(emax - 8 + sh) << 52)));
}

// j: units of 2^(emax - 1085), of either sign and any size
__device__ __forceinline__ double signed_fixed(long long v, int emax)
{
    const double r = (double)v;
    return v == 0 ? 0.0 : __hiloint2double(__double2hiint(r) + (emax - 1085) * (1 << 20), __double2loint(r));
}

// |x| for a comparison (a NaN or infinity compares above every finite bound as its bits do)
__device__ __forceinline__ unsigned long long fabs_bits(double x)
{
    return (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
}

// F in units of 2^(emax - 1085), to nearest; |F| must lie below the largest population's binade
__device__ __forceinline__ long long force_to_fixed(double F, int emax)
{
    const unsigned hi = (unsigned)__double2hiint(F), lo = (unsigned)__double2loint(F);
    const int e = (int)((hi >> 20) & 0x7ffu), sh = 10 - (emax - e);
    const unsigned long long m = ((unsigned long long)((hi & 0xfffffu) | (e ? 0x100000u : 0u)) << 32) | lo;
    const int down = min(-sh, 62);
    const long long v = (long long)(sh >= 0 ? m << sh : (m + (1ull << (down - 1))) >> down);
    return (int)hi < 0 ? -v : v;
}

// One fused step of a node: n, after streaming, becomes the collided populations.  Returns false,
// with n untouched, for a node outside the fixed-point range.  WANT_J: its j, as doubles.
template <int FMASK, bool WANT_J, bool FORMS>
__device__ __forceinline__ bool fused_fixed(double (&n)[Q], const bool fm, const bool fc, const double fx,
                                            const double fy, const double fz, const FlowArgs64 &a, double &ox,
                                            double &oy, double &oz)
{
    const LbConst64 &K = a.K;
    int emax = 0, emin = 0x7ff;
    unsigned sign = 0;
#pragma unroll
    for (int l = 0; l < Q; ++l) {
        const unsigned hi = (unsigned)__double2hiint(n[l]);
        sign |= hi;
        emax = max(emax, (int)(hi >> 20));
        emin = min(emin, (int)(hi >> 20));
    }
    if ((int)sign < 0 || emax >= 0x7ff || emax < 128) return false;
    long long v[Q];
    if (emin >= emax - 7) {   // as almost always: shifts of at most 7 to the left
#pragma unroll
        for (int l = 0; l < Q; ++l)
            v[l] = (long long)(mantissa53(n[l]) << ((7 - (emax - (__double2hiint(n[l]) >> 20))) & 7));
    } else {
#pragma unroll
        for (int l = 0; l < Q; ++l) {
            const int e = __double2hiint(n[l]) >> 20, sh = 7 - (emax - e);
            const unsigned long long m = mantissa53(n[l]);
            const int down = min(max(-sh, 1), 62);   // to nearest: cut off, small populations would lose mass
            v[l] = e == 0 ? 0ll : (long long)(sh >= 0 ? m << sh : (m + (1ull << (down - 1))) >> down);
        }
    }
    // rho in three parts that cannot overflow (each v < 2^60)
    const long long r0 = v[0] + v[1] + v[2] + v[3] + v[4] + v[5] + v[6];
    const long long r1 = v[7] + v[8] + v[9] + v[10] + v[11] + v[12];
    const long long r2 = v[13] + v[14] + v[15] + v[16] + v[17] + v[18];
    const long long R = r0 + r1 + r2;
    constexpr long long LO = 1ll << 59, HI = 1ll << 62;
    if (r0 >= HI || r1 >= HI / 2 || r2 >= HI / 2 || R < LO || R >= HI) return false;
    long long jx = 0, jy = 0, jz = 0, gx = 0, gy = 0, gz = 0, sx = 0, sy = 0, sz = 0;
    if constexpr (FMASK != 0) {
        if (fm || fc) {
            // a force of the populations' size lies outside the range
            const unsigned long long big = (unsigned long long)(unsigned)(emax - 4) << 52;
            if (fabs_bits(fx) >= big || fabs_bits(fy) >= big || fabs_bits(fz) >= big) return false;
            if constexpr (FMASK & 1) gx = force_to_fixed(fx, emax);
            if constexpr (FMASK & 2) gy = force_to_fixed(fy, emax);
            if constexpr (FMASK & 4) gz = force_to_fixed(fz, emax);
            if (fm) {
                jx = (gx + 1) >> 1;
                jy = (gy + 1) >> 1;
                jz = (gz + 1) >> 1;
            }
        }
    }
    static_for<0, 9>([&](auto P) {
        constexpr int l = pair_l(decltype(P)::value);
        constexpr Vel c = vel(l);
        const long long s = v[l] + v[inv(l)], d = v[l] - v[inv(l)];
        v[l] = s;
        v[inv(l)] = d;
        if constexpr (c.x != 0) sx += c.x > 0 ? d : -d;
        if constexpr (c.y != 0) sy += c.y > 0 ? d : -d;
        if constexpr (c.z != 0) sz += c.z > 0 ? d : -d;
    });
    constexpr unsigned long long JR = 1ull << 57;   // no sum wraps: every |d| < R < 2^62, all n >= 0
    if ((unsigned long long)(sx + (long long)JR) >= 2 * JR || (unsigned long long)(sy + (long long)JR) >= 2 * JR ||
        (unsigned long long)(sz + (long long)JR) >= 2 * JR)
        return false;
    jx += 8 * sx;   // in eighths of a unit, |j| < 2^61
    jy += 8 * sy;
    jz += 8 * sz;
    if constexpr (WANT_J) {
        ox = signed_fixed(jx, emax);
        oy = signed_fixed(jy, emax);
        oz = signed_fixed(jz, emax);
    }
    // r = 2^121 / R: the reciprocal of R's 32 leading bits in FP32, then two Newton-Raphson steps
    // r <- r + r (1 - R r), which double its 23 bits to 46 and to the product's 57
    const float q = __frcp_rn((float)(unsigned)(R >> 30));
    long long r = (long long)((unsigned long long)((__float_as_uint(q) & 0x7fffffu) | 0x800000u)
                              << ((__float_as_uint(q) >> 23) - 59u));
#pragma unroll
    for (int k = 0; k < 2; ++k) r += mulhi(r, ((1ll << 57) - mulhi(R, r)) << 7);
    const long long ux = mulhi(jx << 2, r), uy = mulhi(jy << 2, r), uz = mulhi(jz << 2, r);   // u 2^62
    // c2 j / 8, c3 F / 4 and all that follows in eighths of a unit
    const long long px = mulhi(jx, K.fix_c2), py = mulhi(jy, K.fix_c2), pz = mulhi(jz, K.fix_c2);
    long long fqx = 0, fqy = 0, fqz = 0;
    if constexpr (FMASK != 0) {
        if (fc) {
            if constexpr (FMASK & 1) fqx = mulhi(gx, K.fix_c3);
            if constexpr (FMASK & 2) fqy = mulhi(gy, K.fix_c3);
            if constexpr (FMASK & 4) fqz = mulhi(gz, K.fix_c3);
        }
    }
    constexpr long long THIRD = 0x2aaaaaaaaaaaaaabll;   // 2^63 / 3
    const long long hx = px + fqx, hy = py + fqy, hz = pz + fqz;
    const long long bx = mulhi((2 * px + fqx) * 2, THIRD), by = mulhi((2 * py + fqy) * 2, THIRD),
                    bz = mulhi((2 * pz + fqz) * 2, THIRD);
    const long long qx = mulhi(ux, hx * 4), qy = mulhi(uy, hy * 4), qz = mulhi(uz, hz * 4);
    const long long base = 2 * mulhi(R, K.fix_c2_36) - mulhi((qx + qy + qz) * 2, THIRD);
    const long long base_axis = 2 * base;
    long long rest = R - __mulhi((int)(R >> 31), K.fix_loss);
    // the flux after the collision, j - (c2/2) F + c3 F with j = sum c n + F/2: what streams in and F,
    // or the part of F that a step has whose moments or collision alone take it
    auto flux = [&](auto D, long long sum, long long g) {
        if constexpr (!(FMASK & decltype(D)::value)) {
            return sum;
        } else {
            if (!(fm || fc)) return sum;
            long long G = g;
            if (!(fm && fc)) {
                const long long h = mulhi(4 * g, K.fix_c2);   // c2 F / 2
                G = fm ? h : g - h;
            }
            return sum + ((G + (((int)sum >> 3) & 7)) >> 3);
        }
    };
    long long tx = flux(std::integral_constant<int, 1>{}, sx, gx), ty = flux(std::integral_constant<int, 2>{}, sy, gy),
              tz = flux(std::integral_constant<int, 4>{}, sz, gz);
    const long long mxy = mulhi(ux + uy, (hx + hy) * 4), mxz = mulhi(ux + uz, (hx + hz) * 4),
                    myz = mulhi(uy + uz, (hy + hz) * 4);
    // (s, d) of a pair in v[l], v[inv l] -> its collided populations e + o (+ odd) and e - o; A, B to
    // nearest, and half a unit more for the rounding down of the c1 products
    auto pairs = [&](const auto relax) {
        const long long half = relax ? 8 : 4;
        auto put = [&](auto P, long long e, long long o, int odd) {
            constexpr int l = pair_l(decltype(P)::value);
            rest -= 2 * e + odd;
            n[l] = fixed_to_double(e + o + odd, emax);
            n[inv(l)] = fixed_to_double(e - o, emax);
        };
        auto diagonal = [&](auto P, long long A, long long B) {
            constexpr int l = pair_l(decltype(P)::value);
            constexpr Vel c = vel(l);
            long long e = (A + half) >> 3, o = (B + half) >> 3;
            if (relax) {
                e += mulhi(v[l] * 2, K.fix_c1);
                o += mulhi(v[inv(l)] * 2, K.fix_c1);
            }
            if constexpr (c.x != 0) tx -= c.x > 0 ? 2 * o : -2 * o;
            if constexpr (c.y != 0) ty -= c.y > 0 ? 2 * o : -2 * o;
            if constexpr (c.z != 0) tz -= c.z > 0 ? 2 * o : -2 * o;
            put(P, e, o, 0);
        };
        // an axis pair takes what the diagonals leave of its flux t: n_l - n_inv l = 2 o + odd = t
        auto axis = [&](auto P, long long A, long long o, int odd) {
            long long e = (A + half) >> 3;
            if (relax) e += mulhi(v[pair_l(decltype(P)::value)] * 2, K.fix_c1);
            put(P, e, o, odd);
        };
        diagonal(std::integral_constant<int, 3>{}, base + mxy, bx + by);                        // (1, 1, 0)
        diagonal(std::integral_constant<int, 4>{}, base + 2 * (qx + qy) - mxy, by - bx);        // (-1, 1, 0)
        diagonal(std::integral_constant<int, 5>{}, base + mxz, bx + bz);                        // (1, 0, 1)
        diagonal(std::integral_constant<int, 6>{}, base + 2 * (qx + qz) - mxz, bz - bx);        // (-1, 0, 1)
        diagonal(std::integral_constant<int, 7>{}, base + myz, by + bz);                        // (0, 1, 1)
        diagonal(std::integral_constant<int, 8>{}, base + 2 * (qy + qz) - myz, bz - by);        // (0, -1, 1)
        axis(std::integral_constant<int, 0>{}, base_axis + 2 * qx, tx >> 1, (int)tx & 1);
        axis(std::integral_constant<int, 1>{}, base_axis + 2 * qy, ty >> 1, (int)ty & 1);
        axis(std::integral_constant<int, 2>{}, base_axis + 2 * qz, tz >> 1, (int)tz & 1);
    };
    // FORMS: no test of c1 at every pair, for the one warp of a quarter that a small box has (10 x 11 x 14
    // porous, tau 1, 800 steps: 3.38 ms against 3.55); a full device loses more by the registers of both
    // (three components of force 152 us a step against 150)
    if constexpr (FORMS) {
        if (K.fix_c1 != 0) pairs(std::true_type{});
        else pairs(std::false_type{});
    } else {
        pairs(K.fix_c1 != 0);
    }
    n[0] = fixed_to_double(rest, emax);
    return true;
}

// One fused step of a node, in fixed point or, outside its range, in FP64.
template <int FMASK, bool UCF, bool WANT_J, bool FORMS>
__device__ __forceinline__ void fused_step(double (&n)[Q], const bool fm, const bool fc, const double fx,
                                           const double fy, const double fz, const FlowArgs64 &a, double &jx,
                                           double &jy, double &jz)
{
    if (fused_fixed<FMASK, WANT_J, FORMS>(n, fm, fc, fx, fy, fz, a, jx, jy, jz)) return;
    double rho;
    if (fm) moments19_pairs(n, fx / 2.0, fy / 2.0, fz / 2.0, rho, jx, jy, jz);
    else moments19_pairs(n, 0.0, 0.0, 0.0, rho, jx, jy, jz);
    if (fc) collide_node_fused<FMASK, UCF>(n, rho, jx, jy, jz, fx, fy, fz, a);
    else collide_node_fused<0, true>(n, rho, jx, jy, jz, 0.0, 0.0, 0.0, a);
}

// density = SUM(n,4); j = F/2 + sum_l n_l c_l   (equilibration.f90:254,293-300)
__device__ __forceinline__ void moments19(const double (&n)[Q], double fhx, double fhy,
                                          double fhz, double &rho, double &jx, double &jy,
                                          double &jz)
{
    double r = n[0], X = fhx, Y = fhy, Z = fhz;
#pragma unroll
    for (int l = 1; l < Q; ++l) r = r + n[l];
    static_for<0, Q>([&](auto L) {
        constexpr int l = decltype(L)::value;
        constexpr Vel c = vel(l);
        X = addsgn<c.x>(X, n[l]);
        Y = addsgn<c.y>(Y, n[l]);
        Z = addsgn<c.z>(Z, n[l]);
    });
    rho = r;
    jx = X;
    jy = Y;
    jz = Z;
}

// The same sums, each addition with its FP64 rounding, in 64-bit integers: a DADD takes 19 SM cycles
// a warp, an integer addition rounded to 53 bits some 5.  The populations become integers 59 bits below
// the largest one's binade, exact while they lie within 2^7 of it; false (and nothing written) for a
// node with one outside, a negative or non-finite one, or a sum beyond 2^62 units.
__device__ __forceinline__ long long round53(long long t)
{
    const int hi = (int)(t >> 32);
    const int k = max(0, 11 - __clz(hi ^ (hi >> 31)));   // bits beyond 53 (a power of two may count one short: exact anyway)
    const unsigned lo = (unsigned)t, cut = ~(0xffffffffu << k);
    t += (long long)((cut >> 1) + ((lo >> k) & cut & 1u));
    return t & ~(long long)cut;
}

// t units, of at most 53 significant bits, as a double
__device__ __forceinline__ double from_units(long long t, int emax)
{
    const unsigned sign = (unsigned)(t >> 32) & 0x80000000u;
    const unsigned long long mag = (unsigned long long)(t < 0 ? -t : t);
    const int lz = __clzll((long long)mag);
    const unsigned long long m = (mag << (lz & 63)) >> 11;
    const unsigned long long bits = ((unsigned long long)((unsigned)(emax + 3 - lz) << 20 | sign) << 32) + m;
    return t == 0 ? 0.0 : __longlong_as_double((long long)bits);
}

__device__ __forceinline__ bool to_units(double x, int emax, long long &t)
{
    const unsigned hi = (unsigned)__double2hiint(x);
    const int down = emax - (int)((hi >> 20) & 0x7ffu);
    const long long m = (long long)(mantissa53(x) << ((7 - down) & 7));   // of use for down <= 7 only
    t = (int)hi < 0 ? -m : m;
    return (unsigned)down <= 7u;
}

__device__ __forceinline__ bool moments19_units(const double (&n)[Q], bool fm, double fhx, double fhy, double fhz,
                                                double &rho, double &jx, double &jy, double &jz)
{
    int emax = 0;
#pragma unroll
    for (int l = 0; l < Q; ++l) emax = max(emax, __double2hiint(n[l]) >> 20);   // a negative one counts as small
    bool ok = (unsigned)(emax - 512) < 1024u;
    long long v[Q];
#pragma unroll
    for (int l = 0; l < Q; ++l) ok &= to_units(n[l], emax, v[l]) && __double2hiint(n[l]) >= 0;
    // the first addition of j is F/2's, which has finer bits: in FP64
    long long X = v[1], Y = v[3], Z = v[5];
    if (fm) {
        if (__double2hiint(fhx) | __double2loint(fhx)) ok &= to_units(fhx + n[1], emax, X);
        if (__double2hiint(fhy) | __double2loint(fhy)) ok &= to_units(fhy + n[3], emax, Y);
        if (__double2hiint(fhz) | __double2loint(fhz)) ok &= to_units(fhz + n[5], emax, Z);
    }
    long long R = v[0];
    static_for<1, Q>([&](auto L) {
        constexpr int l = decltype(L)::value;
        constexpr Vel c = vel(l);
        R = round53(R + v[l]);
        // no population reaches 2^60: at most 2^62 here keeps 6 more from wrapping unseen
        if constexpr (l == 6 || l == 12 || l == 18) ok &= (unsigned long long)R <= (1ull << 62);
        if constexpr (c.x != 0 && l != 1) X = round53(c.x > 0 ? X + v[l] : X - v[l]);
        if constexpr (c.y != 0 && l != 3) Y = round53(c.y > 0 ? Y + v[l] : Y - v[l]);
        if constexpr (c.z != 0 && l != 5) Z = round53(c.z > 0 ? Z + v[l] : Z - v[l]);
    });
    if (!ok) return false;
    rho = from_units(R, emax);
    jx = from_units(X, emax);
    jy = from_units(Y, emax);
    jz = from_units(Z, emax);
    return true;
}

__device__ __forceinline__ void moments19_fast(const double (&n)[Q], bool fm, double fx, double fy, double fz,
                                               double &rho, double &jx, double &jy, double &jz)
{
    const double hx = fm ? fx / 2.0 : 0.0, hy = fm ? fy / 2.0 : 0.0, hz = fm ? fz / 2.0 : 0.0;
    if (!moments19_units(n, fm, hx, hy, hz, rho, jx, jy, jz)) moments19(n, hx, hy, hz, rho, jx, jy, jz);
}

// n < 0 and NaN / Inf tests on the bits, off the FP64 pipe (a comparison of doubles occupies it like
// an addition): with the sign bit dropped, a non-finite value has a high word of 0x7ff00000 or
// more; n < 0 is a set sign bit on anything but -0 and a NaN.
__device__ __forceinline__ void check_bits(double v, bool &neg, bool &nonfinite)
{
    const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
    const unsigned mag = hi & 0x7fffffffu;
    nonfinite |= mag >= 0x7ff00000u;
    neg |= (int)hi < 0 && (mag | lo) != 0u && (mag < 0x7ff00000u || (mag == 0x7ff00000u && lo == 0u));
}

__device__ __forceinline__ unsigned check19(const double (&n)[Q])
{
    bool neg = false, nonfinite = false;
#pragma unroll
    for (int l = 0; l < Q; ++l) check_bits(n[l], neg, nonfinite);
    return (neg ? (unsigned)LBGPU_ERR_NEGATIVE_POPULATION : 0u) | (nonfinite ? (unsigned)LBGPU_ERR_NONFINITE : 0u);
}

// Reference phase machine, equilibration.f90:346-489 (non-compensated force), for step c.t with the
// maximum of |j - j_old| (its bits) and the status bits of its populations.  Every exit leaves the
// block "advanced": parity names the buffer that the next step would read, and the buffer parity^1
// holds the input of the exit step (exit_force_moment its moment force).  c.redo on return: the
// force was switched on; step t is to be collided again with it, then this is called once more.
__device__ __forceinline__ void decide64(FlowCtl &c, unsigned long long err_bits, unsigned st, double *hist)
{
    const double l2 = __longlong_as_double((long long)err_bits);
    const int t = c.t;
    bool finish = false;
    c.status |= st;
    if (st & (LBGPU_ERR_NEGATIVE_POPULATION | LBGPU_ERR_NONFINITE)) {
        finish = true;
    } else if (c.redo) {
        c.redo = 0;  // repeat of step t with the force switched on; its l2err is not used
    } else {
        if (hist && t - 1 < c.hist_cap) hist[t - 1] = l2;
        c.last_l2err = l2;
        const bool converged = (l2 <= c.target_error) && t > 2;
        if (converged) {
            if (!c.conv_without) c.conv_without = 1;
            else c.conv_with = 1;
            if (c.conv_without && c.conv_with) {
                finish = true;
            } else {
                // first convergence: f_ext acts from the collision of step t+1 on; that
                // collision already ran with the force off, so step t repeats.
                c.force_collide = 1;
                c.redo = 1;
                return;
            }
        }
    }
    c.exit_force_moment = c.force_moment;
    c.exit_step = t;
    c.parity ^= 1;
    c.force_moment = c.force_collide;
    c.t = t + 1;
    if (!finish && c.max_steps > 0 && c.t > c.max_steps) {
        finish = true;
        c.status |= (unsigned)LBGPU_ERR_STEP_CAP;
    }
    if (finish) c.done = 1;
}

}  // namespace lbg
