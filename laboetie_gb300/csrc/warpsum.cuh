// warpsum.cuh -- sums of FP32 terms over a warp, formed exactly in integers: shuffled FP64 additions, five per
// value and warp, take 64 cycles of the warp's quarter of an SM each.
#pragma once

#include <cstdint>

namespace lbg {

// Sum of one FP32 value per lane, formed exactly in integers on a grid 33 bits below the largest
// one and rounded once; valid in every lane as (unit exponent, integer), made a double by
// warp_exact.
// Of no use with a non-finite term (exponent 255): see warp_nonfinite_sum.
__device__ __forceinline__ long long warp_int_sum(float v, int &emax)
{
    const unsigned b = __float_as_uint(v);
    const int e = (int)((b >> 23) & 255u);
    emax = (int)__reduce_max_sync(0xffffffffu, (unsigned)max(e, 1));
    const unsigned m = (b & 0x7fffffu) | (e ? 0x800000u : 0u);
    const int up = 33 - (emax - max(e, 1));
    long long k = up >= 0 ? (long long)((unsigned long long)m << up) : (long long)(m >> min(-up, 31));
    if ((int)b < 0) k = -k;
    const unsigned lo = __reduce_add_sync(0xffffffffu, (unsigned)k & 0x1ffffffu);
    const unsigned mid = __reduce_add_sync(0xffffffffu, (unsigned)(k >> 25) & 0x1ffffffu);
    const int hi = __reduce_add_sync(0xffffffffu, (int)(k >> 50));
    return ((long long)hi << 50) + ((long long)mid << 25) + (long long)lo;
}

__device__ __forceinline__ double warp_exact(long long k, int emax)
{
    const double r = (double)k;   // one unit is 2^(emax - 183)
    return k == 0 ? 0.0 : __hiloint2double(__double2hiint(r) + (emax - 183) * (1 << 20), __double2loint(r));
}

// The sum of values with a non-finite one among them, as FP64 additions form it; valid in every lane.
static __device__ __noinline__ double warp_nonfinite_sum(float v)
{
    double s = (double)v;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s = s + __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// Sums of three finite values per lane: lane d < 3 returns the sum of t[d], NaN with a non-finite term.
__device__ __forceinline__ double warp_sum3_finite(const float (&t)[3])
{
    const int lane = threadIdx.x & 31;
    int e[3];
    long long v[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) v[d] = warp_int_sum(t[d], e[d]);
    if (lane >= 3) return 0.0;
    const int emax = lane == 0 ? e[0] : (lane == 1 ? e[1] : e[2]);
    const double s = warp_exact(lane == 0 ? v[0] : (lane == 1 ? v[1] : v[2]), emax);
    return emax == 255 ? __longlong_as_double(0x7ff8000000000000ll) : s;
}

// The same with whatever FP64 additions make of non-finite terms.
__device__ __forceinline__ double warp_sum3_exact(const float (&t)[3])
{
    const int lane = threadIdx.x & 31;
    int e[3];
    long long v[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) v[d] = warp_int_sum(t[d], e[d]);
    if (max(max(e[0], e[1]), e[2]) == 255) {
        double w[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) w[d] = e[d] == 255 ? warp_nonfinite_sum(t[d]) : warp_exact(v[d], e[d]);
        return lane == 0 ? w[0] : (lane == 1 ? w[1] : w[2]);
    }
    if (lane >= 3) return 0.0;
    return warp_exact(lane == 0 ? v[0] : (lane == 1 ? v[1] : v[2]), lane == 0 ? e[0] : (lane == 1 ? e[1] : e[2]));
}

}  // namespace lbg
