// flow_f64_resident.cu -- many FP64 steps of a small box in one launch (compiled with -fmad=false).
//
// An FP64 instruction occupies its quarter of an SM for 64 cycles whatever the number of its lanes
// (19 cycles of the SM with all quarters busy), so a box with fewer warps of fluid nodes than the GPU
// has quarters is bound by the length of one warp's FP64 chain: some 290 instructions, 9.5 us, to
// which a launch per step adds its gap, a chain of dependent loads and a reduction with a last block.
// Here the steps run in one cooperative launch with a grid barrier (gridsync.cuh) that carries the
// loop's maximum; the pull addresses are formed once; and while there are no more warps than SMs,
// four warps share a node: warp 0 / 1 / 2 / 3 adds up rho / jx / jy / jz, divides one velocity and
// collides the rest and axis / xy / xz / yz velocities, passing values through shared memory.  Every
// operation is the one of the launch-per-step kernel (flow64.cuh), so the states have the same bits.
// us per step of the reference loop in a porous box, as launches / a node per thread / four warps per
// node: 2,457 fluid nodes 16.9 / 12.3 / 6.6, 10,545 17.4 / 12.9 / -, 38,393 28.8 / 26.0 / - (strict);
// 13.3 / 7.9, 13.9 / 8.4, 21.0 / 16.4 (fused, whose chain is half as long and is not split).
#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "ctx.h"
#include "flow.h"
#include "flow64.cuh"
#include "gridsync.cuh"

namespace lbg {
namespace {

constexpr int RT = 256;   // most threads of a block whose threads own a node each

struct ResidentArgs64 {
    FlowArgs64 a;         // parity, force_moment, force_collide: of the first fixed step
    GridSync *sync;
    GridWait wait;
    int nsteps;
    int loop;             // the reference loop on a.ctl; else fixed steps
    int fon;              // fixed steps: force from the second step's moments on
};

// Element offset of the population pulled along l into the node (x, y, z).
__device__ __forceinline__ unsigned pull_offset(const FlowArgs64 &a, int l, unsigned node, uint32_t m, int x, int y, int z)
{
    const unsigned N = (unsigned)a.N;
    if ((m >> l) & 1u) return (unsigned)inv(l) * N + node;
    const Vel c = vel(l);
    const int sx = c.x > 0 ? wrap_minus(x, a.lx) : (c.x < 0 ? wrap_plus(x, a.lx) : x);
    const int sy = c.y > 0 ? wrap_minus(y, a.ly) : (c.y < 0 ? wrap_plus(y, a.ly) : y);
    const int sz = c.z > 0 ? wrap_minus(z, a.lz) : (c.z < 0 ? wrap_plus(z, a.lz) : z);
    return (unsigned)l * N + (unsigned)sx + (unsigned)a.lx * ((unsigned)sy + (unsigned)a.ly * (unsigned)sz);
}

template <int FMASK, bool FUSED, bool SPLIT>
__global__ void __launch_bounds__(SPLIT ? 128 : RT, 1) k_flow64_resident(const ResidentArgs64 r)
{
    constexpr int MINE = SPLIT ? 7 : Q;   // populations a thread pulls
    __shared__ FlowCtl ctl;
    __shared__ double sn[SPLIT ? Q : 1][32], smom[SPLIT ? 4 : 1][32], su[SPLIT ? 4 : 1][32];
    const FlowArgs64 &a = r.a;
    const unsigned tid = threadIdx.x, lane = tid & 31, role = tid >> 5;
    const unsigned i = SPLIT ? blockIdx.x * 32u + lane : blockIdx.x * blockDim.x + tid;
    const bool mine = i < (unsigned)a.Nf;
    const unsigned N = (unsigned)a.N;
    const int l0 = !SPLIT ? 0 : (role == 0 ? 0 : 3 + 4 * (int)role);   // first of the thread's velocities
    const int count = !SPLIT ? Q : (role == 0 ? 7 : 4);
    unsigned node = 0, off[MINE];
    double jold[3] = {0.0, 0.0, 0.0};   // SPLIT: [0] of the warp's component
    double *const J[3] = {a.jx, a.jy, a.jz};
    if (mine) {
        node = a.fidx[i];
        const uint32_t m = a.mask[node];
        const int x = (int)(node % (unsigned)a.lx);
        const unsigned yz = node / (unsigned)a.lx;
        const int y = (int)(yz % (unsigned)a.ly), z = (int)(yz / (unsigned)a.ly);
#pragma unroll
        for (int k = 0; k < MINE; ++k) off[k] = k < count ? pull_offset(a, l0 + k, node, m, x, y, z) : 0u;
        if (r.loop) {
            if constexpr (SPLIT) {
                if (role > 0) jold[0] = J[role - 1][node];
            } else {
                for (int d = 0; d < 3; ++d) jold[d] = J[d][node];
            }
        }
    }
    if (tid == 0 && r.loop) ctl = *a.ctl;
    __syncthreads();
    if (r.loop && ctl.done) return;

    const double fx = a.F[0], fy = a.F[1], fz = a.F[2];
    // one step from the buffer of the given parity into the other one
    auto step = [&](int parity, bool fm, bool fc, unsigned long long &err, unsigned &bad) {
        const double *src = parity ? a.f1 : a.f0;
        double *dst = parity ? a.f0 : a.f1;
        if constexpr (!SPLIT) {
            if (!mine) return;
            double n[Q];
#pragma unroll
            for (int l = 0; l < Q; ++l) n[l] = __ldcg(src + off[l]);
            if (r.loop) bad = check19(n);
            double rho, jx = 0.0, jy = 0.0, jz = 0.0;
            if constexpr (FUSED) fused_step<FMASK, true, true, true>(n, fm, fc, fx, fy, fz, a, jx, jy, jz);
            else moments19_fast(n, fm, fx, fy, fz, rho, jx, jy, jz);
            if (r.loop) {
                const double e = max_nonneg(max_nonneg(fabs(jx - jold[0]), fabs(jy - jold[1])), fabs(jz - jold[2]));
                err = (unsigned long long)__double_as_longlong(e);
                jold[0] = jx;
                jold[1] = jy;
                jold[2] = jz;
            }
            if constexpr (!FUSED) collide_strict<FMASK, true>(n, rho, jx, jy, jz, fx, fy, fz, a, fc);
#pragma unroll
            for (int l = 0; l < Q; ++l) dst[(size_t)l * N + node] = n[l];
        } else {
            double v[7];
            bool neg = false, nonfinite = false;
#pragma unroll
            for (int k = 0; k < 7; ++k) {
                v[k] = mine && k < count ? __ldcg(src + off[k]) : 1.0;
                if (k < count) sn[l0 + k][lane] = v[k];
                check_bits(v[k], neg, nonfinite);
            }
            if (mine)
                bad = (neg ? (unsigned)LBGPU_ERR_NEGATIVE_POPULATION : 0u) | (nonfinite ? (unsigned)LBGPU_ERR_NONFINITE : 0u);
            __syncthreads();
            // rho (warp 0) or one component of j, in the order of moments19
            double mom;
            if (role == 0) {
                mom = sn[0][lane];
#pragma unroll
                for (int l = 1; l < Q; ++l) mom = mom + sn[l][lane];
            } else {
                mom = fm ? (role == 1 ? fx : (role == 2 ? fy : fz)) / 2.0 : 0.0;
                auto sum = [&](auto D) {
                    constexpr int d = decltype(D)::value;
                    static_for<1, Q>([&](auto L) {
                        constexpr int l = decltype(L)::value;
                        constexpr int c = d == 1 ? vel(l).x : (d == 2 ? vel(l).y : vel(l).z);
                        if constexpr (c != 0) mom = addsgn<c>(mom, sn[l][lane]);
                    });
                };
                if (role == 1) sum(std::integral_constant<int, 1>{});
                else if (role == 2) sum(std::integral_constant<int, 2>{});
                else sum(std::integral_constant<int, 3>{});
                if (mine) err = (unsigned long long)__double_as_longlong(fabs(mom - jold[0]));
                jold[0] = mom;
            }
            smom[role][lane] = mom;
            __syncthreads();
            const double rho = smom[0][lane];
            if (role > 0) su[role][lane] = divide(mom, rho);
            __syncthreads();
            const double jx = smom[1][lane], jy = smom[2][lane], jz = smom[3][lane];
            const double ux = su[1][lane], uy = su[2][lane], uz = su[3][lane];
            auto collide = [&](auto R) {
                constexpr int ro = decltype(R)::value, first = ro == 0 ? 0 : 3 + 4 * ro, cnt = ro == 0 ? 7 : 4;
                double n[Q];
#pragma unroll
                for (int k = 0; k < cnt; ++k) n[first + k] = v[k];
                collide_strict_u<FMASK, true, ro>(n, rho, jx, jy, jz, ux, uy, uz, fx, fy, fz, a, fc);
                if (mine)
#pragma unroll
                    for (int k = 0; k < cnt; ++k) dst[(size_t)(first + k) * N + node] = n[first + k];
            };
            if (role == 0) collide(std::integral_constant<int, 0>{});
            else if (role == 1) collide(std::integral_constant<int, 1>{});
            else if (role == 2) collide(std::integral_constant<int, 2>{});
            else collide(std::integral_constant<int, 3>{});
        }
    };

    unsigned round = 0;
    bool ok = true;
    int parity = r.loop ? ctl.parity : a.parity;
    for (int k = 0; k < r.nsteps && ok; ++k) {
        unsigned long long err = 0;
        unsigned bad = 0;
        if (!r.loop) {
            step(parity, (k == 0 ? a.force_moment : r.fon) != 0, a.force_collide != 0, err, bad);
            parity ^= 1;
            if (k + 1 < r.nsteps) ok = grid_barrier<false>(r.sync, round++, r.wait, err, bad);
            continue;
        }
        const bool fm = ctl.force_moment != 0;
        step(parity, fm, ctl.force_collide != 0, err, bad);
        if (!(ok = grid_barrier<true>(r.sync, round++, r.wait, err, bad))) break;
        if (tid == 0) decide64(ctl, err, bad, blockIdx.x == 0 ? a.hist : nullptr);
        __syncthreads();
        if (ctl.redo) {   // the same step again, collided with the force
            unsigned long long e2 = 0;
            unsigned b2 = 0;
            step(parity, fm, true, e2, b2);
            if (!(ok = grid_barrier<false>(r.sync, round++, r.wait, e2, b2))) break;
            if (tid == 0) decide64(ctl, err, bad, nullptr);
            __syncthreads();
        }
        parity = ctl.parity;
        if (ctl.done) break;
    }
    if (r.loop) {
        if (mine && ok) {
            if constexpr (SPLIT) {
                if (role > 0) J[role - 1][node] = jold[0];
            } else {
                for (int d = 0; d < 3; ++d) J[d][node] = jold[d];
            }
        }
        if (blockIdx.x == 0 && tid == 0) store_ctl(a.ctl, ctl);
    }
    if (!ok && tid == 0) atomicOr(&a.ctl->status, (unsigned)LBGPU_ERR_TIMEOUT);
}

using Kernel = void (*)(ResidentArgs64);

template <bool FUSED, bool SPLIT>
Kernel kernel_of(int fmask)
{
    switch (fmask) {
    case 0: return k_flow64_resident<0, FUSED, SPLIT>;
    case 1: return k_flow64_resident<1, FUSED, SPLIT>;
    case 2: return k_flow64_resident<2, FUSED, SPLIT>;
    case 4: return k_flow64_resident<4, FUSED, SPLIT>;
    default: return k_flow64_resident<7, FUSED, SPLIT>;
    }
}

Kernel kernel_of(const ResidentPlan &p, int fmask, bool fused)
{
    return fused ? kernel_of<true, false>(fmask) : (p.split ? kernel_of<false, true>(fmask) : kernel_of<false, false>(fmask));
}

}  // namespace

// LBGPU_F64_RESIDENT=0: one launch per step; =whole: no node shared by four warps.
ResidentPlan plan_resident64(unsigned long long Nf, long long N, int fmask, bool fused)
{
    ResidentPlan p{};
    const char *env = std::getenv("LBGPU_F64_RESIDENT");
    const char *mode = env ? env : "";
    int dev = 0, sms = 0, coop = 0, per_sm = 0;
    if (!std::strcmp(mode, "0") || Nf == 0 || (unsigned long long)Q * (unsigned long long)N >= (1ull << 32) ||
        cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop) {
        cudaGetLastError();
        return p;
    }
    if (Nf > (unsigned long long)sms * RT) return p;
    p.split = !fused && std::strcmp(mode, "whole") && Nf <= 32ull * sms;
    const unsigned t = (unsigned)((Nf + sms - 1) / sms);
    p.threads = p.split ? 128u : (t + 31u) / 32u * 32u;
    const unsigned nodes = p.split ? 32u : p.threads;
    p.blocks = (unsigned)((Nf + nodes - 1) / nodes);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel_of(p, fmask, fused), (int)p.threads, 0) == cudaSuccess &&
        (long long)per_sm * sms >= (long long)p.blocks)
        return p;
    cudaGetLastError();
    return ResidentPlan{};
}

cudaError_t launch_resident64(const ResidentPlan &plan, const FlowArgs64 &a, int fmask, void *sync, int nsteps, bool loop,
                              int fon, cudaStream_t s)
{
    ResidentArgs64 r;
    std::memset(&r, 0, sizeof(r));
    r.a = a;
    r.sync = static_cast<GridSync *>(sync);
    r.wait = grid_wait();
    r.nsteps = nsteps;
    r.loop = loop ? 1 : 0;
    r.fon = fon;
    cudaError_t e = cudaMemsetAsync(sync, 0, sizeof(GridSync), s);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(plan.blocks);
    c.blockDim = dim3(plan.threads);
    c.stream = s;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeCooperative;
    at.val.cooperative = 1;
    c.attrs = &at;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, kernel_of(plan, fmask, a.fused != 0), r);
}

}  // namespace lbg
