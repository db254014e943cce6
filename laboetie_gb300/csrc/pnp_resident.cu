// pnp_resident.cu -- the Poisson-Nernst-Planck loop of a small box in one launch (compiled with
// -fmad=false).
//
// One thread owns one node of the lattice for the whole launch (a cooperative grid of at most one
// 768-thread block per SM); its potential, its densities and their values at the start of the
// outer iteration stay in registers, and the sweeps, the Nernst-Planck update and the convergence
// test follow each other with a grid barrier between them (gridsync.cuh) instead of launches and
// host synchronisations.
//
// A Jacobi sweep of sor.f90:48-70 multiplies each of 18 neighbours by its weight.  The axis and
// diagonal weights are 1/18 and exactly half of it, so a node keeps t = w_axis phi beside phi and a
// neighbour adds t, or t/2 as the exact product of a fused multiply-add: the same roundings as
// w_l phi added term by term, with 26 FP64 instructions per node and sweep instead of 45 (the sweep
// is bound by the FP64 pipe; t/2 differs from w_diag phi only below the smallest normal double).
// The right-hand side (c+ - c-) is formed once per solve.  48^3 touching spheres, per sweep:
// 21.3 us as launches of the term-by-term sweep.
//
// Sums that decide (residual, flux sums, relative changes) are formed in a fixed order: 128 strided
// lanes of a block, then the blocks in order, by every block alike, so all take the same decision.
// So is the sum of |phi| between the solves of one call, whose order the reference fixes (PnpLoop).
#include <algorithm>
#include <cstring>

#include "common.cuh"
#include "ctx.h"
#include "gridsync.cuh"
#include "pnp.h"
#include "pnp_args.cuh"

namespace lbg {
namespace {

constexpr int RT = 768;   // most threads per block: up to 85 registers each

struct Shared {
    double v[2][RT];      // the values being summed
    double part[8];       // per summing warp
    double tot[4];
    unsigned cnt[3];
    int ok;
};

__device__ __forceinline__ double warp_tree(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

struct Grid {
    const PnpResidentArgs &r;
    Shared &sh;
    unsigned round = 0;

    __device__ __forceinline__ bool barrier()
    {
        unsigned long long v;
        unsigned b;
        return grid_barrier<false>(r.sync, round++, r.wait, v, b);
    }

    // Sums over the grid of NV (1 or 2) values per thread, and of 3 counts per thread; the totals in
    // sh.tot / sh.cnt.  DENSE: most threads hold a non-zero value (summed through shared memory: a
    // shuffle tree in every warp would cost 5 FP64 instructions per warp, a fifth of a sweep); else
    // warps without one are skipped.
    template <int NV, bool DENSE, bool COUNTS>
    __device__ __forceinline__ bool sum(double (&v)[NV], unsigned c0 = 0, unsigned c1 = 0, unsigned c2 = 0)
    {
        const unsigned tid = threadIdx.x, T = blockDim.x, lane = tid & 31, wid = tid >> 5;
        double *partial = r.partial + (size_t)(round & 1u) * 8u * gridDim.x;
        if (tid < 3) sh.cnt[tid] = 0;
        __syncthreads();
        if constexpr (COUNTS) {
            c0 = __reduce_add_sync(0xffffffffu, c0);
            c1 = __reduce_add_sync(0xffffffffu, c1);
            c2 = __reduce_add_sync(0xffffffffu, c2);
            if (lane == 0) {
                if (c0) atomicAdd(&sh.cnt[0], c0);
                if (c1) atomicAdd(&sh.cnt[1], c1);
                if (c2) atomicAdd(&sh.cnt[2], c2);
            }
        }
        if constexpr (DENSE) {
            static_assert(NV <= 2, "two values at most");
#pragma unroll
            for (int q = 0; q < NV; ++q) sh.v[q][tid] = v[q];
            __syncthreads();
            if (wid < 4u * NV) {   // four warps per value, one on each quarter of the SM
                const unsigned q = wid >> 2;
                double s = 0.0;
                for (unsigned k = (wid & 3u) * 32u + lane; k < T; k += 128u) s = s + sh.v[q][k];
                s = warp_tree(s);
                if (lane == 0) sh.part[wid] = s;
            }
            __syncthreads();
            if (tid < NV) partial[tid * gridDim.x + blockIdx.x] =
                ((sh.part[4 * tid] + sh.part[4 * tid + 1]) + sh.part[4 * tid + 2]) + sh.part[4 * tid + 3];
        } else {
            // per warp, in warp order: a warp of zeros adds exact zeros and is left out
#pragma unroll
            for (int q = 0; q < NV; ++q) {
                double s = v[q];
                const bool any = __any_sync(0xffffffffu, s != 0.0 || s != s);
                if (any) s = warp_tree(s);
                if (lane == 0) sh.v[1][wid * NV + q] = any ? s : 0.0;
            }
            __syncthreads();
            if (tid < NV) {
                double s = 0.0;
                for (unsigned w = 0; w < T / 32u; ++w) {
                    const double x = sh.v[1][w * NV + tid];
                    if (x != 0.0 || x != x) s = s + x;
                }
                partial[tid * gridDim.x + blockIdx.x] = s;
            }
        }
        unsigned *pc = reinterpret_cast<unsigned *>(partial + 4u * gridDim.x);
        if (COUNTS && tid < 3) pc[tid * gridDim.x + blockIdx.x] = sh.cnt[tid];
        if (!barrier()) return false;   // its first step is a block barrier: the partials are written
        if (wid < NV) {
            double s = 0.0;
            for (unsigned b = lane; b < gridDim.x; b += 32u) {
                const double x = __ldcg(partial + wid * gridDim.x + b);
                if (DENSE || x != 0.0 || x != x) s = s + x;
            }
            if (DENSE || __any_sync(0xffffffffu, s != 0.0 || s != s)) s = warp_tree(s);
            if (lane == 0) sh.tot[wid] = s;
        }
        if (COUNTS && wid >= 4 && wid < 7) {
            unsigned n = 0;
            for (unsigned b = lane; b < gridDim.x; b += 32u) n += __ldcg(pc + (wid - 4u) * gridDim.x + b);
            n = __reduce_add_sync(0xffffffffu, n);
            if (lane == 0) sh.cnt[wid - 4u] = n;
        }
        __syncthreads();
        return true;
    }
};

// |(v - o) / o| of check_charge_distribution_equilibrium.f90:30-37 where |o| > 1e-12, else 0; an
// unchanged value needs no division
__device__ __forceinline__ double rel_change(double v, double o, unsigned &count)
{
    if (!(fabs(o) > 1.0e-12)) return 0.0;
    count = 1;
    const double d = v - o;
    return d == 0.0 ? 0.0 : fabs(d / o);
}

__global__ void __launch_bounds__(RT, 1) k_pnp_resident(const PnpResidentArgs r)
{
    __shared__ Shared sh;
    __shared__ PnpLoop L;
    const PnpArgs &a = r.a;
    const unsigned tid = threadIdx.x, T = blockDim.x;
    const long long N = a.N;
    const long long node = (long long)blockIdx.x * T + tid;
    const bool mine = node < N;
    Grid grid{r, sh};
    int x = 0, y = 0, z = 0;
    int X[3], Y[3], Z[3];   // [c + 1]: offset of the coordinate x - c
    double phi = 0.0, cp = 0.0, cm = 0.0;
    bool fluid = false;
    double *const phi_g = r.phi, *const t0 = r.t0, *const t1 = r.t1;
    if (mine) {
        coords(node, a.lx, a.ly, x, y, z);
        const int sy = a.lx, sz = a.lx * a.ly;
        X[0] = wrap_plus(x, a.lx);       X[1] = x;       X[2] = wrap_minus(x, a.lx);
        Y[0] = wrap_plus(y, a.ly) * sy;  Y[1] = y * sy;  Y[2] = wrap_minus(y, a.ly) * sy;
        Z[0] = wrap_plus(z, a.lz) * sz;  Z[1] = z * sz;  Z[2] = wrap_minus(z, a.lz) * sz;
        phi = phi_g[node];
        cp = r.cp[node];
        cm = r.cm[node];
        fluid = a.mask[node] & FLUID_BIT;
        t0[node] = a.a0[1] * phi;
    }
    if (tid == 0) L = *r.loop;
    if (!grid.barrier()) {
        if (tid == 0) atomicOr(&r.loop->status, (unsigned)LBGPU_ERR_TIMEOUT);
        return;
    }
    // values at the start of the outer iteration (kept across launches in r.bak)
    double phi_old = phi, cp_old = cp, cm_old = cm;
    if (mine && L.in_solve && r.max_outer > 0) {
        phi_old = r.bak[0][node];
        cp_old = r.bak[1][node];
        cm_old = r.bak[2][node];
    }
    double *src = t0, *dst = t1;
    bool ok = true;
    int sweeps = 0;   // of this launch
    for (;;) {
        // ---- a solve (sor.f90:48-78), begun or continued
        if (!L.in_solve) {
            phi_old = phi;
            cp_old = cp;
            cm_old = cm;
        }
        const double rhs = a.factor * (cp - cm);
        int iter = L.in_solve ? L.iter : 0;
        bool conv = L.in_solve && L.resume_conv, capped = !conv && iter >= r.max_iter, undecided = false;
        // N < 2^17 additions in storage order and fewer on the device: the two sums of |phi| lie within
        // 2^-35 of each other.  Compared as bits, in the order of the non-negative doubles they are (a
        // comparison of doubles by every thread costs a sweep what an addition does); -1: never.
        const double limit = L.limit, margin = L.limit_exact ? 0.0 : 0x1p-35 * limit;
        const long long below = limit >= 0.0 ? __double_as_longlong(limit - margin) : -1,
                        above = limit >= 0.0 ? __double_as_longlong(limit + margin) : -1;
        double anorm = L.anorm, residual = 0.0;
        while (ok && !conv && !capped && !undecided && sweeps < r.max_sweeps) {
            double v[2] = {0.0, 0.0};
            if (mine) {
                double s = a.a0[0] * phi;   // 0 + w_0 phi
                static_for<1, Q>([&](auto Lc) {
                    constexpr int l = decltype(Lc)::value;
                    constexpr Vel c = vel(l);
                    const double t = __ldcg(src + (X[c.x + 1] + Y[c.y + 1] + Z[c.z + 1]));
                    if constexpr (wclass(l) == 1) s = s + t;
                    else s = __fma_rn(0.5, t, s);
                });
                s = s + rhs;
                v[0] = fabs(s - phi);
                phi = a.omega * s + a.one_minus_omega * phi;
                v[1] = fabs(phi);
                dst[node] = a.a0[1] * phi;
                phi_g[node] = phi;
            }
            double *w = src;
            src = dst;
            dst = w;
            ok = grid.sum<2, true, false>(v);
            if (!ok) break;
            ++iter;
            ++sweeps;
            residual = sh.tot[0];
            anorm = sh.tot[1];
            const long long bits = __double_as_longlong(residual);
            conv = bits <= below;
            undecided = !conv && bits <= above;
            capped = !conv && !undecided && iter >= r.max_iter;
        }
        if (!ok) break;
        const bool solved = conv || capped;
        __syncthreads();   // every thread has read L and the totals
        if (tid == 0) {
            L.in_solve = solved ? 0 : 1;
            L.iter = iter;
            L.undecided = undecided;
            L.resume_conv = 0;
            L.residual = residual;
            L.anorm = anorm;
            if (solved) {
                L.total += iter - 1;   // the count the reference prints (sor.f90:87)
                L.converged = conv;
                L.anormf0 = anorm;
                L.limit = r.limit_factor * anorm;
                L.limit_exact = 0;
                if (!conv) {
                    L.status |= LBGPU_ERR_STEP_CAP;
                    L.done = 1;
                }
            }
        }
        __syncthreads();
        if (!solved) {   // to be continued by the next launch
            if (mine && r.max_outer > 0) {
                r.bak[0][node] = phi_old;
                r.bak[1][node] = cp_old;
                r.bak[2][node] = cm_old;
            }
            break;
        }
        if (r.max_outer <= 0 || capped) {
            if (tid == 0) L.done = 1;
            break;
        }
        // ---- Nernst-Planck update (just_eq_smolu.f90:61-129)
        int its = 0;
        bool more = true, bad_flux = false;
        while (more) {
            double sp = 0.0, sm = 0.0;
            if (a.loop_bug) {
                // the 9 lx links that start on the line (i, ly, lz), one thread each
                for (long long k = node; k < 9ll * a.lx; k += (long long)gridDim.x * T) {
                    const int p = (int)(k / a.lx), i = (int)(k - (long long)p * a.lx);
                    const long long ro = i + (long long)a.lx * ((a.ly - 1) + (long long)a.ly * (a.lz - 1));
                    const Vel c = vel(2 * p + 1);
                    const long long rb = nb(i, a.ly - 1, a.lz - 1, c.x, c.y, c.z, a.lx, a.ly, a.lz);
                    double Jp = 0.0, Jm = 0.0;
                    if ((a.mask[ro] & FLUID_BIT) && (a.mask[rb] & FLUID_BIT))
                        link_flux_values(a, __ldcg(phi_g + ro), __ldcg(r.cp + ro), __ldcg(r.cm + ro), __ldcg(phi_g + rb),
                                         __ldcg(r.cp + rb), __ldcg(r.cm + rb), p < 3 ? a.delta_axis : a.delta_diag, Jp, Jm);
                    r.link[2 * k] = Jp;
                    r.link[2 * k + 1] = Jm;
                }
                if (!(ok = grid.barrier())) break;
            }
            if (mine && fluid) {
                static_for<0, 9>([&](auto P) {
                    constexpr int p = decltype(P)::value;
                    constexpr int l = 2 * p + 1;   // l = 2, 4, ..., 18 of the reference (:66)
                    constexpr Vel c = vel(l);
                    const int ox = c.x > 0 ? wrap_minus(x, a.lx) : (c.x < 0 ? wrap_plus(x, a.lx) : x);
                    const int oy = c.y > 0 ? wrap_minus(y, a.ly) : (c.y < 0 ? wrap_plus(y, a.ly) : y);
                    const int oz = c.z > 0 ? wrap_minus(z, a.lz) : (c.z < 0 ? wrap_plus(z, a.lz) : z);
                    const long long rb = nb(x, y, z, c.x, c.y, c.z, a.lx, a.ly, a.lz);
                    const long long ro = ox + (long long)a.lx * (oy + (long long)a.ly * oz);
                    if (a.loop_bug) {
                        if (y == a.ly - 1 && z == a.lz - 1 && (a.mask[rb] & FLUID_BIT)) {
                            const double *J = r.link + 2 * ((long long)p * a.lx + x);
                            sp = sp + __ldcg(J);
                            sm = sm + __ldcg(J + 1);
                        }
                        if (oy == a.ly - 1 && oz == a.lz - 1 && (a.mask[ro] & FLUID_BIT)) {
                            const double *J = r.link + 2 * ((long long)p * a.lx + ox);
                            sp = sp - __ldcg(J);
                            sm = sm - __ldcg(J + 1);
                        }
                    } else {
                        const double delta = p < 3 ? a.delta_axis : a.delta_diag;
                        double Jp, Jm;
                        if (a.mask[rb] & FLUID_BIT) {
                            link_flux_values(a, phi, cp, cm, __ldcg(phi_g + rb), __ldcg(r.cp + rb), __ldcg(r.cm + rb),
                                             delta, Jp, Jm);
                            sp = sp + Jp;
                            sm = sm + Jm;
                        }
                        if (a.mask[ro] & FLUID_BIT) {
                            link_flux_values(a, __ldcg(phi_g + ro), __ldcg(r.cp + ro), __ldcg(r.cm + ro), phi, cp, cm,
                                             delta, Jp, Jm);
                            sp = sp - Jp;
                            sm = sm - Jm;
                        }
                    }
                });
            }
            double v[4] = {sp, sm, sp * sp, sm * sm};
            if (!(ok = grid.sum<4, false, false>(v))) break;
            ++its;
            bad_flux = fabs(sh.tot[0]) > (double)1.e-12f || fabs(sh.tot[1]) > (double)1.e-12f;
            if (bad_flux) break;
            if (mine && fluid) {
                cp = cp + sp;
                cm = cm + sm;
                r.cp[node] = cp;
                r.cm[node] = cm;
            }
            // lane 0: tot_p, lane 1: tot_m of the first warp (just_eq_smolu.f90:122-129)
            if (tid < 32) {
                double tot = 1.7976931348623157e308;
                if (r.sigma != 0.0 && a.eDp != 0.0 && a.eDm != 0.0)
                    tot = sqrt((tid & 1) ? sh.tot[3] : sh.tot[2]) / r.count_fluid /
                          (0.5 * r.rho_ch * ((tid & 1) ? a.eDm : a.eDp)) / r.sigma;
                const double other = __shfl_xor_sync(0xffffffffu, tot, 1);
                if (tid == 0) sh.ok = other + tot > (double)5.e-6f && its < 10;
            }
            __syncthreads();
            more = sh.ok != 0;
            // neighbours read the new densities in the next round
            if (more && !(ok = grid.barrier())) break;
        }
        if (!ok) break;
        if (bad_flux) {
            __syncthreads();
            if (tid == 0) {
                L.status |= LBGPU_ERR_FLUX_SUM;
                L.done = 1;
            }
            break;
        }
        // ---- convergence test (check_charge_distribution_equilibrium.f90:24-44)
        unsigned n0 = 0, n1 = 0, n2 = 0;
        double dphi = 0.0, dcp = 0.0, dcm = 0.0;
        if (mine) {
            dphi = rel_change(phi, phi_old, n0);
            dcp = rel_change(cp, cp_old, n1);
            dcm = rel_change(cm, cm_old, n2);
        }
        double w1[2] = {dcp, dcm};
        double w0[1] = {dphi};
        if (!(ok = grid.sum<2, false, false>(w1))) break;
        const double sp1 = sh.tot[0], sm1 = sh.tot[1];
        __syncthreads();
        if (!(ok = grid.sum<1, true, true>(w0, n0, n1, n2))) break;
        if (tid == 0) {
            const double eps = 1.0e-12;
            const double rp = sh.cnt[0] ? sh.tot[0] / (double)sh.cnt[0] : 0.0;
            const double r1 = sh.cnt[1] ? sp1 / (double)sh.cnt[1] : 0.0;
            const double r2 = sh.cnt[2] ? sm1 / (double)sh.cnt[2] : 0.0;
            L.outer += 1;
            if (rp < eps && r1 < eps && r2 < eps) {
                L.equilibrium = 1;
                L.done = 1;
            } else if (L.outer >= r.max_outer) {
                L.done = 1;
            }
            sh.ok = L.done || sweeps >= r.max_sweeps || L.outer - r.outer0 >= r.outers_per_launch;
        }
        __syncthreads();
        if (sh.ok) break;
    }
    if (tid == 0) {
        if (!ok) atomicOr(&r.loop->status, (unsigned)LBGPU_ERR_TIMEOUT);
        if (blockIdx.x == 0) {
            constexpr int WORDS = (int)(offsetof(PnpLoop, status) / sizeof(unsigned));
            for (int k = 0; k < WORDS; ++k) reinterpret_cast<unsigned *>(r.loop)[k] = reinterpret_cast<unsigned *>(&L)[k];
            if (L.status) atomicOr(&r.loop->status, L.status);
        }
    }
}

}  // namespace

size_t pnp_resident_partials(unsigned blocks) { return 2 * 8 * (size_t)blocks; }

PnpResidentPlan plan_pnp_resident(long long N)
{
    PnpResidentPlan p{};
    const char *env = std::getenv("LBGPU_PNP_RESIDENT");   // 0: launches and a host loop
    int dev = 0, sms = 0, coop = 0, per_sm = 0;
    if ((env && std::strcmp(env, "0") == 0) || cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess) {
        cudaGetLastError();
        return p;
    }
    if (!coop || N > (long long)sms * RT) return p;
    const unsigned t = (unsigned)((N + sms - 1) / sms);
    p.threads = std::max(256u, (t + 31u) / 32u * 32u);   // eight warps at least: they share the sums
    p.blocks = (unsigned)((N + p.threads - 1) / p.threads);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_pnp_resident, (int)p.threads, 0) != cudaSuccess ||
        (long long)per_sm * sms < (long long)p.blocks) {
        cudaGetLastError();
        return PnpResidentPlan{};
    }
    return p;
}

cudaError_t launch_pnp_resident(const PnpResidentPlan &plan, PnpResidentArgs &r, cudaStream_t s)
{
    r.wait = grid_wait();
    cudaError_t e = cudaMemsetAsync(r.sync, 0, sizeof(GridSync), s);
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
    return cudaLaunchKernelEx(&c, k_pnp_resident, r);
}

}  // namespace lbg
