// mp_resident.cu -- many tracer steps of a small box in one launch (compiled with -fmad=false; the
// fused operations are explicit).
//
// One thread owns one fluid node for the whole launch: the 18 incoming scattering probabilities
// (fixed for the run; mp_f32.cu recomputes them from V every step, mp_f64.cu reads them from its
// table), its P, its adsorbed part and (u*, D) stay in registers, and a step gathers the 18
// neighbours' P.  As in flow_f32_resident.cu the box lives in a cluster's shared memory where it
// fits, else P goes through L2 with a grid barrier per step.  The per-node operations and their
// order are those of the launch-per-step kernels, so P and P_ads have the same bits.
//
// VACF leaves the step: each warp stores its three sums per step, and a second kernel adds the
// warps in a fixed order after the launch.  The convergence test (it > 2 and |VACF| below both
// thresholds) is made on the host then; the launch leaves the P it started from untouched, so a
// run that turned out to converge inside it is repeated up to that step, and one whose VACF did not stay
// finite is left to the launches per step: the kernels below are for finite P.  Per step, a reduction
// with its last-block decision costs 6 us of FP64 shuffles, fences and dependent reads.  us per
// step, as launches against here: 1 x 50 x 50 cell (2,323 fluid nodes) FP32 11.1 / 1.57, FP64
// 20.0 / 9.2 (most of it its 126 FP64 instructions of 64 cycles each); 30^3 touching spheres
// (8,904) FP32 13.1 / 2.42.
#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "common.cuh"
#include "gridsync.cuh"
#include "mp.h"
#include "mp_slab.cuh"
#include "warpsum.cuh"

namespace lbg {
namespace {

constexpr int RT32 = 512, RT64 = 256;   // most threads per block (128 / 255 registers)
constexpr int RES_CLUSTER = 16;

template <bool F64>
struct Real;
template <>
struct Real<false> {
    using T = float;
    static constexpr int threads = RT32;
    static constexpr int words = 4;   // shared-memory record of a node's P: one 16-byte access
};
template <>
struct Real<true> {
    using T = double;
    static constexpr int threads = RT64;
    static constexpr int words = 3;
};

struct MpResidentArgs {
    MpArgs32 a32;
    MpArgs64 a64;
    GridSync *sync;
    GridWait wait;
    const uint32_t *fidx;    // lattice indices of the Nf fluid nodes, in lattice order
    const uint32_t *place;   // lattice index -> fluid node
    unsigned Nf;
    int par, nsteps;         // reads P[par], A[par]; leaves P, A after nsteps in [par ^ 1]
    float4 *scratch32;       // grid: the other buffer of the steps
    double *scratch64[3];
    double *part;            // [step][warp][3]
    unsigned *failed;
};

__device__ __forceinline__ unsigned map_rank(unsigned addr, unsigned rank)
{
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}

__device__ __forceinline__ float4 ld_cluster4(unsigned addr)
{
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}

__device__ __forceinline__ double ld_cluster_f64(unsigned addr)
{
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(addr) : "memory");
    return v;
}

template <bool F64, bool CLUSTER>
__global__ void __launch_bounds__(Real<F64>::threads, 1) k_mp_resident(const MpResidentArgs r)
{
    using R = typename Real<F64>::T;
    constexpr int W = Real<F64>::words;
    // neighbour addresses [18][T]; CLUSTER: P records [2][T][W]; F64: VACF terms [warps][3][32]
    extern __shared__ __align__(16) unsigned char smraw[];
    const unsigned T = blockDim.x, tid = threadIdx.x, lane = tid & 31;
    const unsigned rank = blockIdx.x;   // CLUSTER: one cluster, block = rank
    const unsigned i = rank * T + tid, nwarps = gridDim.x * (T / 32), warp = i / 32;
    const bool mine = i < r.Nf;
    R *const rec = reinterpret_cast<R *>(smraw);                                  // CLUSTER
    unsigned *const nbr = reinterpret_cast<unsigned *>(smraw + (CLUSTER ? 2 * (size_t)T * W * sizeof(R) : 0)) + tid;
    double *const terms = reinterpret_cast<double *>(nbr - tid + (size_t)18 * T) + (tid / 32) * 96;   // F64
    const unsigned rec0 = CLUSTER ? smem_addr(smraw) : 0u;
    const unsigned flip = CLUSTER ? (unsigned)(T * W * sizeof(R)) : 0u;   // bytes between the two P buffers

    const int lx = F64 ? r.a64.lx : r.a32.lx, ly = F64 ? r.a64.ly : r.a32.ly, lz = F64 ? r.a64.lz : r.a32.lz;
    const bool ads = F64 ? r.a64.ads != 0 : r.a32.ads != 0;
    R s[Q];              // s[l]: scattering from r + c_l into the node
    R p[3] = {}, A[3] = {}, us[3] = {}, D = 0;   // D: net scattering (FP32), remaining fraction (FP64)
    bool inter = false;
    unsigned node = 0;
#pragma unroll
    for (int l = 0; l < Q; ++l) s[l] = 0;
    if (mine) {
        node = r.fidx[i];
        const uint32_t m = F64 ? r.a64.mask[node] : r.a32.mask[node];
        inter = ads && (m & INTERFACIAL_BIT);
        const int x = (int)(node % (unsigned)lx);
        const unsigned yz = node / (unsigned)lx;
        const int y = (int)(yz % (unsigned)ly), z = (int)(yz / (unsigned)ly);
        const int sy = lx, sz = lx * ly;
        const int X[3] = {wrap_minus(x, lx), x, wrap_plus(x, lx)};
        const int Y[3] = {wrap_minus(y, ly) * sy, y * sy, wrap_plus(y, ly) * sy};
        const int Z[3] = {wrap_minus(z, lz) * sz, z * sz, wrap_plus(z, lz) * sz};
        static_for<1, Q>([&](auto L) {
            constexpr int l = decltype(L)::value;
            constexpr Vel c = vel(l);
            const bool blocked = (m >> inv(l)) & 1u;   // r + c_l is solid
            const unsigned rp = (unsigned)(X[c.x + 1] + Y[c.y + 1] + Z[c.z + 1]);
            if constexpr (F64) {
                s[l] = r.a64.coef[(long long)(l - 1) * r.a64.N + node];
            } else {
                const float4 vn = r.a32.V[rp];
                s[l] = mp32_scatter(blocked, r.a32.a1[wclass(l)], mp32_cdot<-c.x, -c.y, -c.z>(vn), r.a32.lwh[wclass(l)]);
            }
            // a blocked link's probability is 0: any record of finite values will do (its own)
            if constexpr (CLUSTER) {
                const unsigned q = blocked ? i : r.place[rp], owner = q / T;
                nbr[(l - 1) * T] = map_rank(rec0 + (unsigned)((q - owner * T) * W * sizeof(R)), owner);
            } else {
                nbr[(l - 1) * T] = blocked ? node : rp;
            }
        });
        if constexpr (F64) {
            for (int d = 0; d < 3; ++d) {
                p[d] = r.a64.P[r.par][d][node];
                us[d] = r.a64.us[d][node];
                if (inter) A[d] = r.a64.A[r.par][d][node];
            }
            D = r.a64.frac[node];
        } else {
            const float4 q = r.a32.P[r.par][node], ax = r.a32.aux[node];
            p[0] = q.x, p[1] = q.y, p[2] = q.z;
            us[0] = ax.x, us[1] = ax.y, us[2] = ax.z;
            D = ax.w;
            if (inter) {
                const float4 qa = r.a32.A[r.par][node];
                A[0] = qa.x, A[1] = qa.y, A[2] = qa.z;
            }
        }
    }
    auto put = [&](unsigned buf) {   // own P into the cluster's buffer
#pragma unroll
        for (int d = 0; d < 3; ++d) rec[(buf * T + tid) * W + d] = p[d];
    };
    if constexpr (CLUSTER) {
        if (mine) put(0);
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else {
        __syncthreads();
    }
    // GRID: step k reads buffer k (0: P[par]), writes buffer k + 1, the last one into P[par ^ 1]
    auto is_out = [&](int k) { return ((r.nsteps - k) & 1) == 0; };   // buffer k (k >= 1) is P[par ^ 1]
    bool ok = true;
    for (int k = 0; k < r.nsteps && ok; ++k) {
        // ---- VACF terms of P(now)
        double *out = r.part + ((size_t)k * nwarps + warp) * 3;
        if constexpr (F64) {
            __syncwarp();
#pragma unroll
            for (int d = 0; d < 3; ++d) terms[d * 32 + lane] = p[d] * us[d];
            __syncwarp();
            // eight lanes per component: 3 + 3 additions, against 15 of a tree per component
            double t = 0.0;
            if (lane < 24) {
                const double *q = terms + (lane >> 3) * 32 + (lane & 7);
                t = ((q[0] + q[8]) + q[16]) + q[24];
            }
            t = t + __shfl_down_sync(0xffffffffu, t, 4);
            t = t + __shfl_down_sync(0xffffffffu, t, 2);
            t = t + __shfl_down_sync(0xffffffffu, t, 1);
            if (lane < 24 && (lane & 7) == 0) out[lane >> 3] = t;
        } else {
            const float t[3] = {p[0] * us[0], p[1] * us[1], p[2] * us[2]};
            const double w = warp_sum3_finite(t);
            if (lane < 3) out[lane] = w;
        }
        // ---- the step
        if (mine) {
            R n[3] = {};
            if constexpr (F64) {
                const double *src[3];
                if constexpr (!CLUSTER)
                    for (int d = 0; d < 3; ++d)
                        src[d] = k == 0 ? r.a64.P[r.par][d] : (is_out(k) ? r.a64.P[r.par ^ 1][d] : r.scratch64[d]);
                static_for<1, Q>([&](auto L) {
                    constexpr int l = decltype(L)::value;
                    double pn[3];
                    if constexpr (CLUSTER) {
                        const unsigned ad = nbr[(l - 1) * T] + (k & 1) * flip;
#pragma unroll
                        for (int d = 0; d < 3; ++d) pn[d] = ld_cluster_f64(ad + 8u * d);
                    } else {
                        const unsigned o = nbr[(l - 1) * T];
#pragma unroll
                        for (int d = 0; d < 3; ++d) pn[d] = __ldcg(src[d] + o);
                    }
#pragma unroll
                    for (int d = 0; d < 3; ++d)
                        n[d] = r.a64.fused ? __fma_rn(pn[d], s[l], n[d]) : n[d] + pn[d] * s[l];
                });
                if (!inter) {
#pragma unroll
                    for (int d = 0; d < 3; ++d)
                        n[d] = r.a64.fused ? __fma_rn(D, p[d], n[d]) : n[d] + D * p[d];
                } else {
                    const double f2 = D - r.a64.ka;
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        n[d] = n[d] + f2 * p[d] + A[d] * r.a64.kd;
                        A[d] = A[d] * r.a64.one_minus_kd + p[d] * r.a64.ka;
                    }
                }
            } else {
                const float4 *src = nullptr;
                if constexpr (!CLUSTER) src = k == 0 ? r.a32.P[r.par] : (is_out(k) ? r.a32.P[r.par ^ 1] : r.scratch32);
                const float4 own = make_float4(p[0], p[1], p[2], 0.0f);
                static_for<1, Q>([&](auto L) {
                    constexpr int l = mp_link_order(decltype(L)::value);
                    float4 pn;
                    if constexpr (CLUSTER) pn = ld_cluster4(nbr[(l - 1) * T] + (k & 1) * flip);
                    else pn = __ldcg(src + nbr[(l - 1) * T]);
                    mp32_link(s[l], pn, own, n[0], n[1], n[2]);
                });
                mp32_finish(own, D, n[0], n[1], n[2]);
                if (inter) {
                    const float4 qa = mp32_adsorb(own, make_float4(A[0], A[1], A[2], 0.0f), r.a32.ka, r.a32.kd,
                                                  r.a32.one_minus_kd, n[0], n[1], n[2]);
                    A[0] = qa.x, A[1] = qa.y, A[2] = qa.z;
                }
            }
#pragma unroll
            for (int d = 0; d < 3; ++d) p[d] = n[d];
            if constexpr (CLUSTER) {
                put((k + 1) & 1);
            } else if constexpr (F64) {
                for (int d = 0; d < 3; ++d) (is_out(k + 1) ? r.a64.P[r.par ^ 1][d] : r.scratch64[d])[node] = p[d];
            } else {
                (is_out(k + 1) ? r.a32.P[r.par ^ 1] : r.scratch32)[node] = make_float4(p[0], p[1], p[2], 0.0f);
            }
        }
        if constexpr (CLUSTER) {
            asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        } else if (k + 1 < r.nsteps) {
            unsigned long long v;
            unsigned b;
            ok = grid_barrier<false>(r.sync, (unsigned)k, r.wait, v, b);
        }
    }
    if (!ok && tid == 0) *r.failed = 1u;
    if (mine && ok) {
        if constexpr (CLUSTER) {
            if constexpr (F64) {
                for (int d = 0; d < 3; ++d) r.a64.P[r.par ^ 1][d][node] = p[d];
            } else {
                r.a32.P[r.par ^ 1][node] = make_float4(p[0], p[1], p[2], 0.0f);
            }
        }
        if (inter) {
            if constexpr (F64) {
                for (int d = 0; d < 3; ++d) r.a64.A[r.par ^ 1][d][node] = A[d];
            } else {
                r.a32.A[r.par ^ 1][node] = make_float4(A[0], A[1], A[2], 0.0f);
            }
        }
    }
}

// vacf[3 k + d] = sum over the warps of part[k][warp][d]: 32 strided lanes, then a tree.
__global__ void __launch_bounds__(96) k_mp_vacf(const double *part, unsigned nwarps, double *vacf)
{
    const unsigned lane = threadIdx.x & 31, d = threadIdx.x >> 5;
    const double *p = part + (size_t)blockIdx.x * nwarps * 3 + d;
    double s = 0.0;
    for (unsigned w = lane; w < nwarps; w += 32u) s = s + p[3 * (size_t)w];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s = s + __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) vacf[3 * (size_t)blockIdx.x + d] = s;
}

__global__ void k_mp_place(const uint32_t *fidx, unsigned nf, uint32_t *place)
{
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nf) place[fidx[i]] = i;
}

__global__ void k_mp_fidx(const uint32_t *cpos, unsigned nf, int lx, int ly, int xbits, int ybits, uint32_t *fidx)
{
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nf) return;
    const unsigned c = cpos[i], x = c & ((1u << xbits) - 1u), y = (c >> xbits) & ((1u << ybits) - 1u), z = c >> (xbits + ybits);
    fidx[i] = x + (unsigned)lx * (y + (unsigned)ly * z);
}

template <bool F64, bool CLUSTER>
size_t smem_of(unsigned T)
{
    using R = typename Real<F64>::T;
    return (size_t)18 * T * sizeof(unsigned) + (CLUSTER ? 2 * (size_t)T * Real<F64>::words * sizeof(R) : 0) +
           (F64 ? (size_t)T / 32 * 96 * sizeof(double) : 0);
}

template <bool F64, bool CLUSTER>
cudaLaunchConfig_t config(unsigned blocks, unsigned threads, cudaLaunchAttribute *at, cudaStream_t s)
{
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(blocks);
    c.blockDim = dim3(threads);
    c.dynamicSmemBytes = smem_of<F64, CLUSTER>(threads);
    c.stream = s;
    if (CLUSTER) {
        at->id = cudaLaunchAttributeClusterDimension;
        at->val.clusterDim.x = blocks;
        at->val.clusterDim.y = at->val.clusterDim.z = 1;
    } else {
        at->id = cudaLaunchAttributeCooperative;
        at->val.cooperative = 1;
    }
    c.attrs = at;
    c.numAttrs = 1;
    return c;
}

template <bool F64, bool CLUSTER>
bool fits(unsigned blocks, unsigned threads, int sms)
{
    auto *k = k_mp_resident<F64, CLUSTER>;
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem_of<F64, CLUSTER>(Real<F64>::threads)) != cudaSuccess)
        return false;
    if (CLUSTER) {
        cudaLaunchAttribute at;
        cudaLaunchConfig_t c = config<F64, CLUSTER>(blocks, threads, &at, nullptr);
        int n = 0;
        return cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
               cudaOccupancyMaxActiveClusters(&n, k, &c) == cudaSuccess && n >= 1;
    }
    int per_sm = 0;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, (int)threads, smem_of<F64, CLUSTER>(threads)) ==
               cudaSuccess &&
           (long long)per_sm * sms >= (long long)blocks;
}

template <bool F64>
bool plan_of(unsigned Nf, const char *mode, int sms, bool coop, MpResidentPlan &p)
{
    auto round32 = [](unsigned n) { return (n + 31u) / 32u * 32u; };
    // cluster: FP64 keeps one warp per quarter of an SM (its instructions are what a step costs)
    const unsigned most = F64 && std::strcmp(mode, "cluster") ? 128u : (unsigned)Real<F64>::threads;
    if (std::strcmp(mode, "grid") && Nf <= RES_CLUSTER * most) {
        p.blocks = RES_CLUSTER;
        while (p.blocks > 1 && 32u * (p.blocks / 2) >= Nf) p.blocks /= 2;
        p.threads = round32((Nf + p.blocks - 1) / p.blocks);
        p.cluster = true;
        if (fits<F64, true>(p.blocks, p.threads, sms)) return true;
        cudaGetLastError();
    }
    p = MpResidentPlan{};
    if (!coop || Nf > (unsigned)(sms * Real<F64>::threads)) return false;
    p.threads = std::max(F64 ? 32u : 128u, round32((Nf + sms - 1) / sms));
    p.blocks = (Nf + p.threads - 1) / p.threads;
    if (fits<F64, false>(p.blocks, p.threads, sms)) return true;
    cudaGetLastError();
    p = MpResidentPlan{};
    return false;
}

}  // namespace

// LBGPU_MP_RESIDENT=0: one launch per step; =grid / =cluster: that form where it fits.
MpResidentPlan plan_mp_resident(unsigned Nf, bool f64)
{
    MpResidentPlan p{};
    const char *env = std::getenv("LBGPU_MP_RESIDENT");
    const char *mode = env ? env : "";
    int dev = 0, sms = 0, coop = 0;
    if (!std::strcmp(mode, "0") || Nf == 0 || cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess) {
        cudaGetLastError();
        return p;
    }
    if (f64) plan_of<true>(Nf, mode, sms, coop != 0, p);
    else plan_of<false>(Nf, mode, sms, coop != 0, p);
    return p;
}

size_t mp_resident_sync_bytes() { return sizeof(GridSync); }

cudaError_t launch_mp_place(const uint32_t *fidx, unsigned nf, uint32_t *place, cudaStream_t s)
{
    k_mp_place<<<(nf + 255) / 256, 256, 0, s>>>(fidx, nf, place);
    return cudaGetLastError();
}

cudaError_t launch_mp_fidx(const uint32_t *cpos, unsigned nf, int lx, int ly, int xbits, int ybits, uint32_t *fidx,
                           cudaStream_t s)
{
    k_mp_fidx<<<(nf + 255) / 256, 256, 0, s>>>(cpos, nf, lx, ly, xbits, ybits, fidx);
    return cudaGetLastError();
}

cudaError_t launch_mp_resident(const MpResident &m, const MpArgs64 *a64, const MpArgs32 *a32, int par, int nsteps,
                               double *vacf, cudaStream_t s)
{
    MpResidentArgs r;
    std::memset(&r, 0, sizeof(r));
    if (a64) r.a64 = *a64;
    else r.a32 = *a32;
    r.wait = grid_wait();
    r.sync = static_cast<GridSync *>(m.sync);
    r.fidx = m.fidx;
    r.place = m.place;
    r.Nf = m.Nf;
    r.par = par;
    r.nsteps = nsteps;
    r.scratch32 = static_cast<float4 *>(m.scratch);
    if (a64)
        for (int d = 0; d < 3; ++d) r.scratch64[d] = static_cast<double *>(m.scratch) + d * a64->N;
    r.part = m.part;
    r.failed = m.failed;
    cudaError_t e = cudaMemsetAsync(m.failed, 0, sizeof(unsigned), s);
    if (e == cudaSuccess && !m.plan.cluster) e = cudaMemsetAsync(m.sync, 0, sizeof(GridSync), s);
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute at;
    const unsigned b = m.plan.blocks, t = m.plan.threads;
    if (a64 && m.plan.cluster) {
        cudaLaunchConfig_t c = config<true, true>(b, t, &at, s);
        e = cudaLaunchKernelEx(&c, k_mp_resident<true, true>, r);
    } else if (a64) {
        cudaLaunchConfig_t c = config<true, false>(b, t, &at, s);
        e = cudaLaunchKernelEx(&c, k_mp_resident<true, false>, r);
    } else if (m.plan.cluster) {
        cudaLaunchConfig_t c = config<false, true>(b, t, &at, s);
        e = cudaLaunchKernelEx(&c, k_mp_resident<false, true>, r);
    } else {
        cudaLaunchConfig_t c = config<false, false>(b, t, &at, s);
        e = cudaLaunchKernelEx(&c, k_mp_resident<false, false>, r);
    }
    if (e != cudaSuccess) return e;
    k_mp_vacf<<<(unsigned)nsteps, 96, 0, s>>>(m.part, b * (t / 32), vacf);
    return cudaGetLastError();
}

}  // namespace lbg
