// flow_f32_resident.cu -- many FP32 in-place steps of one box in one launch.
//
// A box whose step takes a few microseconds spends most of its time between launches (1.04 us in a
// CUDA graph, 3.3 us on a stream) and, in the reference loop, in the check launch's reduction and
// decision.  Here one thread owns one fluid node for the whole launch: its gather offsets are
// formed once, a step is a load, a collision and a store, and the steps are separated by a barrier:
//
//   * up to 16 x 512 fluid nodes (fixed steps) or 16 x 160 (the reference loop): one thread-block cluster holds every population in its blocks'
//     shared memory; odd steps gather and scatter through distributed shared memory, the barrier is
//     the cluster's (about 0.2 us);
//   * up to one 512-thread block per SM (77,824 fluid nodes): a cooperative grid, populations in
//     global memory (L2), gridsync.cuh's barrier.
//
// The reference loop needs no second barrier for its decision: S_t is collided ahead of it, the
// maximum of |j - j_old| over S_t travels with the barrier that ends that collision, and when the
// decision is another one than assumed (exit, or force switched on), each thread still has the 19
// values it read and puts them back into the slots they came from (the same slots it wrote; no
// other thread touches them between two barriers).  The arithmetic is aa32.cuh's, so the states are
// those of the launch-per-step path bit for bit.
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <string>

#include "aa32.cuh"
#include "compact.cuh"
#include "ctx.h"
#include "flow.h"
#include "gridsync.cuh"

namespace lbg {
namespace {

constexpr int RES_THREADS = 512;     // per block: up to 128 registers, the collision and 19 kept values
constexpr int RES_CLUSTER = 16;      // blocks of a cluster (16 needs the non-portable size)
constexpr unsigned STRIDE = 1u << 20;   // slot l of node i as l * STRIDE + i while the offsets are formed

struct ResidentArgs {
    FlowArgs32 a;
    GridSync *sync;
    GridWait wait;
    int nsteps;          // steps of this launch (reference loop: at most)
    int phase;           // AA phase of the state (1: swapped)
    int fm0, fc0, fon;   // fixed steps: moment / collision force of the first step, force of the later ones
};

__device__ __forceinline__ float ld_cluster(unsigned addr)
{
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}

__device__ __forceinline__ void st_cluster(unsigned addr, float v)
{
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}

__device__ __forceinline__ unsigned map_to_rank(unsigned addr, unsigned rank)
{
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}

__device__ __forceinline__ unsigned cluster_rank()
{
    unsigned r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

__device__ __forceinline__ void cluster_barrier()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The node's populations: where they live and how the in-place step reads and writes them.
template <bool CLUSTER>
struct Slots {
    unsigned *off;    // this thread's column of the offset table, [l * T]
    float *own;       // CLUSTER: this thread's column of the populations, [l * T]; else g0 + i
    float *g;
    unsigned T, Nf;

    __device__ __forceinline__ void load(float (&f)[Q], int phase) const
    {
        if (phase) {
#pragma unroll
            for (int l = 0; l < Q; ++l) f[l] = CLUSTER ? ld_cluster(off[l * T]) : __ldcg(g + off[l * T]);
        } else {
#pragma unroll
            for (int l = 0; l < Q; ++l) f[l] = CLUSTER ? own[l * T] : __ldcg(own + (size_t)l * Nf);
        }
    }
    // the collided populations f, each to the slot its opposite was read from
    __device__ __forceinline__ void store(const float (&f)[Q], int phase) const
    {
        if (phase) {
#pragma unroll
            for (int l = 0; l < Q; ++l) put(off[inv(l) * T], f[l]);
        } else {
#pragma unroll
            for (int l = 0; l < Q; ++l) put_own(l, f[inv(l)]);
        }
    }
    // f as load() read it, back to the same slots
    __device__ __forceinline__ void restore(const float (&f)[Q], int phase) const
    {
#pragma unroll
        for (int l = 0; l < Q; ++l) {
            if (phase) put(off[l * T], f[l]);
            else put_own(l, f[l]);
        }
    }

private:
    __device__ __forceinline__ void put(unsigned o, float v) const
    {
        if constexpr (CLUSTER) st_cluster(o, v);
        else g[o] = v;
    }
    __device__ __forceinline__ void put_own(int l, float v) const
    {
        if constexpr (CLUSTER) own[l * T] = v;
        else own[(size_t)l * Nf] = v;
    }
};

// Per rendezvous parity, the values of the cluster's blocks (written into every block's copy).
struct ClusterSlots {
    unsigned long long value[2][RES_CLUSTER];
    unsigned bits[2][RES_CLUSTER];
};

template <bool CLUSTER, bool LOOP>
__global__ void __launch_bounds__(RES_THREADS, 1) k_aa_resident(const ResidentArgs r)
{
    extern __shared__ unsigned sm[];   // offsets [Q][T]; CLUSTER: populations [Q][T]
    __shared__ FlowCtl ctl;            // LOOP: this block's copy of the control block
    __shared__ ClusterSlots cs;
    __shared__ unsigned long long wval[RES_THREADS / 32];
    __shared__ unsigned wbit[RES_THREADS / 32];
    const FlowArgs32 &a = r.a;
    const unsigned T = blockDim.x, tid = threadIdx.x;
    const unsigned rank = CLUSTER ? cluster_rank() : blockIdx.x;
    const unsigned i = rank * T + tid;
    const bool mine = i < a.Nf;
    Slots<CLUSTER> s;
    s.off = sm + tid;
    s.g = a.g0;
    s.own = CLUSTER ? reinterpret_cast<float *>(sm) + (size_t)Q * T + tid : a.g0 + i;
    s.T = T;
    s.Nf = a.Nf;
    unsigned pos = 0;
    if (mine) {
        FlowArgs32 b = a;
        if (CLUSTER) b.Nf = STRIDE;
        pos = a.cpos[i];
        const unsigned pop0 = CLUSTER ? smem_addr(sm + (size_t)Q * T) : 0u;
        aa_gather_offsets(b, i, pos, a.cmask[i], [&](int l, unsigned o) {
            if constexpr (CLUSTER) {
                const unsigned slot = o / STRIDE, node = o % STRIDE, owner = node / T;
                s.off[l * T] = map_to_rank(pop0 + 4u * (slot * T + (node - owner * T)), owner);
            } else {
                s.off[l * T] = o;
            }
        });
        if constexpr (CLUSTER) {
#pragma unroll
            for (int l = 0; l < Q; ++l) s.own[l * T] = a.g0[(size_t)l * a.Nf + i];
        }
    }
    if (LOOP && tid == 0) ctl = *a.ctl;
    if constexpr (CLUSTER) cluster_barrier();
    else __syncthreads();

    unsigned round = 0;
    bool ok = true;
    auto barrier = [&]() {
        if constexpr (CLUSTER) {
            cluster_barrier();
        } else {
            unsigned long long v;
            unsigned b;
            ok = grid_barrier<false>(r.sync, round++, r.wait, v, b);
        }
    };
    int phase = r.phase;
    float f[Q];
    if constexpr (!LOOP) {
        for (int k = 0; k < r.nsteps && ok; ++k) {
            if (mine) {
                s.load(f, phase);
                aa_relax<7>(f, a, k == 0 ? r.fm0 : (k == 1 ? r.fc0 : r.fon), k == 0 ? r.fc0 : r.fon);
                s.store(f, phase);
            }
            phase ^= 1;
            if (CLUSTER || k + 1 < r.nsteps) barrier();
        }
    } else {
        // the barrier that ends a collision, with the maximum of v and the OR of b over the box
        auto exchange = [&](unsigned long long &v, unsigned &b) {
            if constexpr (!CLUSTER) {
                ok = grid_barrier<true>(r.sync, round++, r.wait, v, b);
            } else {
                const unsigned lane = tid & 31, par = round++ & 1u, nb = gridDim.x;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    const unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o);
                    v = w > v ? w : v;
                }
                b = __reduce_or_sync(0xffffffffu, b);
                if (lane == 0) {
                    wval[tid >> 5] = v;
                    wbit[tid >> 5] = b;
                }
                __syncthreads();
                if (tid < nb) {   // one destination block per thread
                    for (unsigned w = 0; w < T / 32; ++w) {
                        v = wval[w] > v ? wval[w] : v;
                        b |= wbit[w];
                    }
                    asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(map_to_rank(smem_addr(&cs.value[par][rank]), tid)),
                                 "l"(v) : "memory");
                    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(map_to_rank(smem_addr(&cs.bits[par][rank]), tid)),
                                 "r"(b) : "memory");
                }
                cluster_barrier();
                v = 0;
                b = 0;
                for (unsigned q = 0; q < nb; ++q) {
                    v = cs.value[par][q] > v ? cs.value[par][q] : v;
                    b |= cs.bits[par][q];
                }
            }
        };
        double jx = 0.0, jy = 0.0, jz = 0.0;
        const unsigned p = mine ? lattice_of(a, pos) : 0u;
        if (mine) {
            jx = a.jx[p];
            jy = a.jy[p];
            jz = a.jz[p];
            s.load(f, phase);
            aa_relax<7>(f, a, ctl.aa_fm, ctl.aa_fc);
            s.store(f, phase);
        }
        phase ^= 1;
        barrier();
        for (int k = 1; ok; ++k) {
            // S_t: check it, and collide it ahead of the decision unless the launch ends with it
            const bool last = k >= r.nsteps || (ctl.max_steps > 0 && ctl.t >= ctl.max_steps);
            const int fm = ctl.check_fm, fc = ctl.aa_fc;
            unsigned long long err = 0;
            unsigned bad = 0;
            if (mine) {
                s.load(f, phase);
                double nx, ny, nz;
                exact_flux(f, nx, ny, nz);
                if (fm) {
                    nx += a.half_force[0];
                    ny += a.half_force[1];
                    nz += a.half_force[2];
                }
                err = flux_change_bits(nx - jx, ny - jy, nz - jz);
                bad = check_dev19(f, a);
                jx = nx;
                jy = ny;
                jz = nz;
                if (!last) {
                    float q[Q];
#pragma unroll
                    for (int l = 0; l < Q; ++l) q[l] = f[l];
                    aa_relax<7>(q, a, fm, fc);
                    s.store(q, phase);
                }
            }
            exchange(err, bad);
            if (!ok) break;
            __syncthreads();   // every thread has read the control block
            if (tid == 0) decide32(ctl, err, bad, phase, rank == 0 ? a.hist : nullptr);
            __syncthreads();
            if (last) break;
            if (ctl.done) {
                if (mine) s.restore(f, phase);
                break;
            }
            if (ctl.aa_fc != fc) {   // the force acts from this collision on: again, with it
                if (mine) {
                    aa_relax<7>(f, a, fm, ctl.aa_fc);
                    s.store(f, phase);
                }
                barrier();
            }
            phase ^= 1;
        }
        if (mine && ok) {
            a.jx[p] = jx;
            a.jy[p] = jy;
            a.jz[p] = jz;
        }
        if (rank == 0 && tid == 0) store_ctl(a.ctl, ctl);
    }
    if constexpr (CLUSTER) {
        cluster_barrier();   // a block's shared memory holds its nodes' populations
        if (mine) {
#pragma unroll
            for (int l = 0; l < Q; ++l) a.g0[(size_t)l * a.Nf + i] = s.own[l * T];
        }
    } else if (!ok && tid == 0) {
        atomicOr(&a.ctl->status, (unsigned)LBGPU_ERR_TIMEOUT);
    }
}

size_t smem_bytes(bool cluster, unsigned T) { return (size_t)Q * T * sizeof(unsigned) * (cluster ? 2 : 1); }

template <bool CLUSTER, bool LOOP>
cudaError_t launch(const ResidentPlan &plan, const ResidentArgs &r, cudaStream_t s)
{
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(plan.blocks);
    c.blockDim = dim3(plan.threads);
    c.dynamicSmemBytes = smem_bytes(CLUSTER, plan.threads);
    c.stream = s;
    cudaLaunchAttribute at;
    if (CLUSTER) {
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = plan.blocks;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
    } else {
        at.id = cudaLaunchAttributeCooperative;
        at.val.cooperative = 1;
    }
    c.attrs = &at;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, k_aa_resident<CLUSTER, LOOP>, r);
}

template <bool CLUSTER, bool LOOP>
bool fits(unsigned blocks, unsigned threads, int sms)
{
    auto *k = k_aa_resident<CLUSTER, LOOP>;
    const size_t bytes = smem_bytes(CLUSTER, threads);
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes(CLUSTER, RES_THREADS)) != cudaSuccess)
        return false;
    if (CLUSTER) {
        if (cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) return false;
        cudaLaunchConfig_t c = {};
        c.gridDim = dim3(blocks);
        c.blockDim = dim3(threads);
        c.dynamicSmemBytes = bytes;
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = blocks;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        c.attrs = &at;
        c.numAttrs = 1;
        int n = 0;
        return cudaOccupancyMaxActiveClusters(&n, k, &c) == cudaSuccess && n >= 1;
    }
    int per_sm = 0;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, (int)threads, bytes) == cudaSuccess &&
           (long long)per_sm * sms >= (long long)blocks;
}

}  // namespace

// Where the box's steps run (see the head of this file).  The lines: fixed steps run in a cluster
// wherever the box fits one, the reference loop while a block has at most 5 warps (its check keeps
// 16 SMs busier than the grid's barrier costs), both on a grid up to one node per thread of one
// block per SM; larger boxes keep one launch per step.  us per step, launch per step / grid /
// cluster:
//   fluid nodes   fixed steps           reference loop
//      2,457      5.06 / 2.03 / 1.00     8.47 / 3.59 / 3.23
//      6,346      5.12 / 2.02 / 1.47     8.46 / 3.63 / 4.92
//     38,393      5.12 / 2.68 / -        9.69 / 4.78 / -
//     74,460      5.63 / 3.37 / -       12.1  / 6.57 / -
// LBGPU_AA_RESIDENT=0 keeps one launch per step, =grid and =cluster take that form where it fits.
ResidentPlan plan_resident32(unsigned Nf, bool wide, bool loop)
{
    ResidentPlan p{};
    const char *env = std::getenv("LBGPU_AA_RESIDENT");
    const std::string mode = env ? env : "";
    int dev = 0, sms = 0, coop = 0;
    if (mode == "0" || wide || Nf == 0 || cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess) {
        cudaGetLastError();
        return p;
    }
    auto round32 = [](unsigned n) { return (n + 31u) / 32u * 32u; };
    const unsigned most = loop && mode != "cluster" ? 160u : (unsigned)RES_THREADS;
    if (mode != "grid" && Nf <= RES_CLUSTER * most) {
        p.blocks = RES_CLUSTER;
        while (p.blocks > 1 && 32u * (p.blocks / 2) >= Nf) p.blocks /= 2;   // no empty block
        p.threads = round32((Nf + p.blocks - 1) / p.blocks);
        p.cluster = true;
        if (loop ? fits<true, true>(p.blocks, p.threads, sms) : fits<true, false>(p.blocks, p.threads, sms)) return p;
        cudaGetLastError();
        p = ResidentPlan{};
    }
    if (!coop || Nf > (unsigned)(sms * RES_THREADS)) return p;
    p.threads = std::max(128u, round32((Nf + sms - 1) / sms));
    p.blocks = (Nf + p.threads - 1) / p.threads;
    if (loop ? fits<false, true>(p.blocks, p.threads, sms) : fits<false, false>(p.blocks, p.threads, sms)) return p;
    cudaGetLastError();
    return ResidentPlan{};
}

size_t grid_sync_bytes() { return sizeof(GridSync); }

static cudaError_t run(const ResidentPlan &plan, ResidentArgs &r, void *sync, bool loop, cudaStream_t s)
{
    r.wait = grid_wait();
    r.sync = static_cast<GridSync *>(sync);
    if (plan.cluster) return loop ? launch<true, true>(plan, r, s) : launch<true, false>(plan, r, s);
    const cudaError_t e = cudaMemsetAsync(sync, 0, sizeof(GridSync), s);
    if (e != cudaSuccess) return e;
    return loop ? launch<false, true>(plan, r, s) : launch<false, false>(plan, r, s);
}

cudaError_t launch_resident_steps32(const ResidentPlan &plan, const FlowArgs32 &a, void *sync, int nsteps, int phase,
                                    int fm0, int fc0, int fon, cudaStream_t s)
{
    ResidentArgs r{};
    r.a = a;
    r.nsteps = nsteps;
    r.phase = phase;
    r.fm0 = fm0;
    r.fc0 = fc0;
    r.fon = fon;
    return run(plan, r, sync, false, s);
}

cudaError_t launch_resident_loop32(const ResidentPlan &plan, const FlowArgs32 &a, void *sync, int nsteps, int phase,
                                   cudaStream_t s)
{
    ResidentArgs r{};
    r.a = a;
    r.nsteps = nsteps;
    r.phase = phase;
    return run(plan, r, sync, true, s);
}

}  // namespace lbg
