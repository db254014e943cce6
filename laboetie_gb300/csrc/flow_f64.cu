// flow_f64.cu -- FP64 D3Q19 kernels (compiled with -fmad=false): the strict form, and the fused
// step of LBGPU_FP64_FUSED (64-bit fixed point, or explicit fused multiply-adds; flow64.cuh).
//
// Bit-exactness with the reference.  Every product and sum is evaluated in the operand order
// of the Fortran source with separate roundings (no fused multiply-add in this translation
// unit).  Terms that the reference multiplies by a velocity component of 0 are exactly +-0 and
// are left out; terms multiplied by +-1 are exact and become additions or subtractions.  Both
// transformations keep every intermediate value identical (at most the sign of an exact zero
// can differ), so the populations, densities and fluxes equal the reference's operation for
// operation.  This matters on GB300 beyond parity: FP64 issues at a small fraction of FP32,
// so every FP64 operation skipped is time saved.
//
// Streaming.  The reference swaps populations across fluid/solid links and then pushes
// (equilibration.f90:204-243).  Each population takes part in at most one swap, so the pair is
// exactly the pull rule  n_new(x,l) = n*(x - c_l, l)  if nature(x - c_l) == nature(x),
// else n*(x, inv l).  The kernels pull; bit l of the node flag word says which source to use.
#include "common.cuh"
#include "flow.h"
#include "flow64.cuh"
#include "lbgpu.h"

namespace lbg {
namespace {

constexpr int BLOCK = 256, STEP_BLOCK = 128;

struct Coords {
    int x, y, z;
    long long X[3], Y[3], Z[3];  // [c+1]: offset of coordinate (x - c) along each axis
};

__device__ __forceinline__ Coords coords_of(long long node, int lx, int ly, int lz)
{
    Coords k;
    const unsigned nd = (unsigned)node;
    k.x = (int)(nd % (unsigned)lx);
    const unsigned yz = nd / (unsigned)lx;
    k.y = (int)(yz % (unsigned)ly);
    k.z = (int)(yz / (unsigned)ly);
    const long long sx = 1, sy = lx, sz = (long long)lx * ly;
    // index [c+1] holds the coordinate of (x - c): c = -1 -> x+1, c = 0 -> x, c = 1 -> x-1
    k.X[0] = wrap_plus(k.x, lx) * sx;  k.X[1] = k.x * sx;  k.X[2] = wrap_minus(k.x, lx) * sx;
    k.Y[0] = wrap_plus(k.y, ly) * sy;  k.Y[1] = k.y * sy;  k.Y[2] = wrap_minus(k.y, ly) * sy;
    k.Z[0] = wrap_plus(k.z, lz) * sz;  k.Z[1] = k.z * sz;  k.Z[2] = wrap_minus(k.z, lz) * sz;
    return k;
}

// Pull the 19 populations of `node` from src with halfway bounce-back (equilibration.f90:204-243).
__device__ __forceinline__ void pull19(double (&n)[Q], const double *__restrict__ src,
                                       long long node, uint32_t m, const Coords &k, long long N)
{
    static_for<0, Q>([&](auto L) {
        constexpr int l = decltype(L)::value;
        constexpr Vel c = vel(l);
        if constexpr (l == 0) {
            n[0] = src[node];
        } else {
            const long long s = k.X[c.x + 1] + k.Y[c.y + 1] + k.Z[c.z + 1];
            n[l] = ((m >> l) & 1u) ? src[(long long)inv(l) * N + node] : src[(long long)l * N + s];
        }
    });
}

__device__ __forceinline__ double warp_max(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = max_nonneg(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ unsigned warp_or(unsigned v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v |= __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Block-wide max/or (any number of full warps up to BLOCK / 32); result valid in thread 0.
__device__ __forceinline__ void block_max_or(double &err, unsigned &bad)
{
    __shared__ double se[BLOCK / 32];
    __shared__ unsigned sb[BLOCK / 32];
    err = warp_max(err);
    bad = warp_or(bad);
    if (blockDim.x == 32) return;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) { se[wid] = err; sb[wid] = bad; }
    __syncthreads();
    if (wid == 0) {
        err = lane < (blockDim.x >> 5) ? se[lane] : 0.0;
        bad = lane < (blockDim.x >> 5) ? sb[lane] : 0u;
        err = warp_max(err);
        bad = warp_or(bad);
    }
}

// The phase machine of a step (decide64), executed by its last block once every block has
// contributed its |j - j_old| maximum.
__device__ void control_step(FlowCtl *c, double *hist)
{
    const unsigned long long eb = atomicExch(&c->err_bits, 0ull);
    const unsigned st = atomicOr(&c->status, 0u);
    FlowCtl d = *c;
    d.err_bits = 0ull;
    d.blocks_done = 0u;
    decide64(d, eb, st, hist);
    *c = d;
}

// Blocks per SM asked for, of 128 threads: measured on the same boxes, strict 237.5 us a step with 4,
// 239.9 with 5, 239.3 with 6, 248 with 8; fused 149.4 with 4, 140.2 with 5, 160 with 6.
template <int FMASK, bool FIELD, bool CHECK, bool REF, bool FUSED>
__global__ void __launch_bounds__(STEP_BLOCK, FUSED ? 5 : 4) k_flow_step(const FlowArgs64 a)
{
    int parity = a.parity, fm = a.force_moment, fc = a.force_collide;
    if constexpr (REF) {
        // written by the last block only, after every block has read it: plain loads, which one
        // request per SM serves
        if (a.ctl->done) return;
        parity = a.ctl->parity;
        fm = a.ctl->force_moment;
        fc = a.ctl->force_collide;
    }
    const double *__restrict__ src = parity ? a.f1 : a.f0;
    double *__restrict__ dst = parity ? a.f0 : a.f1;
    const long long N = a.N;
    // one thread per fluid node through the list (every lane of a warp does work), else one per
    // lattice node
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long node = a.fidx ? (i < a.Nf ? (long long)a.fidx[i] : N) : i;
    double err = 0.0;
    unsigned bad = 0;
    if (node < N) {
        const uint32_t m = a.mask[node];
        if (m & FLUID_BIT) {
            const Coords k = coords_of(node, a.lx, a.ly, a.lz);
            double n[Q];
            pull19(n, src, node, m, k, N);
            if constexpr (CHECK) bad = check19(n);
            double fx = 0.0, fy = 0.0, fz = 0.0;
            if constexpr (FIELD) {
                fx = a.Fx[node];
                fy = a.Fy[node];
                fz = a.Fz[node];
            } else {
                fx = a.F[0];
                fy = a.F[1];
                fz = a.F[2];
            }
            double rho, jx = 0.0, jy = 0.0, jz = 0.0;
            if constexpr (FUSED && !FIELD) {
                fused_step<FMASK, true, CHECK, false>(n, fm != 0, fc != 0, fx, fy, fz, a, jx, jy, jz);
            } else if constexpr (FUSED) {
                if (fm) moments19_pairs(n, fx / 2.0, fy / 2.0, fz / 2.0, rho, jx, jy, jz);
                else moments19_pairs(n, 0.0, 0.0, 0.0, rho, jx, jy, jz);
            } else {
                moments19_fast(n, fm != 0, fx, fy, fz, rho, jx, jy, jz);
            }
            if constexpr (CHECK) {
                const double ox = a.jx[node], oy = a.jy[node], oz = a.jz[node];
                err = max_nonneg(max_nonneg(fabs(jx - ox), fabs(jy - oy)), fabs(jz - oz));
            }
            if constexpr (FUSED && FIELD) {
                if (fc) collide_node_fused<FMASK, false>(n, rho, jx, jy, jz, fx, fy, fz, a);
                else collide_node_fused<0, true>(n, rho, jx, jy, jz, 0.0, 0.0, 0.0, a);
            } else if constexpr (!FUSED) {
                collide_strict<FMASK, !FIELD>(n, rho, jx, jy, jz, fx, fy, fz, a, fc != 0);
            }
#pragma unroll
            for (int l = 0; l < Q; ++l) dst[(long long)l * N + node] = n[l];
            // j last, as far as may be from the loads of the same lines: stored right after them, it
            // held the loads of the other warps up (1.26 M fluid nodes, fused loop: 411 us a step, 196
            // here; strict loop 541 and 511)
            if constexpr (CHECK) {
                a.jx[node] = jx;
                a.jy[node] = jy;
                a.jz[node] = jz;
            }
        }
    }
    if constexpr (CHECK) {
        block_max_or(err, bad);
        if (threadIdx.x == 0) {
            unsigned long long *eb = REF ? &a.ctl->err_bits : a.err_bits;
            unsigned *st = REF ? &a.ctl->status : a.status;
            atomic_max_nonneg(eb, err);
            if (bad) atomicOr(st, bad);
            if constexpr (REF) {
                __threadfence();
                const unsigned prev = atomicAdd(&a.ctl->blocks_done, 1u);
                if (prev == gridDim.x - 1) {
                    __threadfence();
                    control_step(a.ctl, a.hist);
                }
            }
        }
    }
}

// Collision only: pre-collision n in buffer `parity` (all fluid nodes), density and j from
// a.rho/a.j*, post-collision populations written to the other buffer; solid nodes copied.
template <int FMASK, bool FIELD>
__global__ void __launch_bounds__(BLOCK) k_collide(const FlowArgs64 a)
{
    const double *__restrict__ src = a.parity ? a.f1 : a.f0;
    double *__restrict__ dst = a.parity ? a.f0 : a.f1;
    const long long N = a.N;
    const long long node = (long long)blockIdx.x * BLOCK + threadIdx.x;
    if (node >= N) return;
    double n[Q];
#pragma unroll
    for (int l = 0; l < Q; ++l) n[l] = src[(long long)l * N + node];
    const uint32_t m = a.mask[node];
    if (m & FLUID_BIT) {
        double fx, fy, fz;
        if constexpr (FIELD) {
            fx = a.Fx[node];
            fy = a.Fy[node];
            fz = a.Fz[node];
        } else {
            fx = a.F[0];
            fy = a.F[1];
            fz = a.F[2];
        }
        collide_strict<FMASK, !FIELD>(n, a.rho[node], a.jx[node], a.jy[node], a.jz[node], fx, fy, fz, a,
                                      a.force_collide != 0);
    }
#pragma unroll
    for (int l = 0; l < Q; ++l) dst[(long long)l * N + node] = n[l];
}

// Bounce-back + streaming for every node (solid included): buffer `parity` -> nout.
__global__ void __launch_bounds__(BLOCK) k_stream(const FlowArgs64 a)
{
    const double *__restrict__ src = a.parity ? a.f1 : a.f0;
    const long long N = a.N;
    const long long node = (long long)blockIdx.x * BLOCK + threadIdx.x;
    if (node >= N) return;
    const uint32_t m = a.mask[node];
    const Coords k = coords_of(node, a.lx, a.ly, a.lz);
    double n[Q];
    pull19(n, src, node, m, k, N);
#pragma unroll
    for (int l = 0; l < Q; ++l) a.nout[(long long)l * N + node] = n[l];
}

// Moments of the populations in buffer `parity` at every node (equilibration.f90:248-343).
template <bool FIELD, bool PULL>
__global__ void __launch_bounds__(BLOCK) k_moments(const FlowArgs64 a)
{
    const double *__restrict__ src = a.parity ? a.f1 : a.f0;
    const long long N = a.N;
    const long long node = (long long)blockIdx.x * BLOCK + threadIdx.x;
    double err = 0.0;
    unsigned bad = 0;
    if (node < N) {
        const uint32_t m = a.mask[node];
        double n[Q];
        if constexpr (PULL) {
            const Coords k = coords_of(node, a.lx, a.ly, a.lz);
            pull19(n, src, node, m, k, N);
        } else {
#pragma unroll
            for (int l = 0; l < Q; ++l) n[l] = src[(long long)l * N + node];
        }
        bad = check19(n);
        double fx = 0.0, fy = 0.0, fz = 0.0;
        if constexpr (FIELD) {
            fx = a.Fx[node];
            fy = a.Fy[node];
            fz = a.Fz[node];
        } else if (a.force_moment && (m & FLUID_BIT)) {
            fx = a.F[0];
            fy = a.F[1];
            fz = a.F[2];
        }
        double rho, jx, jy, jz;
        moments19(n, fx / 2.0, fy / 2.0, fz / 2.0, rho, jx, jy, jz);
        const double ox = a.jx[node], oy = a.jy[node], oz = a.jz[node];
        err = max_nonneg(max_nonneg(fabs(jx - ox), fabs(jy - oy)), fabs(jz - oz));
        a.rho[node] = rho;
        a.jx[node] = jx;
        a.jy[node] = jy;
        a.jz[node] = jz;
        if (PULL && a.nout) {
#pragma unroll
            for (int l = 0; l < Q; ++l) a.nout[(long long)l * N + node] = n[l];
        }
    }
    block_max_or(err, bad);
    if (threadIdx.x == 0) {
        if (a.err_bits) atomic_max_nonneg(a.err_bits, err);
        if (bad && a.status) atomicOr(a.status, bad);
    }
}

// init_simu.f90:31-39 and equilibration.f90:75-80: raw n = w_l*rho into buffer `parity`.
__global__ void __launch_bounds__(BLOCK) k_init(const FlowArgs64 a, const double rho0)
{
    double *__restrict__ dst = a.parity ? a.f1 : a.f0;
    const long long N = a.N;
    const long long node = (long long)blockIdx.x * BLOCK + threadIdx.x;
    if (node >= N) return;
    const uint32_t m = a.mask[node];
    const double rho = (m & FLUID_BIT) ? rho0 : 0.0;
    a.rho[node] = rho;
    a.jx[node] = 0.0;
    a.jy[node] = 0.0;
    a.jz[node] = 0.0;
    static_for<0, Q>([&](auto L) {
        constexpr int l = decltype(L)::value;
        dst[(long long)l * N + node] = rho * a.K.a0[wclass(l)];
    });
}

unsigned grid_of(long long N) { return (unsigned)((N + BLOCK - 1) / BLOCK); }

// Threads per block of a step over n nodes.  A warp instruction of doubles occupies its quarter of
// an SM for 64 cycles whatever its lanes, so a small box is spread over the SMs warp by warp: up to
// 608 warps (152 SMs x 4 quarters) as one-warp blocks, then two-warp blocks up to 64 warps an SM.
// Above, four-warp blocks: a block's load, integer and FP64 phases overlap with those of the blocks
// beside it, and smaller blocks leave at finer grain (0.52 M fluid nodes, strict loop: 248 us a step
// with 256 threads, 241 with 128, 242 with 64; fused, 1.26 M: 154, 150, 151).
unsigned step_block(long long n)
{
    const long long warps = (n + 31) / 32;
    return warps <= 608 ? 32u : (warps <= 152 * 64 ? 64u : (unsigned)STEP_BLOCK);
}

template <bool FIELD, bool CHECK, bool REF, bool FUSED>
cudaError_t step_dispatch(const FlowArgs64 &a, int fmask, unsigned grid, unsigned block, cudaStream_t s)
{
    switch (fmask) {
    case 0: k_flow_step<0, FIELD, CHECK, REF, FUSED><<<grid, block, 0, s>>>(a); break;
    case 1: k_flow_step<1, FIELD, CHECK, REF, FUSED><<<grid, block, 0, s>>>(a); break;
    case 2: k_flow_step<2, FIELD, CHECK, REF, FUSED><<<grid, block, 0, s>>>(a); break;
    case 4: k_flow_step<4, FIELD, CHECK, REF, FUSED><<<grid, block, 0, s>>>(a); break;
    default: k_flow_step<7, FIELD, CHECK, REF, FUSED><<<grid, block, 0, s>>>(a); break;
    }
    return cudaGetLastError();
}

template <bool FUSED>
cudaError_t launch_step(const FlowArgs64 &a, int fmask, bool field, bool check, bool ref,
                        unsigned grid, unsigned block, cudaStream_t s)
{
    if (field) {
        // a per-node force field: every component may be non-zero
        if (ref) k_flow_step<7, true, true, true, FUSED><<<grid, block, 0, s>>>(a);
        else if (check) k_flow_step<7, true, true, false, FUSED><<<grid, block, 0, s>>>(a);
        else k_flow_step<7, true, false, false, FUSED><<<grid, block, 0, s>>>(a);
        return cudaGetLastError();
    }
    if (ref) return step_dispatch<false, true, true, FUSED>(a, fmask, grid, block, s);
    return check ? step_dispatch<false, true, false, FUSED>(a, fmask, grid, block, s)
                 : step_dispatch<false, false, false, FUSED>(a, fmask, grid, block, s);
}

}  // namespace

cudaError_t launch_flow_step_f64(const FlowArgs64 &a, int fmask, bool field, bool check,
                                 bool ref, cudaStream_t s)
{
    const long long n = a.fidx ? a.Nf : a.N;
    const unsigned block = step_block(n), grid = (unsigned)((n + block - 1) / block);
    return a.fused ? launch_step<true>(a, fmask, field, check, ref, grid, block, s)
                   : launch_step<false>(a, fmask, field, check, ref, grid, block, s);
}

cudaError_t launch_collide_f64(const FlowArgs64 &a, int fmask, bool field, cudaStream_t s)
{
    const unsigned g = grid_of(a.N);
    if (field) {
        k_collide<7, true><<<g, BLOCK, 0, s>>>(a);
    } else {
        switch (fmask) {
        case 0: k_collide<0, false><<<g, BLOCK, 0, s>>>(a); break;
        case 1: k_collide<1, false><<<g, BLOCK, 0, s>>>(a); break;
        case 2: k_collide<2, false><<<g, BLOCK, 0, s>>>(a); break;
        case 4: k_collide<4, false><<<g, BLOCK, 0, s>>>(a); break;
        default: k_collide<7, false><<<g, BLOCK, 0, s>>>(a); break;
        }
    }
    return cudaGetLastError();
}

cudaError_t launch_stream_f64(const FlowArgs64 &a, cudaStream_t s)
{
    k_stream<<<grid_of(a.N), BLOCK, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_moments_f64(const FlowArgs64 &a, bool field, cudaStream_t s)
{
    if (field) k_moments<true, false><<<grid_of(a.N), BLOCK, 0, s>>>(a);
    else k_moments<false, false><<<grid_of(a.N), BLOCK, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_finalize_f64(const FlowArgs64 &a, bool field, cudaStream_t s)
{
    if (field) k_moments<true, true><<<grid_of(a.N), BLOCK, 0, s>>>(a);
    else k_moments<false, true><<<grid_of(a.N), BLOCK, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_init_f64(const FlowArgs64 &a, double rho0, cudaStream_t s)
{
    k_init<<<grid_of(a.N), BLOCK, 0, s>>>(a, rho0);
    return cudaGetLastError();
}

}  // namespace lbg
