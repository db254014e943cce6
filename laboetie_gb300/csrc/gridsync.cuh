// gridsync.cuh -- a barrier over the blocks of one cooperative launch that also forms the maximum of
// a 64-bit value and the OR of status bits over the grid.
//
// Thread 0 of a block adds the block's values to the round's slot, arrives on a counter (release)
// and polls it (acquire) until every block has arrived.  The three slots rotate: after a round has
// passed, the slot of the round before it is read by nobody any more and is cleared for the round
// after next.  The poll is bounded.  A block whose wait runs out sets a high bit of the counter, which ends
// the waits of the others, as failed ones too; each such block reports it to the host itself, as the others may
// all have passed the launch's last rendezvous.  (A flag of its own beside the counter cost a step of 16,752
// fluid nodes 0.05 of 9.05 us.)
// 152 blocks: 1.2 us without values, 1.6 us with them (a launch in a CUDA graph costs 1.04 us, and
// a step that decides on a reduction needs its tail besides).
#pragma once

#include <cstdint>
#include <cstdlib>

#include "tma.cuh"

namespace lbg {

struct alignas(128) GridSync {
    struct alignas(128) Slot {
        unsigned long long value;
        unsigned bits;
    } slot[3];
    alignas(128) unsigned arrived;   // and GRID_FAILED
};
constexpr unsigned GRID_FAILED = 1u << 30;   // beyond the arrivals of a launch's some 10^4 rendezvous

// How a launch waits: the limit of each wait, and for tests, so that waits run out without any fault,
// arrivals to wait for beyond the grid's own (0) and the rendezvous, counted from 1, at which the last
// block takes its wait as run out although all have arrived (0: none).
struct GridWait {
    unsigned long long limit_ns;
    unsigned extra;
    unsigned give_up;
};

// LBGPU_TEST_GRID_WAIT (tests only): 1: every wait runs out, after 50 ms; k > 1: the last block gives up at
// the rendezvous k - 1.
inline GridWait grid_wait()
{
    const char *env = std::getenv("LBGPU_TEST_GRID_WAIT");
    const int test = env ? std::atoi(env) : 0;
    GridWait w;
    w.limit_ns = test > 0 ? 50000000ull : 2000000000ull;
    w.extra = test == 1 ? 1u : 0u;
    w.give_up = test > 1 ? (unsigned)(test - 1) : 0u;
    return w;
}

__device__ __forceinline__ unsigned ld_acquire_gpu(const unsigned *p)
{
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// The grid's rendezvous number `round` (0, 1, ...; all blocks count alike, and the structure is zero
// before the launch).  VALUES: value / bits become the maximum / OR over every thread of the grid.
// False, in every thread of the block, when the wait ran out.  Data that other blocks wrote before it
// must be read from L2 (__ldcg).
template <bool VALUES>
__device__ __forceinline__ bool grid_barrier(GridSync *g, unsigned round, const GridWait &wait,
                                             unsigned long long &value, unsigned &bits)
{
    __shared__ unsigned long long sval[32], rval;
    __shared__ unsigned sbit[32], rbit;
    __shared__ int ok;
    if constexpr (VALUES) {
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long v = __shfl_xor_sync(0xffffffffu, value, o);
            value = v > value ? v : value;
        }
        bits = __reduce_or_sync(0xffffffffu, bits);
        if (lane == 0) {
            sval[wid] = value;
            sbit[wid] = bits;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        GridSync::Slot *s = &g->slot[round % 3u];
        if constexpr (VALUES) {
            for (unsigned w = 1; w < (blockDim.x >> 5); ++w) {
                value = sval[w] > value ? sval[w] : value;
                bits |= sbit[w];
            }
            if (value) atomicMax(&s->value, value);
            if (bits) atomicOr(&s->bits, bits);
        }
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&g->arrived) : "memory");
        const unsigned target = (round + 1u) * (gridDim.x + wait.extra);
        bool done = false;
        unsigned long long t0 = 0;
        for (unsigned it = 0; it < (1u << 28); ++it) {
            const unsigned n = ld_acquire_gpu(&g->arrived);
            if (n >= target) {
                done = n < GRID_FAILED;
                break;
            }
            if ((it & 255u) == 255u) {
                const unsigned long long t = global_ns();
                if (t0 == 0) t0 = t;
                else if (t - t0 > wait.limit_ns) {
                    atomicOr(&g->arrived, GRID_FAILED);
                    break;
                }
            }
        }
        if constexpr (VALUES) {
            rval = __ldcg(&s->value);
            rbit = __ldcg(&s->bits);
        }
        if (blockIdx.x == 0 && done) {
            GridSync::Slot *z = &g->slot[(round + 2u) % 3u];
            z->value = 0;
            z->bits = 0;
        }
        ok = done;
    }
    __syncthreads();
    if constexpr (VALUES) {
        value = rval;
        bits = rbit;
    }
    if (wait.give_up == round + 1u && blockIdx.x == gridDim.x - 1u) return false;
    return ok != 0;
}

}  // namespace lbg
