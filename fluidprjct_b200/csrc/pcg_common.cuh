// pcg_common.cuh -- device helpers shared by the persistent PCG kernels:
// a bounded grid barrier for cooperative launches and deterministic FP64
// block / grid reductions.
#pragma once

#include "kernels.hpp"

namespace fp {
namespace {

// note_clock of a persistent solver, as a call: inlined, it changed the code of
// the iterations so that they took 1 % longer.
__device__ __noinline__ void note_solve(unsigned long long* at) { note_clock(at); }

// ---------------------------------------------------------------- grid barrier
// Grid barrier for a cooperative launch on one 32-bit word: every block adds
// 1 except block 0, which adds 2^31 - (nblocks - 1), so the word's top bit
// flips exactly when the last block arrives and no reset is needed between
// barriers.  The block whose arrival flips the bit knows it from the
// atomic's result and does not poll.  The wait is bounded: after bar->limit
// polls (kDefaultWaitPolls = 2^27 unless the solver's owner set another
// limit) the block records DEV_TIMEOUT and leaves; callers check the status
// after every barrier and return, so no block waits forever.  The arrival is
// an acquire-release atomic and the poll an acquire load (the pattern of a
// release-acquire grid barrier), so plain loads after it see every write made
// before it by any block.
__device__ __forceinline__ bool grid_barrier(GridBar* bar, unsigned nblocks, int* status) {
    __shared__ int s_ok;
    __syncthreads();
    // A one-block launch (a small grid) has no other block to wait for: the
    // block barrier alone orders its threads' global writes and reads.
    if (nblocks == 1u) return true;
    if (threadIdx.x == 0) {
        // The status and limit loads are issued before the arrival so that
        // their latency overlaps the atomic; a timeout recorded by another
        // block is seen at this or the next barrier, and every wait below is
        // bounded.
        const int st0 = *(volatile int*)status;
        const unsigned limit = *(volatile unsigned*)&bar->limit;  // at least 1
        const unsigned inc = blockIdx.x == 0 ? 0x80000000u - (nblocks - 1u) : 1u;
        // arrival with release semantics: after the block barrier above it
        // publishes every write this block made before the grid barrier
        unsigned old;
        // acquire as well: the last block to arrive reads the value the
        // other arrivals' release RMWs wrote, so it has their writes and need
        // not poll.  That takes one L2 round trip off the barrier's critical
        // path: 0.974 -> 0.964 ms per warm-started MG solve at 128^3.
        asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], %2;\n"
                     : "=r"(old)
                     : "l"(&bar->count), "r"(inc)
                     : "memory");
        const bool last = ((old ^ (old + inc)) & 0x80000000u) != 0u;
        bool ok = st0 == DEV_OK;
        unsigned polls = 0;
        for (; !last;) {
            // acquire load: writes published by the other blocks' arrivals are
            // visible to this block once the top bit has flipped
            unsigned cur;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(cur) : "l"(&bar->count) : "memory");
            if (((old ^ cur) & 0x80000000u) != 0u) break;
            if (++polls >= limit) {
                atomicExch(status, DEV_TIMEOUT);
                if (bar->gave_up) *bar->gave_up = clock_ns();
                ok = false;
                break;
            }
        }
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// Grid-wide sums of N doubles per thread, the same bits in every thread of
// every block, around one grid barrier: block partials to part[N][nb] (two
// buffers that alternate from call to call suffice), the barrier, then mid()
// -- loads that wait on the barrier but not on the sums, so that their round
// trip overlaps the partials' -- and the total, one warp per sum with all its
// loads issued together.  Returns false if the barrier gave up.  Fixed order
// throughout.  (One block barrier and half of the shuffle steps fewer per
// reduction than sums over the whole block before the barrier and a two-level
// tree over the whole block after it.)
template <int N, class Mid>
__device__ __forceinline__ bool grid_reduce(double (&v)[N], double* part, GridBar* bar, int nb, int* status, Mid mid) {
    __shared__ double sh[N][32];
    __shared__ double res[N];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = int(blockDim.x >> 5);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < N; ++k) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < N; ++k) sh[k][wid] = v[k];
    __syncthreads();
    double x = 0.0;
    if (wid < N) {
        x = lane < nw ? sh[wid][lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if (lane == 0) {
            if (nb == 1) res[wid] = x;
            else part[wid * nb + int(blockIdx.x)] = x;
        }
    }
    if (!grid_barrier(bar, unsigned(nb), status)) return false;
    mid();
    if (nb > 1 && wid < N) {
        // written by other CTAs in this launch: read through L2
        constexpr int B = 5;  // 160 CTAs in one batch of loads
        x = 0.0;
        for (int t0 = lane; t0 < nb; t0 += 32 * B) {
            double y[B];
#pragma unroll
            for (int b = 0; b < B; ++b) y[b] = t0 + 32 * b < nb ? __ldcg(part + wid * nb + t0 + 32 * b) : 0.0;
#pragma unroll
            for (int b = 0; b < B; ++b) x += y[b];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if (lane == 0) res[wid] = x;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = res[k];
    return true;
}
template <int N>
__device__ __forceinline__ bool grid_reduce(double (&v)[N], double* part, GridBar* bar, int nb, int* status) {
    return grid_reduce<N>(v, part, bar, nb, status, [] {});
}

}  // namespace
}  // namespace fp
