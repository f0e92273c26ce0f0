// Barriers of the persistent kernels (the coloured pair solve and the exact-cone NCP sweep).  The
// grid's: one arrival counter that only grows within a launch.
//
// Barrier k of a launch (k = 1, 2, ...): every thread of the CTA finishes its writes
// (__syncthreads), then thread 0 adds 1 to the counter with a release reduction at GPU scope
// (red.release: fire-and-forget, no value comes back, so the arrival costs no round trip) and
// polls the counter with acquire loads until it reaches k x gridDim, then releases the CTA with
// __syncthreads (relaxed polls and a fence.acq_rel.gpu after the last cost one more trip to L2
// a barrier).  Measured on B200 (no work between barriers, one 256-thread CTA per
// SM): 1.31 us per barrier over 148 CTAs, 1.25 us over 74, against 2.20 us for an atomic
// arrival count with a separate generation word (arrivals that return a value, then a second
// round trip for the release) and 2.58 us for one flag per CTA polled by a warp; a
// thread-block cluster's hardware barrier takes 0.22 us over 16 CTAs.
//
// The counter restarts from zero every launch: the host clears it (cudaMemsetAsync, a graph
// node inside a captured step) before each cooperative launch, so no count survives a launch,
// a checkpoint load or a change of grid size.
//
// Every wait is bounded: after timeout_ns of %globaltimer the waiting thread sets err_bit in
// *err, the CTA leaves the barrier with false, and the kernel returns (its other CTAs give up at
// their own next wait).  The host reads the bit and raises; the context stays usable.
#pragma once

#include <cstdint>

namespace b2c {

constexpr int kBarrierWords = 32;      // the counter, alone on its 128-byte line
constexpr int kBarrierMaxCTAs = 4096;  // a cooperative grid is capped at this (counts stay < 2^31)

__device__ __forceinline__ unsigned long long barrier_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ unsigned int counter_load_acquire(const unsigned int *p)
{
    unsigned int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Arrival at a thread-block cluster's hardware barrier, for all the writes of the CTA; every thread
// of the CTA calls it, and barrier.cluster.wait.acquire after it.  A release waits until the writes
// before it have reached L2, and a release by every warp takes each of them through that on its
// own; here the CTA's writes are ordered before one warp's release by __syncthreads, and the other
// warps arrive relaxed.  Measured on a B200 (cycles a phase over 16 CTAs, a store to and a load from
// L2 by every thread between barriers): 2 023 -> 1 706 with 256 threads, 2 218 -> 1 741 with 384,
// 2 322 -> 1 795 with 640; without stores 416 -> 470, 471 -> 485, 516 -> 523.  The coloured pair
// solve arrives warp by warp all the same: its warps are done at different times, and waiting for
// the slowest before any of them loads its next task cost a pile of 3 000 boxes 1 909 -> 1 950 us.
__device__ __forceinline__ void cluster_arrive()
{
    __syncthreads();
    if (threadIdx.x < 32) asm volatile("barrier.cluster.arrive.release;\n" ::: "memory");
    else asm volatile("barrier.cluster.arrive.relaxed;\n" ::: "memory");
}

// arrival at barrier `epoch` (1, 2, ... within a launch); every thread of the CTA calls it
__device__ __forceinline__ void grid_arrive(unsigned int *counter)
{
    __syncthreads();
    if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;\n" ::"l"(counter) : "memory");
}

// wait until every CTA has arrived at barrier `epoch`; every thread of the CTA calls it.
// Returns false when the wait ran out (or another CTA's had, as *err tells), after setting err_bit.
__device__ __forceinline__ bool grid_wait(const unsigned int *counter, unsigned int epoch, long long timeout_ns,
                                          int *err, int err_bit)
{
    __shared__ int s_grid_ok;
    if (threadIdx.x == 0) {
        const unsigned int target = epoch * gridDim.x;
        const unsigned long long t0 = barrier_ns();
        int ok = 1;
        while ((int)(counter_load_acquire(counter) - target) < 0) {
            if (barrier_ns() - t0 > (unsigned long long)timeout_ns) {
                atomicOr(err, err_bit);
                ok = 0;
                break;
            }
        }
        s_grid_ok = ok && !(*(volatile int *)err & err_bit);
    }
    __syncthreads();
    return s_grid_ok != 0;
}

}  // namespace b2c
