// Barrier of a kernel whose blocks wait on one another: all blocks of a
// cooperative launch (one counter in global memory), or the blocks of one
// thread-block cluster (the hardware's cluster barrier). Both order global
// memory: what a block wrote before it arrived is seen, through L2 (__ldcg),
// by every block after it waited. arrive() is a barrier of the block in both
// forms: a warp goes on behind it only when no other of the block's still reads
// or writes shared memory before it. (The cluster's own arrive does not wait, so
// a warp past it could write what another was about to read.)
#pragma once

#include <cuda_runtime.h>

namespace regot {

// Polls `count` until it has reached `target` (the difference counts as signed), at
// most kMaxPolls times; `polls` and *err are looked at every 1024. With `polls` as
// the loop's bound, or with a bound of 2^31, every barrier took some 140 clocks
// longer: FP64 BCD 1 to 2 %, mixed Newton at 4096 x 4096 9.69 -> 9.79 ms.
constexpr unsigned kPollStep = 1024, kMaxPolls = 1u << 22;
__device__ __forceinline__ bool poll_count(const unsigned* count, unsigned target, unsigned polls,
                                           const int* err) {
    for (unsigned s = 0; s < kMaxPolls; ++s) {
        unsigned c;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(count) : "memory");
        if ((int)(c - target) >= 0) return true;
        if ((s & (kPollStep - 1)) == kPollStep - 1 && (*(const volatile int*)err || s >= polls))
            return false;
    }
    return false;
}
// What the first generation starts from: with a limit of 0 a count that none reaches,
// so that the first wait gives up after its first 1024 polls.
__device__ __forceinline__ unsigned first_target(unsigned polls) { return polls ? 0u : 1u << 30; }

template <bool CLUSTER>
struct GridBarrier;

// count starts at 0 and only grows; generation g is complete at g * gridDim.x
// arrivals. A wait gives up at the first 1024 polls (each a round trip to L2, about
// a microsecond) that reach `polls` (grid_polls()) and sets *err. Its block leaves,
// so no later generation completes, and the waits for one end within 1024 polls of
// *err; a wait whose generation was complete still returns true. The host looks at
// *err after every launch.
template <>
struct GridBarrier<false> {
    unsigned* count;
    int* err;
    unsigned target, polls;
    int* s_ok;  // one int of shared memory

    __device__ GridBarrier(unsigned* c, int* e, unsigned p, int* s)
        : count(c), err(e), target(first_target(p)), polls(p), s_ok(s) {}
    __device__ void arrive() {
        __syncthreads();
        target += gridDim.x;
        if (threadIdx.x == 0)
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
    }
    __device__ bool wait() {
        if (threadIdx.x == 0) {
            const bool ok = poll_count(count, target, polls, err);
            if (!ok) atomicOr(err, 1);
            *s_ok = ok;
        }
        __syncthreads();
        return *s_ok != 0;
    }
};

template <>
struct GridBarrier<true> {
    __device__ GridBarrier(unsigned*, int*, unsigned, int*) {}
    __device__ void arrive() {
        __syncthreads();
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    }
    __device__ bool wait() {
        __syncwarp();
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        return true;
    }
};

}  // namespace regot
