// uns_sweep.cuh -- the pairing of warps that runs the LU-SGS sweeps.
//
// A sweep is a chain of items, each a few dozen dependent FP64 operations on
// values that other warps have just published.  One warp doing both (loads
// and polls in flight during its arithmetic) takes about twice the time of
// the arithmetic: the results of loads and of FP64 instructions share the
// warp's few scoreboards, so an addition's result waits for an outstanding
// load.  So each sweep warp has a feeder warp beside it (same SM
// sub-partition): the feeder walks the same list of items ahead of it, loads
// an item's inputs, polls its neighbours' records and puts everything into a
// small ring in shared memory, laid out per lane; the sweep warp takes an
// entry from the ring, does the arithmetic and publishes.  Its only global
// accesses are the stores.
//
// The ring's entries are handed over through mbarriers: `full` (the feeder's
// lane 0 arrives once its warp has written the entry) and `empty` (the sweep
// warp's lane 0 arrives once its warp has read it).  Every wait is bounded,
// and a warp that gives up raises `abort`, on which its partner returns.
#pragma once
#include "uns_common.cuh"

namespace uns {

constexpr int kSweepPairs = 4;                      // sweep warps per block: one per SM sub-partition
constexpr int kSweepBlock = 64 * kSweepPairs;       // sweep warps, then their feeders
constexpr int kSweepStages = 3;

// One pair's ring: NF 8-byte fields per lane and stage, and the item.
template <int NF>
struct __align__(16) SweepRing {
    unsigned long long full[kSweepStages], empty[kSweepStages];
    double f[kSweepStages][NF][32];
    int4 item[kSweepStages];
    int abort;
    int pad[3];
};

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

template <int NF>
__device__ __forceinline__ void ring_init(SweepRing<NF>& R) {
    for (int s = 0; s < kSweepStages; ++s) {
        asm volatile("mbarrier.init.shared.b64 [%0], 1;" : : "r"(smem_addr(&R.full[s])) : "memory");
        asm volatile("mbarrier.init.shared.b64 [%0], 1;" : : "r"(smem_addr(&R.empty[s])) : "memory");
    }
    R.abort = 0;
}

__device__ __forceinline__ void mbar_arrive(unsigned long long* b) {
    asm volatile("mbarrier.arrive.release.cta.shared.b64 _, [%0];" : : "r"(smem_addr(b)) : "memory");
}

// Waits (all lanes) until the phase of the given parity has completed: false
// once the partner has aborted or `limit` cycles have passed.
__device__ __forceinline__ bool mbar_wait(unsigned long long* b, unsigned parity, const int* abort, long long limit) {
    const unsigned a = smem_addr(b);
    long long t0 = 0;
    for (int spins = 0;; ++spins) {
        unsigned ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cta.shared.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok) : "r"(a), "r"(parity) : "memory");
        if (ok) return true;
        if (spins == 0) t0 = clock64();
        if ((spins & 15) == 15 && (*(const volatile int*)abort || clock64() - t0 > limit)) return false;
    }
}

// Position in the ring: stage and the parity of its next phase.
struct RingPos {
    int stage = 0;
    unsigned phase = 0;
    __device__ __forceinline__ void next() {
        if (++stage == kSweepStages) { stage = 0; phase ^= 1; }
    }
};

// The sweep warp's wait for an entry outlasts the feeder's own for a record.
__device__ __forceinline__ long long ring_limit(long long wait_cycles) { return 4 * wait_cycles + 100000000LL; }

}  // namespace uns
