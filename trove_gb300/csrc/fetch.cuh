// Fetching a scatter's destination into L2 ahead of its writes, and the sample of
// the indices that tells when there is nothing to gain (scatter_parts.cu says
// why; the batched kernel does the same ahead of a scatter task's tiles).
#pragma once

#include <cuda_runtime.h>

#include "rules.h"

namespace trv {

// Whether indices mostly step from one row to the next (sorted, runs): then
// the writes of neighbouring rows meet in L2 by themselves, and neither remedy
// is needed.  Every warp takes the same 32 pairs of the index array, so every
// warp of a launch comes to the same answer.
struct IndexSample {
    int a, b;
    __device__ __forceinline__ IndexSample(const int* __restrict__ idx, long long n, int lane) {
        const long long p = sample_position(lane, n);  // n >= 2
        a = __ldg(idx + p);
        b = __ldg(idx + p + 1);
    }
    __device__ __forceinline__ bool local(int row_bytes) const {
        return __popc(__ballot_sync(0xFFFFFFFFu, sample_near(a, b, row_bytes))) >= near_pairs(row_bytes);
    }
    // Whether neighbouring lanes' rows mostly lie in the same sectors, or hardly any
    // are valid: then a thread per row does best for narrow rows.
    __device__ __forceinline__ bool rows_adjoin(int row_bytes) const {
        const long long d = (long long)b - a;
        return __popc(__ballot_sync(0xFFFFFFFFu, (d < 0 ? -d : d) * row_bytes <= 64)) >= 20;
    }
    // Whether half of the sampled indices or fewer lie below `bound`.
    __device__ __forceinline__ bool mostly_skipped(unsigned bound) const {
        return __popc(__ballot_sync(0xFFFFFFFFu, unsigned(a) < bound)) +
                   __popc(__ballot_sync(0xFFFFFFFFu, unsigned(b) < bound)) <= kSamples;
    }
    // The rows [first, first + rows) that the sampled indices below `bound` lie in.
    __device__ __forceinline__ void span(unsigned bound, unsigned& first, unsigned& rows) const {
        const bool va = unsigned(a) < bound, vb = unsigned(b) < bound;
        const unsigned lo = __reduce_min_sync(0xFFFFFFFFu, min(va ? unsigned(a) : bound, vb ? unsigned(b) : bound));
        const unsigned hi = __reduce_max_sync(0xFFFFFFFFu, max(va ? unsigned(a) + 1 : 0u, vb ? unsigned(b) + 1 : 0u));
        first = lo;
        rows = hi > lo ? hi - lo : 0u;
    }
};

// Fetches [p0, p1) into L2: block c of `blocks`, 4 KiB an instruction.
__device__ __forceinline__ void fetch_part(unsigned long long p0, unsigned long long p1, unsigned c, unsigned blocks) {
    p0 = (p0 + 15) & ~15ull;
    p1 &= ~15ull;
    const unsigned long long step = (unsigned long long)blocks * blockDim.x * 4096;
    for (unsigned long long p = p0 + ((unsigned long long)c * blockDim.x + threadIdx.x) * 4096; p < p1; p += step) {
        const unsigned bytes = p1 - p < 4096 ? unsigned(p1 - p) : 4096u;
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
    }
}

}  // namespace trv
