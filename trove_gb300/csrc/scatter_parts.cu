// Scatters onto large destinations.
//
// A row that does not fill whole 32-byte sectors is a partial-sector write.
// Scattered over a destination that L2 does not hold yet, each one makes L2
// fill the rest of its sector from DRAM at the rate of random accesses, and
// over one larger than L2 the sector leaves before its other rows arrive and
// is filled and written again.  Two remedies:
//  - the destination (or the part at hand) is fetched into L2 first, in
//    address order at the full DRAM rate, so that the writes find their
//    sectors (2^21 rows of 24 bytes: 52 -> 25 us plus the fetch);
//  - a destination larger than L2 is written in parts that fit, one pass each.
#include <cuda_runtime.h>

#include "fetch.cuh"
#include "ops.h"
#include "rules.h"

namespace trv {
namespace {

// Loads of what a kernel reads once: 64-byte fetches, first to leave L2.
__device__ __forceinline__ unsigned long long l2_evict_first_policy() {
    unsigned long long pol;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}
__device__ __forceinline__ uint4 ld_once(const uint4* p, unsigned long long pol) {
    uint4 v;
    asm volatile("ld.global.nc.L2::cache_hint.L2::64B.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p), "l"(pol));
    return v;
}
__device__ __forceinline__ uint2 ld_once(const uint2* p, unsigned long long pol) {
    uint2 v;
    asm volatile("ld.global.nc.L2::cache_hint.L2::64B.v2.u32 {%0, %1}, [%2], %3;"
                 : "=r"(v.x), "=r"(v.y)
                 : "l"(p), "l"(pol));
    return v;
}
__device__ __forceinline__ unsigned ld_once(const unsigned* p, unsigned long long pol) {
    unsigned v;
    asm volatile("ld.global.nc.L2::cache_hint.L2::64B.u32 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(pol));
    return v;
}
__device__ __forceinline__ int ld_once(const int* p, unsigned long long pol) {
    return int(ld_once(reinterpret_cast<const unsigned*>(p), pol));
}

// Ahead of a one-pass scatter: what the sampled indices span of the destination.
__global__ void __launch_bounds__(256)
fetch_destination_kernel(const unsigned char* dst, unsigned bound, const int* __restrict__ idx, long long n,
                         int row_bytes, unsigned long long plain) {
    const IndexSample sample(idx, n, int(threadIdx.x & 31u));
    if (sample.local(row_bytes)) return;
    unsigned first, rows;
    sample.span(bound, first, rows);
    if (rows * (unsigned long long)unsigned(row_bytes) <= plain) return;  // L2 holds them as it is
    const unsigned long long p = reinterpret_cast<unsigned long long>(dst) + first * (unsigned long long)unsigned(row_bytes);
    fetch_part(p, p + rows * (unsigned long long)unsigned(row_bytes), blockIdx.x, gridDim.x);
}

// Scatter in passes: pass p moves the rows whose index lies in the p-th part
// of the destination.  One launch, the passes' blocks in order, so a pass
// starts as the one before it drains; between two passes come the blocks that
// fetch the next part.
//
// A warp reads the indices of a slab of kSlab structs (all loads in flight at
// once), compacts the ones of its pass into a list in shared memory, and moves
// the listed structs with every lane busy: word q = l + 32k of the list's
// words is word q % m of struct list[q / m].  A pass so reads the index array
// and its own share of the source, not the whole of both, and both are first
// to leave L2, which keeps the part being written.
//
// Bound by DRAM: 2^24 random rows of 12 bytes in four passes move about 1.35 GB
// in 230 us (one pass of the row-form kernel 544 us, three passes of it over
// 64 MiB parts 380 us); of 24 bytes 406 us (one pass 717), of 48 bytes 680 us
// (1143), of 60 bytes 888 us (1509).
constexpr int kPassWarps = 8;

struct PassPlan {
    unsigned bound;          // rows of the destination
    unsigned rows_per_pass;
    unsigned passes;
    unsigned body;           // blocks that move a pass's structs
    unsigned fetch;          // blocks that fetch a part
};

// Every row in one pass, where the sample says that the parts have nothing to
// give.  The rows are read in their own order, whatever their indices.  A launch
// with its most blocks to a part works in slabs with as many blocks as one part
// has; the others take about 1 ns each to leave, so for rows of 8- and 16-byte
// words, which are bound by DRAM, every passes-th block works and the others leave
// meanwhile (2^24 sorted rows of 24 / 40 / 48 bytes 143 / 229 / 261 us, 148 / 239 /
// 278 where they leave at the end; of 36 bytes, bound by instructions, 278 and 264
// where the first blocks work).  On fewer rows, slabs would come to hardly more
// than a wave of blocks, and all blocks take kOrderRows rows to a warp (200 MiB of
// sorted rows of 80 bytes 83 us in slabs, 68 so, 66 plain).
constexpr int kOrderRows = 128, kOrderWideRows = 64;
constexpr int kBodyBlocks = 2048;  // blocks that move a part's structs, at most (launch_passes)

template <typename V, int G>
__device__ __forceinline__ void scatter_in_order(const V* __restrict__ src, const int* __restrict__ idx,
                                                 V* __restrict__ dst, long long n, int m, const PassPlan& plan, int* to,
                                                 unsigned long long pol, int lane, int warp) {
    const bool slabs = plan.body == kBodyBlocks;
    const unsigned each = slabs && sizeof(V) > 4 ? plan.passes : 1u;
    const unsigned c = blockIdx.x / each, blocks = slabs ? plan.body : gridDim.x;
    if (c * each != blockIdx.x || c >= blocks) return;
    const int rows = slabs ? kSlab : m * int(sizeof(V)) > 64 ? kOrderWideRows : kOrderRows;
    const int step_j = 32 / m, step_r = 32 % m;
    for (long long base = ((long long)c * kPassWarps + warp) * rows; base < n;
         base += (long long)blocks * kPassWarps * rows) {
        const int rem = n - base < rows ? int(n - base) : rows;
        __syncwarp();  // the previous rows' list has been read
        for (int t0 = lane; t0 < rem; t0 += 128) {
            int v[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) v[t] = t0 + 32 * t < rem ? ld_once(idx + base + t0 + 32 * t, pol) : -1;
#pragma unroll
            for (int t = 0; t < 4; ++t)
                if (t0 + 32 * t < rem) to[t0 + 32 * t] = unsigned(v[t]) < plan.bound ? v[t] : -1;
        }
        __syncwarp();
        const V* from = src + base * m;
        const int words = rem * m;
        int j = lane / m, r = lane % m;
        for (int q = lane; q < words; q += 32 * G) {
            V val[G];
#pragma unroll
            for (int g = 0; g < G; ++g)
                if (q + 32 * g < words) val[g] = ld_once(from + q + 32 * g, pol);
#pragma unroll
            for (int g = 0; g < G; ++g) {
                if (q + 32 * g < words && to[j] >= 0) dst[(long long)to[j] * m + r] = val[g];
                j += step_j;
                r += step_r;
                if (r >= m) {
                    r -= m;
                    ++j;
                }
            }
        }
    }
}

template <typename V, int G>
__global__ void __launch_bounds__(32 * kPassWarps)
scatter_passes_kernel(const V* __restrict__ src, const int* __restrict__ idx, V* __restrict__ dst, long long n, int m,
                      PassPlan plan) {
    __shared__ int s_to[kPassWarps][kSlab];
    __shared__ unsigned short s_at[kPassWarps][kSlab];
    const int lane = int(threadIdx.x & 31u), warp = int(threadIdx.x >> 5);
    const unsigned long long row = (unsigned long long)m * sizeof(V);
    const IndexSample sample(idx, n, lane);
    unsigned first, spanned;
    sample.span(plan.bound, first, spanned);
    int* to = s_to[warp];
    const unsigned long long pol = l2_evict_first_policy();
    const int step_j = 32 / m, step_r = 32 % m;
    unsigned lo = 0, rows = plan.bound, c;
    if (sample.mostly_skipped(plan.bound)) {
        // One pass over everything, by lists of the valid rows: the source of the others
        // is not read (2^22 rows of 80 bytes, nine in ten skipped: 58 us, 84 where it is).
        const unsigned each = sizeof(V) > 4 ? plan.passes : 1u;
        c = blockIdx.x / each;
        if (c * each != blockIdx.x || c >= plan.body) return;
    } else if (sample.local(int(row)) || spanned * row <= kPlainScatterBytes) {
        scatter_in_order<V, G>(src, idx, dst, n, m, plan, to, pol, lane, warp);
        return;
    } else {
        const unsigned pass = blockIdx.x / (plan.fetch + plan.body);
        c = blockIdx.x - pass * (plan.fetch + plan.body);
        unsigned passes = plan.passes, step = plan.rows_per_pass;
        if (spanned < plan.bound / 4 * 3) {
            // All of the sample within three quarters of the destination (of 64 rows at
            // random, one time in a million): as many parts as those rows need, the
            // outer ones with what lies outside.
            passes = (spanned + plan.rows_per_pass - 1) / plan.rows_per_pass;
            if (pass >= passes) return;
            step = (spanned + passes - 1) / passes;
        } else {
            first = 0;
        }
        lo = first + pass * step;
        unsigned end = plan.bound - lo < step ? plan.bound : lo + step;
        if (c < plan.fetch) {
            const unsigned long long p = reinterpret_cast<unsigned long long>(dst);
            fetch_part(p + lo * row, p + end * row, c, plan.fetch);
            return;
        }
        if (pass == 0) lo = 0;
        if (pass == passes - 1) end = plan.bound;
        rows = end - lo;
        c -= plan.fetch;
    }
    unsigned short* at = s_at[warp];
    for (long long base = ((long long)c * kPassWarps + warp) * kSlab; base < n;
         base += (long long)plan.body * kPassWarps * kSlab) {
        const int rem = n - base < kSlab ? int(n - base) : kSlab;
        int v[kSlabRounds];
#pragma unroll
        for (int t = 0; t < kSlabRounds; ++t) v[t] = t * 32 + lane < rem ? ld_once(idx + base + t * 32 + lane, pol) : -1;
        int cnt = 0;
        __syncwarp();  // the previous slab's list has been read
#pragma unroll
        for (int t = 0; t < kSlabRounds; ++t) {
            const bool mine = unsigned(v[t]) - lo < rows;  // a negative index is 2^31 or more, lo + rows at most 2^31
            const unsigned b = __ballot_sync(0xFFFFFFFFu, mine);
            if (mine) {
                const int k = cnt + __popc(b & ((1u << lane) - 1u));
                to[k] = v[t];
                at[k] = (unsigned short)(t * 32 + lane);
            }
            cnt += __popc(b);
        }
        __syncwarp();
        const V* from = src + base * m;
        const int words = cnt * m;
        int j = lane / m, r = lane % m;
        for (int q = lane; q < words; q += 32 * G) {
            V val[G];
            V* out[G];
#pragma unroll
            for (int g = 0; g < G; ++g) {
                out[g] = nullptr;
                if (q + 32 * g < words) {
                    val[g] = ld_once(from + unsigned(at[j]) * unsigned(m) + r, pol);
                    out[g] = dst + (long long)to[j] * m + r;
                }
                j += step_j;
                r += step_r;
                if (r >= m) {
                    r -= m;
                    ++j;
                }
            }
#pragma unroll
            for (int g = 0; g < G; ++g)
                if (out[g]) *out[g] = val[g];
        }
    }
}

constexpr int kFetchBlocks = 64;
// kBodyBlocks: few enough to leave quickly where the indices are local, enough that
// two passes overlap only briefly.  2^24 / 3 * 2^24 random rows of 24 bytes: 458 /
// 2073 us at 608 (one resident wave), 406 / 1840 at 2048, 395 / 1793 at 4096; 2^24
// sorted rows of 48 bytes, the others leaving at the end: 264 / 277 / 331 us.

template <typename V, int G>
void launch_passes(const IndexArgs& a, int m, int passes, cudaStream_t st) {
    const unsigned bound = a.bound > 0x80000000ll ? 0x80000000u : unsigned(a.bound);
    PassPlan p;
    p.bound = bound;
    p.rows_per_pass = unsigned((bound + (long long)passes - 1) / passes);
    p.passes = (bound + p.rows_per_pass - 1) / p.rows_per_pass;
    const long long slabs = (a.n + kSlab * kPassWarps - 1) / (kSlab * kPassWarps);
    p.body = unsigned(slabs < kBodyBlocks ? slabs : kBodyBlocks);
    p.fetch = kFetchBlocks;
    scatter_passes_kernel<V, G><<<p.passes * (p.fetch + p.body), 32 * kPassWarps, 0, st>>>(
        static_cast<const V*>(a.src), a.idx, static_cast<V*>(a.dst), a.n, m, p);
}
}  // namespace

void launch_fetch_destination(const IndexArgs& a, int row_bytes, uint64_t plain, cudaStream_t st) {
    fetch_destination_kernel<<<kFetchBlocks, 256, 0, st>>>(static_cast<const unsigned char*>(a.dst), unsigned(a.bound > 0x80000000ll ? 0x80000000ll : a.bound),
                                                           a.idx, a.n, row_bytes, plain);
}

void launch_scatter_passes(int word_bytes, const IndexArgs& a, int m, int passes, cudaStream_t st) {
    if (word_bytes == 16)
        launch_passes<uint4, 4>(a, m, passes, st);
    else if (word_bytes == 8)
        launch_passes<uint2, 8>(a, m, passes, st);
    else
        launch_passes<unsigned, 8>(a, m, passes, st);
}

}  // namespace trv
