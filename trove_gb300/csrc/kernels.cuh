// Kernel templates of the C ABI.  Every struct-typed kernel moves
// trove::array<unsigned, S> (S = width / 4) through this library's device API
// (include/trove), so the library's host entry points run exactly the code a
// user kernel written against that API would run.
//
// Work decomposition: a warp owns chunks of 32*U consecutive structs; within
// a chunk lane l owns structs base + u*32 + l (u < U).  All U loads of a
// chunk are issued before its U stores, which keeps U structs per lane in
// flight (the memory-level parallelism HBM needs: ~5 MB in flight chip-wide
// at 6.8 TB/s).  By default the grid has one chunk per warp and the kernels
// have no loop (measured on GB300 a few percent faster than a persistent
// grid-stride grid, and free of the loop's registers); grid-stride forms
// serve a grid chosen through trv_launch.grid_blocks.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <trove/aos.h>
#include <trove/block.h>
#include <trove/ptr.h>

#include "ops.h"

namespace trv {

template <int S>
using aos = trove::array<unsigned, S>;

enum Api { API_WARP = 0, API_BLOCK = 1, API_DIRECT = 2 };

// Whether the struct's first word w has w % d == d - 1.  That is w >= d - 1 and d
// divides w - (d - 1); and d = q * 2^k (q odd) divides x when x times q's inverse
// modulo 2^32, rotated right by k, is at most (2^32 - 1) / d (Granlund and
// Montgomery, "Division by Invariant Integers using Multiplication", section 9).
// Five instructions where the remainder of a run-time d takes about twenty, of the
// 84 that 32 structs of 12 bytes cost: 1 GiB of 4 bytes 308.5 -> 305.2 us, of 12 bytes
// 318.7 -> 306.4, of 20 bytes 313 -> 306.5, of 32 bytes 303.7 -> 301.8.  It pays for
// lanes of few words, which are bound by instructions (exit_multiply).  Lanes of more
// words wait for DRAM either way, and the multiplication's operands cost them
// registers (12 bytes, 8 structs to a lane, 42 and 48: 314 -> 325 us; 28 bytes, 2 to a
// lane, 32 and 40: 301 -> 308; 36 bytes 299.6 -> 300.5): they keep the remainder.
template <bool MULTIPLY, int S>
__device__ __forceinline__ bool exits(const aos<S>& v, const ExitTest& t) {
    const unsigned w = unsigned(v.head);
    if constexpr (!MULTIPLY) return w % t.modulus == t.modulus - 1u;
    const unsigned x = (w - t.low) * t.inverse;
    return w >= t.low && __funnelshift_r(x, x, t.rotate) <= t.most;
}

// Load/store of struct i when the caller's warp is converged and its lanes
// address consecutive structs.
template <int S, int API>
__device__ __forceinline__ aos<S> load_conv(const aos<S>* src, long long i) {
    if constexpr (API == API_WARP)
        return trove::load_warp_contiguous(src + i);
    else if constexpr (API == API_BLOCK)
        return trove::load_array_warp_contiguous<S>(reinterpret_cast<const unsigned*>(src), i);
    else
        return src[i];
}

template <int S, int API>
__device__ __forceinline__ void store_conv(aos<S>* dst, long long i, const aos<S>& v) {
    if constexpr (API == API_WARP)
        trove::store_warp_contiguous(v, dst + i);
    else if constexpr (API == API_BLOCK)
        trove::store_array_warp_contiguous(reinterpret_cast<unsigned*>(dst), i, v);
    else
        dst[i] = v;
}

// The same when the warp is not converged.
template <int S, int API>
__device__ __forceinline__ aos<S> load_div(const aos<S>* src, long long i) {
    if constexpr (API == API_BLOCK)
        return trove::load_array<S>(reinterpret_cast<const unsigned*>(src), i);
    else if constexpr (API == API_WARP)
        return trove::detail::divergent_load(src + i);
    else
        return src[i];
}

template <int S, int API>
__device__ __forceinline__ void store_div(aos<S>* dst, long long i, const aos<S>& v) {
    if constexpr (API == API_BLOCK)
        trove::store_array(reinterpret_cast<unsigned*>(dst), i, v);
    else if constexpr (API == API_WARP)
        trove::detail::divergent_store(v, dst + i);
    else
        dst[i] = v;
}

template <int S, int API>
__device__ __forceinline__ aos<S> load_any(const aos<S>* src, long long i) {
    if constexpr (API == API_DIRECT) return src[i];
    if (trove::warp_converged()) return load_conv<S, API>(src, i);
    return load_div<S, API>(src, i);
}

template <int S, int API>
__device__ __forceinline__ void store_any(aos<S>* dst, long long i, const aos<S>& v) {
    if constexpr (API == API_DIRECT) {
        dst[i] = v;
    } else {
        if (trove::warp_converged())
            store_conv<S, API>(dst, i, v);
        else
            store_div<S, API>(dst, i, v);
    }
}

struct WarpGrid {
    int lane;
    long long warp, warps;
    __device__ __forceinline__ WarpGrid() {
        lane = int(threadIdx.x & 31u);
        warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
        warps = ((long long)gridDim.x * blockDim.x) >> 5;
    }
};

// dst[i] = src[i], optionally skipping structs whose first word hits the
// early-exit predicate (EXIT).  Full chunks are warp-uniform, so their loads
// run with all 32 lanes; stores after an exit see a partial warp and fall back.
// The one partial chunk at the end of the array is plain per-lane struct
// copies: its transposing form would be a second inlined copy of the tile
// schedule, and every register that copy holds lowers the occupancy of the
// whole kernel.
//
// LOOP = false: the grid has one chunk per warp (the default launch) and the
// kernel has no loop.  The grid-stride loop's 64-bit induction state costs
// 4-8 registers per thread, enough to push narrow structs at U = 1 from 24
// to 32+ registers and below full occupancy (2048 threads per SM), which is
// where a one-chunk kernel gets its loads in flight.  LOOP = true serves
// caller-chosen and persistent grids.
//
// Resident blocks that the early-exit copy is built for, by the words of a lane: up
// to 16 words fit 32 registers (of 12 bytes, 4 to a lane, with 8 bytes spilled), but
// ptxas takes 34-48 where it may (1 GiB of 12 bytes, 4 structs to a lane, 326 us at 40
// registers and 306 at 32; 24 bytes, 2 to a lane, 319 and 302).  One struct of more
// than 8 words to a lane is left alone: fewer warps fill the memory system (44 bytes
// 301.8 us, 303.6 at 64 warps).  0: as ptxas likes, which a bound of 1 is not (64
// bytes 32 registers, 38 with it: 16 MiB 5.5 us and 6.1).
template <int S, int U>
constexpr int exit_blocks = S * U <= (U > 1 ? 16 : 8) ? 8 : 0;
template <int S, int U>
constexpr bool exit_multiply = S * U <= (U > 1 ? 12 : 8);

template <int S, int U, int API, bool EXIT, bool MULTIPLY>
__device__ __forceinline__ void copy_chunk(const aos<S>* __restrict__ src, aos<S>* __restrict__ dst, long long n,
                                           const ExitTest& test, long long base, int lane) {
    constexpr int CH = 32 * U;
    if (base + CH <= n) {
        aos<S> v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = load_conv<S, API>(src, base + u * 32 + lane);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (!EXIT || !exits<MULTIPLY>(v[u], test)) {
                if constexpr (EXIT)
                    store_any<S, API>(dst, base + u * 32 + lane, v[u]);
                else
                    store_conv<S, API>(dst, base + u * 32 + lane, v[u]);
            }
        }
    } else {
#pragma unroll 1
        for (int u = 0; u < U; ++u) {
            const long long i = base + u * 32 + lane;
            if (i < n) {
                const aos<S> v = src[i];
                if (!EXIT || !exits<MULTIPLY>(v, test)) dst[i] = v;
            }
        }
    }
}

template <int S, int U, int API, bool EXIT, bool LOOP>
__global__ void __launch_bounds__(256, EXIT && !LOOP ? exit_blocks<S, U> : 0)
copy_kernel(const aos<S>* __restrict__ src, aos<S>* __restrict__ dst, long long n, ExitTest test) {
    const WarpGrid g;
    constexpr int CH = 32 * U;
    if constexpr (LOOP) {
        for (long long base = g.warp * CH; base < n; base += g.warps * CH)
            copy_chunk<S, U, API, EXIT, false>(src, dst, n, test, base, g.lane);
    } else {
        const long long base = g.warp * CH;
        if (base < n) copy_chunk<S, U, API, EXIT, exit_multiply<S, U>>(src, dst, n, test, base, g.lane);
    }
}

// MODE 0: coalesced_ptr (trove::load / trove::store); MODE 1: compiler
// direct.  Index loads of a chunk are coalesced; every load of the chunk is
// issued before its stores.
enum { MODE_COALESCED = 0, MODE_DIRECT = 1 };

template <int S, int U, int MODE>
__global__ void __launch_bounds__(256)
gather_kernel(const aos<S>* __restrict__ src, long long src_n, const int* __restrict__ idx,
              aos<S>* __restrict__ dst, long long n) {
    const WarpGrid g;
    constexpr int CH = 32 * U;
    trove::coalesced_ptr<aos<S> > S_(const_cast<aos<S>*>(src));
    trove::coalesced_ptr<aos<S> > D_(dst);
    for (long long base = g.warp * CH; base < n; base += g.warps * CH) {
        int id[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const long long i = base + u * 32 + g.lane;
            id[u] = i < n ? __ldg(idx + i) : -1;
        }
        aos<S> v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (id[u] >= 0 && (long long)id[u] < src_n) {
                if constexpr (MODE == MODE_COALESCED)
                    v[u] = S_[id[u]];
                else
                    v[u] = src[id[u]];
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const long long i = base + u * 32 + g.lane;
            if (id[u] >= 0 && (long long)id[u] < src_n) {
                if constexpr (MODE == MODE_COALESCED)
                    D_[i] = v[u];
                else
                    dst[i] = v[u];
            }
        }
    }
}

template <int S, int U, int MODE>
__global__ void __launch_bounds__(256)
scatter_kernel(const aos<S>* __restrict__ src, const int* __restrict__ idx, aos<S>* __restrict__ dst,
               long long dst_n, long long n) {
    const WarpGrid g;
    constexpr int CH = 32 * U;
    trove::coalesced_ptr<aos<S> > S_(const_cast<aos<S>*>(src));
    trove::coalesced_ptr<aos<S> > D_(dst);
    for (long long base = g.warp * CH; base < n; base += g.warps * CH) {
        int id[U];
        aos<S> v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const long long i = base + u * 32 + g.lane;
            id[u] = i < n ? __ldg(idx + i) : -1;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const long long i = base + u * 32 + g.lane;
            if (i < n) {
                if constexpr (MODE == MODE_COALESCED)
                    v[u] = S_[i];
                else
                    v[u] = src[i];
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (id[u] >= 0 && (long long)id[u] < dst_n) {
                if constexpr (MODE == MODE_COALESCED)
                    D_[id[u]] = v[u];
                else
                    dst[id[u]] = v[u];
            }
        }
    }
}

// The default grid of coalesced_ptr: one chunk per warp, without the loop's
// registers: 34 instead of 48 at 36 bytes, 40 instead of 60 at 64, so up to 56 warps
// an SM instead of 40.  2^23 structs in runs of 32, 36 bytes 145.5 -> 133.0 us, 64
// bytes 199.3 -> 171.9.  Compiler-generated access has the loop always: without it
// 2^23 sorted structs of 24 bytes took 94 us at 4 to a lane instead of 80.
template <int S, int U>
__device__ __forceinline__ void gather_chunk(const aos<S>* __restrict__ src, long long src_n,
                                             const int* __restrict__ idx, aos<S>* __restrict__ dst, int rem, int lane) {
    trove::coalesced_ptr<aos<S> > S_(const_cast<aos<S>*>(src));
    trove::coalesced_ptr<aos<S> > D_(dst);
    int id[U];
#pragma unroll
    for (int u = 0; u < U; ++u) id[u] = u * 32 + lane < rem ? __ldg(idx + u * 32 + lane) : -1;
    aos<S> v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        if (id[u] >= 0 && (long long)id[u] < src_n) v[u] = S_[id[u]];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        if (id[u] >= 0 && (long long)id[u] < src_n) D_[u * 32 + lane] = v[u];
    }
}

template <int S, int U>
__device__ __forceinline__ void scatter_chunk(const aos<S>* __restrict__ src, const int* __restrict__ idx,
                                              aos<S>* __restrict__ dst, long long dst_n, int rem, int lane) {
    trove::coalesced_ptr<aos<S> > S_(const_cast<aos<S>*>(src));
    trove::coalesced_ptr<aos<S> > D_(dst);
    int id[U];
    aos<S> v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) id[u] = u * 32 + lane < rem ? __ldg(idx + u * 32 + lane) : -1;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        if (u * 32 + lane < rem) v[u] = S_[u * 32 + lane];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        if (id[u] >= 0 && (long long)id[u] < dst_n) D_[id[u]] = v[u];
    }
}

template <int S, int U>
__global__ void __launch_bounds__(256)
gather_once_kernel(const aos<S>* __restrict__ src, long long src_n, const int* __restrict__ idx,
                   aos<S>* __restrict__ dst, long long n) {
    const WarpGrid g;
    constexpr int CH = 32 * U;
    const long long base = g.warp * CH;
    if (base >= n) return;
    const int rem = n - base < CH ? int(n - base) : CH;
    gather_chunk<S, U>(src, src_n, idx + base, dst + base, rem, g.lane);
}

template <int S, int U>
__global__ void __launch_bounds__(256)
scatter_once_kernel(const aos<S>* __restrict__ src, const int* __restrict__ idx, aos<S>* __restrict__ dst,
                    long long dst_n, long long n) {
    const WarpGrid g;
    constexpr int CH = 32 * U;
    const long long base = g.warp * CH;
    if (base >= n) return;
    const int rem = n - base < CH ? int(n - base) : CH;
    scatter_chunk<S, U>(src + base, idx + base, dst, dst_n, rem, g.lane);
}

// ---- cache policies of the row-form kernels ----------------------------
// 0: default (read-only path for loads, plain stores)
// 1: the index stream and the contiguous side are streamed (evict-first), so
//    L2 keeps the random side's sectors: structs narrower than a 32-byte
//    sector share sectors, and a sector that stays in L2 is fetched once
// 2: as 1, and the random side bypasses L1 (L2 only)
// 3: as 1, and the random side is marked evict-last in L2
// 4: as 1, and random-side loads carry a 64-byte L2 prefetch-size hint
__device__ __forceinline__ unsigned long long l2_evict_last_policy() {
    unsigned long long pol;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}

__device__ __forceinline__ int ld_index(const int* p, int policy) { return policy ? __ldcs(p) : __ldg(p); }

__device__ __forceinline__ uint4 ld_hint(const uint4* p, unsigned long long pol) {
    uint4 v;
    asm volatile("ld.global.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p), "l"(pol));
    return v;
}
__device__ __forceinline__ uint2 ld_hint(const uint2* p, unsigned long long pol) {
    uint2 v;
    asm volatile("ld.global.L2::cache_hint.v2.u32 {%0, %1}, [%2], %3;" : "=r"(v.x), "=r"(v.y) : "l"(p), "l"(pol));
    return v;
}
__device__ __forceinline__ unsigned ld_hint(const unsigned* p, unsigned long long pol) {
    unsigned v;
    asm volatile("ld.global.L2::cache_hint.u32 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(pol));
    return v;
}
__device__ __forceinline__ void st_hint(uint4* p, uint4 v, unsigned long long pol) {
    asm volatile("st.global.L2::cache_hint.v4.u32 [%0], {%1, %2, %3, %4}, %5;" ::"l"(p), "r"(v.x), "r"(v.y),
                 "r"(v.z), "r"(v.w), "l"(pol)
                 : "memory");
}
__device__ __forceinline__ void st_hint(uint2* p, uint2 v, unsigned long long pol) {
    asm volatile("st.global.L2::cache_hint.v2.u32 [%0], {%1, %2}, %3;" ::"l"(p), "r"(v.x), "r"(v.y), "l"(pol)
                 : "memory");
}
__device__ __forceinline__ void st_hint(unsigned* p, unsigned v, unsigned long long pol) {
    asm volatile("st.global.L2::cache_hint.u32 [%0], %1, %2;" ::"l"(p), "r"(v), "l"(pol) : "memory");
}

// Random-side loads with a 64-byte L2 prefetch-size hint: on a miss L2 is
// asked for the 64-byte half line holding the word instead of the whole
// 128-byte line.
__device__ __forceinline__ uint4 ld_pf64(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.nc.L2::64B.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}
__device__ __forceinline__ uint2 ld_pf64(const uint2* p) {
    uint2 v;
    asm volatile("ld.global.nc.L2::64B.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ unsigned ld_pf64(const unsigned* p) {
    unsigned v;
    asm volatile("ld.global.nc.L2::64B.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

// The same with a 128-byte prefetch-size hint: a miss fetches the whole
// 128-byte line, whose neighbouring structs a narrow gather over a source
// near the L2 size often reads while the line is still cached.
__device__ __forceinline__ uint4 ld_pf128(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.nc.L2::128B.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}
__device__ __forceinline__ uint2 ld_pf128(const uint2* p) {
    uint2 v;
    asm volatile("ld.global.nc.L2::128B.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ unsigned ld_pf128(const unsigned* p) {
    unsigned v;
    asm volatile("ld.global.nc.L2::128B.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

template <typename V>
__device__ __forceinline__ V ld_random(const V* p, int policy, unsigned long long pol) {
    if (policy == 5) return ld_pf128(p);
    if (policy == 4) return ld_pf64(p);
    if (policy == 3) return ld_hint(p, pol);
    if (policy == 2) return __ldcg(p);
    return __ldg(p);
}
template <typename V>
__device__ __forceinline__ V ld_contig(const V* p, int policy) {
    return policy ? __ldcs(p) : __ldg(p);
}
template <typename V>
__device__ __forceinline__ void st_random(V* p, V v, int policy, unsigned long long pol) {
    if (policy == 3)
        st_hint(p, v, pol);
    else if (policy == 2)
        __stcg(p, v);
    else
        *p = v;
}
template <typename V>
__device__ __forceinline__ void st_contig(V* p, V v, int policy) {
    if (policy)
        __stcs(p, v);
    else
        *p = v;
}

// Row-form gather / scatter (TRV_PATH_WARP for index ops).  The C ABI knows
// both sides of the operation, and one side is contiguous, so no struct ever
// needs to sit in one lane: the warp moves 32 structs as m = 4S/sizeof(V)
// rounds of 32 words V.  In round k lane l carries word q = l + 32k of the
// chunk, i.e. word q % m of struct j = q / m, whose index comes from lane j
// by one 32-bit shuffle.  Gather: the random side is the load (adjacent lanes
// read adjacent words of one struct in the same instruction), the store lands
// at word q of the contiguous destination chunk (fully coalesced).  Scatter is
// the mirror image.  No transposes, no 64-bit pointer broadcasts.

// Struct and word of the round-k word of lane l, stepped from round to round
// (two or three integer instructions instead of a division per round).
template <int m>
struct RowStep {
    int j, r;
    __device__ __forceinline__ explicit RowStep(int lane) : j(lane / m), r(lane - (lane / m) * m) {}
    __device__ __forceinline__ void next() {
        j += 32 / m;
        if constexpr (32 % m != 0) {
            r += 32 % m;
            if (r >= m) {
                r -= m;
                ++j;
            }
        }
    }
};

// A random-side load that is skipped where `at` < 0 (predicated, no branch:
// a branch around each load made the warp's loads of a chunk issue one
// divergence region at a time).  POL as the cache policies above.
template <int POL>
__device__ __forceinline__ void ld_row(uint4& v, const void* p, int at) {
    if constexpr (POL == 4)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ge.s32 p, %5, 0;\n\t"
                     "@p ld.global.nc.L2::64B.v4.u32 {%0, %1, %2, %3}, [%4];\n\t}"
                     : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p), "r"(at));
    else if constexpr (POL == 5)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ge.s32 p, %5, 0;\n\t"
                     "@p ld.global.nc.L2::128B.v4.u32 {%0, %1, %2, %3}, [%4];\n\t}"
                     : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p), "r"(at));
    else
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ge.s32 p, %5, 0;\n\t"
                     "@p ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];\n\t}"
                     : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p), "r"(at));
}
template <int POL>
__device__ __forceinline__ void ld_row(uint2& v, const void* p, int at) {
    if constexpr (POL == 4)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ge.s32 p, %3, 0;\n\t"
                     "@p ld.global.nc.L2::64B.v2.u32 {%0, %1}, [%2];\n\t}"
                     : "=r"(v.x), "=r"(v.y) : "l"(p), "r"(at));
    else if constexpr (POL == 5)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ge.s32 p, %3, 0;\n\t"
                     "@p ld.global.nc.L2::128B.v2.u32 {%0, %1}, [%2];\n\t}"
                     : "=r"(v.x), "=r"(v.y) : "l"(p), "r"(at));
    else
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ge.s32 p, %3, 0;\n\t"
                     "@p ld.global.nc.v2.u32 {%0, %1}, [%2];\n\t}"
                     : "=r"(v.x), "=r"(v.y) : "l"(p), "r"(at));
}
template <int POL>
__device__ __forceinline__ void ld_row(unsigned& v, const void* p, int at) {
    if constexpr (POL == 4)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ge.s32 p, %2, 0;\n\t@p ld.global.nc.L2::64B.u32 %0, [%1];\n\t}"
                     : "=r"(v) : "l"(p), "r"(at));
    else if constexpr (POL == 5)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ge.s32 p, %2, 0;\n\t@p ld.global.nc.L2::128B.u32 %0, [%1];\n\t}"
                     : "=r"(v) : "l"(p), "r"(at));
    else
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ge.s32 p, %2, 0;\n\t@p ld.global.nc.u32 %0, [%1];\n\t}"
                     : "=r"(v) : "l"(p), "r"(at));
}

// One chunk of 32*U structs by the calling warp: the default launches.  The
// cache policy is a template argument and every access is predicated: per word
// a shuffle, an address and the two accesses are left (with the policy tested
// at run time a 24-byte gather issued 45 instructions per word).  Large random
// gathers are bound by DRAM's random accesses and stay as they were; what the
// instructions bound got faster: 4096 structs of 28 bytes 3.78 -> 1.79 us
// (gather) and 3.14 -> 1.80 us (scatter), 2^20 of 36 bytes 27.0 -> 16.0 us,
// 2^20 of 20 bytes 15.0 -> 11.2 us.  32 registers up to 9 words in flight.
// `bound` is the random side's length, at most 2^31 (int32 indices reach no
// further); an index outside [0, bound) skips its struct.
template <int S, typename V, int U, int POL>
__device__ __forceinline__ void gather_rows_chunk(const V* __restrict__ src, unsigned bound,
                                                  const int* __restrict__ idx, V* __restrict__ dst, int rem,
                                                  int lane) {
    constexpr int m = S * 4 / int(sizeof(V));
    int id[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int v = u * 32 + lane < rem ? ld_index(idx + u * 32 + lane, POL) : -1;
        id[u] = unsigned(v) < bound ? v : -1;
    }
    V val[U][m];
    int from[U][m];
    RowStep<m> at(lane);
#pragma unroll
    for (int k = 0; k < m; ++k) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            from[u][k] = __shfl_sync(0xFFFFFFFFu, id[u], at.j);
            ld_row<POL>(val[u][k], reinterpret_cast<const char*>(src) + (unsigned long long)unsigned(from[u][k]) * (4u * S) +
                                       unsigned(at.r) * unsigned(sizeof(V)),
                        from[u][k]);
        }
        at.next();
    }
#pragma unroll
    for (int k = 0; k < m; ++k)
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (from[u][k] >= 0) st_contig(dst + u * 32 * m + 32 * k + lane, val[u][k], POL);
}

template <int S, typename V, int U, int POL>
__device__ __forceinline__ void scatter_rows_chunk(const V* __restrict__ src, const int* __restrict__ idx,
                                                   V* __restrict__ dst, unsigned bound, int rem, int lane) {
    constexpr int m = S * 4 / int(sizeof(V));
    int id[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int v = u * 32 + lane < rem ? ld_index(idx + u * 32 + lane, POL) : -1;
        id[u] = unsigned(v) < bound ? v : -1;
    }
    V val[U][m];
    int to[U][m];
    const RowStep<m> first(lane);
    RowStep<m> at = first;
#pragma unroll
    for (int k = 0; k < m; ++k) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            to[u][k] = __shfl_sync(0xFFFFFFFFu, id[u], at.j);
            if (to[u][k] >= 0) val[u][k] = ld_contig(src + u * 32 * m + 32 * k + lane, POL);
        }
        at.next();
    }
    at = first;
#pragma unroll
    for (int k = 0; k < m; ++k) {
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (to[u][k] >= 0)
                *reinterpret_cast<V*>(reinterpret_cast<char*>(dst) + (unsigned long long)unsigned(to[u][k]) * (4u * S) +
                                      unsigned(at.r) * unsigned(sizeof(V))) = val[u][k];
        at.next();
    }
}

template <int S, typename V, int U, int POL>
__global__ void __launch_bounds__(256)
gather_rows_once_kernel(const V* __restrict__ src, unsigned bound, const int* __restrict__ idx, V* __restrict__ dst,
                        long long n) {
    constexpr int m = S * 4 / int(sizeof(V));
    const long long base = ((long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * (32 * U);
    if (base >= n) return;
    const int rem = n - base < 32 * U ? int(n - base) : 32 * U;
    gather_rows_chunk<S, V, U, POL>(src, bound, idx + base, dst + base * m, rem, int(threadIdx.x & 31u));
}

template <int S, typename V, int U, int POL>
__global__ void __launch_bounds__(256)
scatter_rows_once_kernel(const V* __restrict__ src, const int* __restrict__ idx, V* __restrict__ dst, unsigned bound,
                         long long n) {
    constexpr int m = S * 4 / int(sizeof(V));
    const long long base = ((long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * (32 * U);
    if (base >= n) return;
    const int rem = n - base < 32 * U ? int(n - base) : 32 * U;
    scatter_rows_chunk<S, V, U, POL>(src + base * m, idx + base, dst, bound, rem, int(threadIdx.x & 31u));
}

// The grid-stride form with the policy given at run time: caller-chosen and
// persistent grids, and cache policies 2 and 3.  A scatter writes the rows
// [lo, dst_n) of its destination.
template <int S, typename V, int U>
__global__ void __launch_bounds__(256)
gather_rows_kernel(const V* __restrict__ src, long long src_n, const int* __restrict__ idx, V* __restrict__ dst,
                   long long n, int policy) {
    constexpr int m = S * 4 / int(sizeof(V));
    const WarpGrid g;
    constexpr int CH = 32 * U;
    const unsigned long long pol = policy == 3 ? l2_evict_last_policy() : 0ull;
    for (long long base = g.warp * CH; base < n; base += g.warps * CH) {
        int id[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const long long i = base + u * 32 + g.lane;
            const int v = i < n ? ld_index(idx + i, policy) : -1;
            id[u] = (v >= 0 && (long long)v < src_n) ? v : -1;
        }
        V val[U][m];
        int from[U][m];
#pragma unroll
        for (int u = 0; u < U; ++u) {
#pragma unroll
            for (int k = 0; k < m; ++k) {
                const int q = g.lane + 32 * k;
                const int j = q / m;
                from[u][k] = __shfl_sync(0xFFFFFFFFu, id[u], j);
                if (from[u][k] >= 0) val[u][k] = ld_random(src + (long long)from[u][k] * m + (q - j * m), policy, pol);
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
#pragma unroll
            for (int k = 0; k < m; ++k)
                if (from[u][k] >= 0) st_contig(dst + (base + u * 32) * m + g.lane + 32 * k, val[u][k], policy);
        }
    }
}

template <int S, typename V, int U>
__global__ void __launch_bounds__(256)
scatter_rows_kernel(const V* __restrict__ src, const int* __restrict__ idx, V* __restrict__ dst, long long lo,
                    long long dst_n, long long n, int policy) {
    constexpr int m = S * 4 / int(sizeof(V));
    const WarpGrid g;
    constexpr int CH = 32 * U;
    const unsigned long long pol = policy == 3 ? l2_evict_last_policy() : 0ull;
    for (long long base = g.warp * CH; base < n; base += g.warps * CH) {
        int id[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const long long i = base + u * 32 + g.lane;
            const int v = i < n ? ld_index(idx + i, policy) : -1;
            id[u] = ((long long)v >= lo && (long long)v < dst_n) ? v : -1;
        }
        V val[U][m];
        int to[U][m];
#pragma unroll
        for (int u = 0; u < U; ++u) {
#pragma unroll
            for (int k = 0; k < m; ++k) {
                const int q = g.lane + 32 * k;
                to[u][k] = __shfl_sync(0xFFFFFFFFu, id[u], q / m);
                if (to[u][k] >= 0) val[u][k] = ld_contig(src + (base + u * 32) * m + q, policy);
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
#pragma unroll
            for (int k = 0; k < m; ++k) {
                const int q = g.lane + 32 * k;
                if (to[u][k] >= 0) st_random(dst + (long long)to[u][k] * m + (q - (q / m) * m), val[u][k], policy, pol);
            }
        }
    }
}

// Row-form gather / scatter with the word count m given at run time: one
// kernel per word type serves every width that is a multiple of 4 bytes,
// including structs wider than the per-width tables cover (> 64 bytes).  Same
// scheme as the compile-time kernels above; the m rounds of a chunk run in
// groups of G so the live registers stay bounded for any m.
template <typename V, int G, bool GATHER>
__global__ void __launch_bounds__(256)
index_rows_rt_kernel(const V* __restrict__ src, const int* __restrict__ idx, V* __restrict__ dst, long long bound,
                     long long n, int m, int policy) {
    const WarpGrid g;
    const unsigned long long pol = policy == 3 ? l2_evict_last_policy() : 0ull;
    for (long long base = g.warp * 32; base < n; base += g.warps * 32) {
        const long long i = base + g.lane;
        const int v = i < n ? ld_index(idx + i, policy) : -1;
        const int id = (v >= 0 && (long long)v < bound) ? v : -1;
        for (int k0 = 0; k0 < m; k0 += G) {
            V val[G];
            int other[G];
#pragma unroll
            for (int t = 0; t < G; ++t) {
                const int k = k0 + t;
                other[t] = -1;
                if (k < m) {  // m is uniform: the whole warp takes the same branch
                    const int q = g.lane + 32 * k;
                    const int j = q / m;
                    other[t] = __shfl_sync(0xFFFFFFFFu, id, j);
                    if (other[t] >= 0)
                        val[t] = GATHER ? ld_random(src + (long long)other[t] * m + (q - j * m), policy, pol)
                                        : ld_contig(src + base * m + q, policy);
                }
            }
#pragma unroll
            for (int t = 0; t < G; ++t) {
                if (other[t] < 0) continue;
                const int q = g.lane + 32 * (k0 + t);
                if (GATHER)
                    st_contig(dst + base * m + q, val[t], policy);
                else
                    st_random(dst + (long long)other[t] * m + (q % m), val[t], policy, pol);
            }
        }
    }
}

// Wide rows (any number of words): a warp moves R rows as consecutive words, G
// of each lane in flight, stepping the row and the word from round to round.
// The grid-stride form above gives a warp 32 rows whatever the length of the
// array and divides for every word: few long warps on short arrays (2^12 rows
// of 228 bytes 15.3 us, 2.3 us here with 4 rows to a warp), and bound by its
// instructions with 4-byte words (2^18 rows of 132 bytes 23.6 -> 16.7 us).
template <typename V, int R, int G, int POL, bool GATHER>
__global__ void __launch_bounds__(256)
wide_rows_kernel(const V* __restrict__ src, const int* __restrict__ idx, V* __restrict__ dst, unsigned bound,
                 long long n, int m) {
    const int lane = int(threadIdx.x & 31u);
    const long long base = ((long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * R;
    if (base >= n) return;
    const int rem = n - base < R ? int(n - base) : R;
    const int v = lane < rem ? ld_index(idx + base + lane, 1) : -1;
    const int id = unsigned(v) < bound ? v : -1;
    const V* in = GATHER ? src : src + base * m;
    V* out = GATHER ? dst + base * m : dst;
    const unsigned row_bytes = unsigned(m) * unsigned(sizeof(V));
    const int step_j = 32 / m, step_r = 32 % m;
    int j = lane / m, r = lane % m;
    const int words = rem * m;
    for (int q0 = 0; q0 < words; q0 += 32 * G) {
        const int q = q0 + lane;
        V val[G];
        int other[G], word[G];
#pragma unroll
        for (int g = 0; g < G; ++g) {
            other[g] = __shfl_sync(0xFFFFFFFFu, id, j);
            if (q + 32 * g >= words) other[g] = -1;
            word[g] = r;
            if (GATHER)
                ld_row<POL>(val[g], reinterpret_cast<const char*>(in) + (unsigned long long)unsigned(other[g]) * row_bytes +
                                        unsigned(r) * unsigned(sizeof(V)), other[g]);
            else if (other[g] >= 0)
                val[g] = ld_contig(in + q + 32 * g, 1);
            j += step_j;
            r += step_r;
            if (r >= m) {
                r -= m;
                ++j;
            }
        }
#pragma unroll
        for (int g = 0; g < G; ++g) {
            if (other[g] < 0) continue;
            if (GATHER)
                st_contig(out + q + 32 * g, val[g], 1);
            else
                *reinterpret_cast<V*>(reinterpret_cast<char*>(out) + (unsigned long long)unsigned(other[g]) * row_bytes +
                                      unsigned(word[g]) * unsigned(sizeof(V))) = val[g];
        }
    }
}

// AoS <-> SoA for structs of S 32-bit fields: field j of struct i sits at
// aos[i].word(j) and soa[j * n + i].  The AoS side moves through the device
// API (load/store_warp_contiguous: coalesced rounds + transpose); the SoA side
// is S coalesced 32-bit streams, one per field.
// One chunk of 32*U structs; the partial chunk at the end moves per lane.
template <int S, int U>
__device__ __forceinline__ void aos_to_soa_chunk(const aos<S>* __restrict__ src, unsigned* __restrict__ dst,
                                                 long long n, long long base, int lane) {
    constexpr int CH = 32 * U;
    aos<S> v[U];
    const bool full = base + CH <= n;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const long long i = base + u * 32 + lane;
        if (full)
            v[u] = trove::load_warp_contiguous(src + i);
        else if (i < n)
            v[u] = src[i];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const long long i = base + u * 32 + lane;
        if (!full && i >= n) continue;
        const trove::detail::regs<unsigned, S> w = trove::detail::to_regs(v[u]);
#pragma unroll
        for (int j = 0; j < S; ++j) __stcs(dst + (long long)j * n + i, w.v[j]);
    }
}

template <int S, int U>
__device__ __forceinline__ void soa_to_aos_chunk(const unsigned* __restrict__ src, aos<S>* __restrict__ dst,
                                                 long long n, long long base, int lane) {
    constexpr int CH = 32 * U;
    const bool full = base + CH <= n;
    trove::detail::regs<unsigned, S> w[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const long long i = base + u * 32 + lane;
        if (full || i < n) {
#pragma unroll
            for (int j = 0; j < S; ++j) w[u].v[j] = __ldcs(src + (long long)j * n + i);
        }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const long long i = base + u * 32 + lane;
        const aos<S> v = trove::detail::from_regs(w[u]);
        if (full)
            trove::store_warp_contiguous(v, dst + i);
        else if (i < n)
            dst[i] = v;
    }
}

// LOOP as for copy_kernel: false = one chunk per warp (the default grid).
template <int S, int U, bool LOOP>
__global__ void __launch_bounds__(256)
aos_to_soa_kernel(const aos<S>* __restrict__ src, unsigned* __restrict__ dst, long long n) {
    const WarpGrid g;
    constexpr int CH = 32 * U;
    if constexpr (LOOP) {
        for (long long base = g.warp * CH; base < n; base += g.warps * CH)
            aos_to_soa_chunk<S, U>(src, dst, n, base, g.lane);
    } else {
        const long long base = g.warp * CH;
        if (base < n) aos_to_soa_chunk<S, U>(src, dst, n, base, g.lane);
    }
}

template <int S, int U, bool LOOP>
__global__ void __launch_bounds__(256)
soa_to_aos_kernel(const unsigned* __restrict__ src, aos<S>* __restrict__ dst, long long n) {
    const WarpGrid g;
    constexpr int CH = 32 * U;
    if constexpr (LOOP) {
        for (long long base = g.warp * CH; base < n; base += g.warps * CH)
            soa_to_aos_chunk<S, U>(src, dst, n, base, g.lane);
    } else {
        const long long base = g.warp * CH;
        if (base < n) soa_to_aos_chunk<S, U>(src, dst, n, base, g.lane);
    }
}

}  // namespace trv
