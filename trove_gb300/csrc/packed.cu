// Gather / scatter of structs of any width from kLeastPackedWidth bytes up at any
// alignment (packed records: 6, 13 bytes, or 4-byte widths at odd addresses), in
// 4-byte words.
//
// The contiguous side is dealt out by aligned 32-bit words, so a warp reads or
// writes whole sectors of it; the four bytes of a word come from one row, or
// where it straddles a row's end from two.  The
// random side is read as the aligned words that hold the bytes, joined by a
// funnel shift.  Bytes that no full word covers (a row's ends on the random
// side of a scatter, skipped rows, the ends of the arrays) move one by one, and
// no word is read that is not wholly inside the source array.
//
// One thread per row moving bytes was bound by its load / store instructions,
// each touching 32 rows: 2^22 rows of 13 bytes, gather 153 us (10 % of DRAM's
// rate) -> 45, scatter 435 -> 114; of 47 bytes 1235 -> 138 and 1567 -> 267.
// What is left is the instructions of the joins, about 80 for a warp's 32 words.
#include <cuda_runtime.h>
#include <stdint.h>

#include "fetch.cuh"
#include "flat.h"

namespace trv {
namespace {

constexpr int kWarps = 8;
constexpr int kFly = 4;     // words of a lane in flight

__device__ __forceinline__ unsigned ld_word(const unsigned char* p) {
    unsigned v;
    asm volatile("ld.global.nc.L2::64B.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

// The `need` (1 to 4) bytes at p in the low end of a word; what lies above them
// is undefined.  [lo, hi) is the array that p points into.
__device__ __forceinline__ unsigned ld_bytes(const unsigned char* p, int need, const unsigned char* lo,
                                             const unsigned char* hi) {
    const unsigned off = unsigned(reinterpret_cast<uintptr_t>(p)) & 3u;
    const unsigned char* a = p - off;
    const bool two = off + unsigned(need) > 4u;
    if (a >= lo && a + (two ? 8 : 4) <= hi) {
        const unsigned w0 = ld_word(a);
        const unsigned w1 = two ? ld_word(a + 4) : 0u;
        return __funnelshift_r(w0, w1, off * 8u);
    }
    unsigned v = 0;
    for (int b = 0; b < need; ++b) v |= unsigned(p[b]) << (8 * b);
    return v;
}

// The same, skipped where `want` is false, with nothing checked.
__device__ __forceinline__ void ld_word_if(unsigned& v, const unsigned char* p, bool want) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %2, 0;\n\t@p ld.global.nc.L2::64B.u32 %0, [%1];\n\t}"
                 : "+r"(v)
                 : "l"(p), "r"(int(want)));
}

// One warp: the destination bytes of kRows rows at a time, as the aligned words
// inside them and up to 3 bytes at either end.
template <int kRows>
__global__ void __launch_bounds__(32 * kWarps)
gather_packed_kernel(const unsigned char* __restrict__ src, unsigned bound, const int* __restrict__ idx,
                     unsigned char* __restrict__ dst, long long n, int width) {
    __shared__ int s_id[kWarps][kRows + 1];
    const int lane = int(threadIdx.x & 31u), warp = int(threadIdx.x >> 5);
    const unsigned char* hi = src + (unsigned long long)bound * unsigned(width);
    // the same for every chunk: kRows rows are a multiple of 4 bytes
    const int head = int((4u - (reinterpret_cast<uintptr_t>(dst) & 3u)) & 3u);
    const int bytes = kRows * width, tail = (bytes - head) & 3, words = (bytes - head) / 4;
    const int step_j = 128 / width, step_r = 128 % width;
    int* id = s_id[warp];
    if (lane == 0) id[kRows] = -1;  // read, never used
    for (long long base = ((long long)blockIdx.x * kWarps + warp) * kRows; base < n;
         base += (long long)gridDim.x * kWarps * kRows) {
        __syncwarp();
        bool inner = true;  // every row valid, and its words inside the array whatever its alignment
#pragma unroll
        for (int t = 0; t < kRows; t += 32) {
            if (kRows < 32 && lane >= kRows) break;
            const int v = base + t + lane < n ? __ldcs(idx + base + t + lane) : -1;
            id[t + lane] = unsigned(v) < bound ? v : -1;
            inner &= v >= 1 && (long long)v + 3 <= (long long)bound;
        }
        __syncwarp();
        inner = __all_sync(0xFFFFFFFFu, inner);
        unsigned char* out = dst + base * width;
        if (lane < head + tail) {  // the ends, byte by byte
            const int o = lane < head ? lane : bytes - tail + lane - head;
            const int v = id[o / width];
            if (v >= 0) out[o] = src[(long long)v * width + o % width];
        }
        out += head;
        int j = (head + 4 * lane) / width;
        int r = head + 4 * lane - j * width;
        if (inner) {
            for (int q = lane; q < words; q += 32 * kFly) {
                unsigned w0[kFly], w1[kFly], w2[kFly], w3[kFly], at0[kFly], at1[kFly], cut[kFly];
#pragma unroll
                for (int f = 0; f < kFly; ++f) {
                    const bool in = q + 32 * f < words;
                    const int row = in ? j : 0, have = width - r;
                    const unsigned char* p0 = src + (unsigned long long)unsigned(id[row]) * unsigned(width) + unsigned(r);
                    const unsigned char* p1 = src + (unsigned long long)unsigned(id[row + 1]) * unsigned(width);
                    const unsigned o0 = unsigned(reinterpret_cast<uintptr_t>(p0)) & 3u;
                    const unsigned o1 = unsigned(reinterpret_cast<uintptr_t>(p1)) & 3u;
                    const bool straddles = have < 4;
                    w0[f] = w1[f] = w2[f] = w3[f] = 0;
                    ld_word_if(w0[f], p0 - o0, in);
                    ld_word_if(w1[f], p0 - o0 + 4, in && int(o0) + (straddles ? have : 4) > 4);
                    ld_word_if(w2[f], p1 - o1, in && straddles);
                    ld_word_if(w3[f], p1 - o1 + 4, in && straddles && int(o1) > have);
                    at0[f] = o0 * 8;
                    at1[f] = o1 * 8;
                    cut[f] = straddles ? unsigned(32 - 8 * have) : 0u;
                    j += step_j;
                    r += step_r;
                    if (r >= width) {
                        r -= width;
                        ++j;
                    }
                }
#pragma unroll
                for (int f = 0; f < kFly; ++f) {
                    // the first row's bytes below the second's
                    const unsigned v0 = __funnelshift_r(w0[f], w1[f], at0[f]);
                    const unsigned v1 = __funnelshift_r(w2[f], w3[f], at1[f]);
                    if (q + 32 * f < words)
                        __stcs(reinterpret_cast<unsigned*>(out) + q + 32 * f, __funnelshift_r(v0 << cut[f], v1, cut[f]));
                }
            }
            continue;
        }
        for (int q = lane; q < words; q += 32) {
            unsigned val = 0, keep = 0;  // keep: the bytes to write, as a mask
            const int first = id[j], have = width - r < 4 ? width - r : 4;
            if (first >= 0) {
                val = ld_bytes(src + (long long)first * width + r, have, src, hi);
                keep = 0xFFFFFFFFu >> (8 * (4 - have));
            }
            if (have < 4) {
                const int second = id[j + 1];
                if (second >= 0) {
                    const unsigned v = ld_bytes(src + (long long)second * width, 4 - have, src, hi);
                    val = (val & keep) | (v << (8 * have));
                    keep |= 0xFFFFFFFFu << (8 * have);
                }
            }
            if (keep == 0xFFFFFFFFu) {
                __stcs(reinterpret_cast<unsigned*>(out) + q, val);
            } else if (keep) {
                for (int b = 0; b < 4; ++b)
                    if ((keep >> (8 * b)) & 1u) out[4 * q + b] = (unsigned char)(val >> (8 * b));
            }
            j += step_j;
            r += step_r;
            if (r >= width) {
                r -= width;
                ++j;
            }
        }
    }
}

// Whether a quarter of a scatter's kRows are valid at most.  Rows wider than 64 bytes
// move faster by words all the same, and chunks of fewer than 32 rows are not asked.
constexpr int kFewRowsWidth = 64;
template <int kRows>
__device__ __forceinline__ bool few_rows(int valid) {
    return __reduce_add_sync(0xFFFFFFFFu, unsigned(valid)) * 4u <= unsigned(kRows);
}

// Their bytes one by one over the lanes: the words of the rest would be walked through
// for nothing (2^20 rows of 13 bytes, nine in ten skipped: 13.4 us by words, 12.8 by a
// thread per row).  `at` lists the valid rows' places in the chunk.
template <int kRows>
__device__ __forceinline__ void scatter_few_rows(const unsigned char* from, unsigned char* dst, const int* id,
                                                 unsigned char* at, int width, int lane) {
    int cnt = 0;
#pragma unroll 1
    for (int t = 0; t < kRows; t += 32) {
        const bool mine = id[t + lane] >= 0;
        const unsigned b = __ballot_sync(0xFFFFFFFFu, mine);
        if (mine) at[cnt + __popc(b & ((1u << lane) - 1u))] = (unsigned char)(t + lane);
        cnt += __popc(b);
    }
    __syncwarp();
    const int bytes = cnt * width, step_j = 32 / width, step_r = 32 % width;
    int j = lane / width, r = lane % width;
    for (int q = lane; q < bytes; q += 32) {
        const unsigned row = at[j];
        dst[(unsigned long long)unsigned(id[row]) * unsigned(width) + unsigned(r)] = from[row * unsigned(width) + unsigned(r)];
        j += step_j;
        r += step_r;
        if (r >= width) {
            r -= width;
            ++j;
        }
    }
}

// One warp: kRows source rows, each as the `slots` aligned words of its
// destination row; slot k of a row that starts c bytes past a 4-byte boundary
// holds its bytes 4k - c to 4k - c + 3.
template <int kRows, bool SAMPLED>
__global__ void __launch_bounds__(32 * kWarps)
scatter_packed_kernel(const unsigned char* __restrict__ src, const int* __restrict__ idx,
                      unsigned char* __restrict__ dst, unsigned bound, long long n, int width) {
    __shared__ int s_id[kWarps][kRows];
    __shared__ unsigned char s_at[kWarps][kRows >= 32 ? kRows : 1];
    const int lane = int(threadIdx.x & 31u), warp = int(threadIdx.x >> 5);
    if constexpr (SAMPLED)
        if (IndexSample(idx, n, lane).rows_adjoin(width)) return;
    const unsigned char* hi = src + n * (long long)width;
    const int slots = (width + 6) / 4;
    const int step_j = 32 / slots, step_k = 32 % slots;
    int* id = s_id[warp];
    for (long long base = ((long long)blockIdx.x * kWarps + warp) * kRows; base < n;
         base += (long long)gridDim.x * kWarps * kRows) {
        __syncwarp();
        int valid = 0;  // the lane's valid rows
#pragma unroll
        for (int t = 0; t < kRows; t += 32) {
            if (kRows < 32 && lane >= kRows) break;
            const int v = base + t + lane < n ? __ldcs(idx + base + t + lane) : -1;
            id[t + lane] = unsigned(v) < bound ? v : -1;
            valid += unsigned(v) < bound;
        }
        __syncwarp();
        const unsigned char* from = src + base * width;
        if constexpr (kRows >= 32) {
            if (width <= kFewRowsWidth && few_rows<kRows>(valid)) {
                scatter_few_rows<kRows>(from, dst, id, s_at[warp], width, lane);
                continue;
            }
        }
        const int rows = n - base < kRows ? int(n - base) : kRows;
        const bool inner = base > 0 && base + rows + 2 <= n;  // words that reach past the rows are inside the array
        int j = lane / slots, k = lane % slots;
        while (j < rows) {
            unsigned w0[kFly], w1[kFly];
            unsigned at[kFly];
            unsigned char* out[kFly];
            int o[kFly];  // the row's byte at the word's start; nothing to write: `width`
#pragma unroll
            for (int f = 0; f < kFly; ++f) {
                const int v = j < rows ? id[j] : -1;
                unsigned char* d = dst + (unsigned long long)unsigned(v) * unsigned(width);
                o[f] = v >= 0 ? 4 * k - int(reinterpret_cast<uintptr_t>(d) & 3u) : width;
                out[f] = d + o[f];
                const unsigned char* p = from + (long long)(j * width) + o[f];
                const bool some = o[f] < width;
                if (inner) {
                    at[f] = (unsigned(reinterpret_cast<uintptr_t>(p)) & 3u) * 8;
                    w0[f] = w1[f] = 0;
                    ld_word_if(w0[f], p - (reinterpret_cast<uintptr_t>(p) & 3u), some);
                    ld_word_if(w1[f], p - (reinterpret_cast<uintptr_t>(p) & 3u) + 4, some && at[f] != 0);
                } else {
                    const int skip = o[f] < 0 ? -o[f] : 0;
                    const int last = width - o[f] < 4 ? width - o[f] : 4;
                    at[f] = 0;
                    if (skip < last) w0[f] = ld_bytes(p + skip, last - skip, src, hi) << (8 * skip);
                }
                j += step_j;
                k += step_k;
                if (k >= slots) {
                    k -= slots;
                    ++j;
                }
            }
#pragma unroll
            for (int f = 0; f < kFly; ++f) {
                const unsigned val = inner ? __funnelshift_r(w0[f], w1[f], at[f]) : w0[f];
                if (o[f] >= 0 && o[f] + 4 <= width) {
                    *reinterpret_cast<unsigned*>(out[f]) = val;
                } else {
#pragma unroll
                    for (int b = 0; b < 4; ++b)
                        if (unsigned(o[f] + b) < unsigned(width)) out[f][b] = (unsigned char)(val >> (8 * b));
                }
            }
        }
    }
}

unsigned clamp_bound(long long n) { return n > 0x80000000ll ? 0x80000000u : unsigned(n); }

}  // namespace

template <int ROWS>
static void launch(bool gather, const void* src, const int* idx, void* dst, long long bound, long long n, int width,
                   int grid, bool sampled, cudaStream_t st) {
    const unsigned char* s = static_cast<const unsigned char*>(src);
    unsigned char* d = static_cast<unsigned char*>(dst);
    if (grid <= 0) {
        const long long need = (n + kWarps * ROWS - 1) / (kWarps * ROWS);
        grid = need < 0x7FFFFFFFll ? int(need) : 0x7FFFFFFF;
    }
    if (gather)
        gather_packed_kernel<ROWS><<<grid, 32 * kWarps, 0, st>>>(s, clamp_bound(bound), idx, d, n, width);
    else if (ROWS == 128 && sampled)
        scatter_packed_kernel<128, true><<<grid, 32 * kWarps, 0, st>>>(s, idx, d, clamp_bound(bound), n, width);
    else
        scatter_packed_kernel<ROWS, false><<<grid, 32 * kWarps, 0, st>>>(s, idx, d, clamp_bound(bound), n, width);
}

// Rows to a warp, 8 to 128.  More rows to a warp waste less on its start and its
// last round of 32 words; fewer keep more warps busy where the rows are few, and
// the wider the rows, the fewer make up a warp's work.  Random gathers in us at 8 /
// 16 / 32 / 64 / 128: 2^16 rows of 13 bytes 4.5 / 3.7 / 4.1 / 5.6 / 8.9, 2^20 of them
// 47.6 / 25.5 / 16.1 / 14.5 / 16.7, 2^22 185 / 96 / 57 / 47 / 45; 2^17 of 29 bytes 7.3
// / 5.0 / 6.5 / 9.6 / 16.0, 2^20 48.8 / 29.5 / 25.6 / 25.6 / 30.4; 2^18 of 47 bytes
// 14.9 / 12.3 / 12.8 / 18.1 / 31.0, 2^20 54.0 / 42.3 / 34.0 / 37.4 / 47.4; 2^20 of 217
// bytes 142 / 127 / 133 / 156 / 202.  Scatters lie the same way (2^17 of 29 bytes 8.6
// / 6.6 / 6.9 / 8.6 / 12.9; 2^20 of 47 bytes 75.5 / 63.4 / 59.9 / 61.1 / 66.9); sorted
// ones of many rows want the most (2^20 of 7 bytes 51 / 27 / 14.6 / 13.6 / 11.8).
static int rows_to_a_warp(int width, long long n) {
    constexpr long long K = 1 << 10, M = 1 << 20, never = 1ll << 62;
    constexpr long long from[6][4] = {  // the least n for 16, 32, 64 and 128 rows
        {32 * K, 64 * K, 512 * K, 1 * M},   // up to 8 bytes
        {32 * K, 128 * K, 768 * K, 3 * M},  // up to 16
        {48 * K, 256 * K, 1 * M, 8 * M},    // up to 32
        {128 * K, 512 * K, 2 * M, 6 * M},   // up to 64
        {384 * K, 1 * M, never, never},     // up to 128
        {384 * K, 2 * M, never, never}};
    const long long* at = from[width <= 8 ? 0 : width <= 16 ? 1 : width <= 32 ? 2 : width <= 64 ? 3 : width <= 128 ? 4 : 5];
    int rows = 8;
    for (int k = 0; k < 4 && n >= at[k]; ++k) rows *= 2;
    return rows;
}

void launch_index_packed(bool gather, const void* src, const int* idx, void* dst, long long bound, long long n,
                         int width, int grid, bool sampled, cudaStream_t st) {
    switch (sampled ? 128 : rows_to_a_warp(width, n)) {
        case 8: return launch<8>(gather, src, idx, dst, bound, n, width, grid, sampled, st);
        case 16: return launch<16>(gather, src, idx, dst, bound, n, width, grid, sampled, st);
        case 32: return launch<32>(gather, src, idx, dst, bound, n, width, grid, sampled, st);
        case 64: return launch<64>(gather, src, idx, dst, bound, n, width, grid, sampled, st);
        default: return launch<128>(gather, src, idx, dst, bound, n, width, grid, sampled, st);
    }
}

}  // namespace trv
