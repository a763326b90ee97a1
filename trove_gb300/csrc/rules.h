// The rules by which the C ABI chooses among its kernels where the caller and the
// autotuner leave the choice open: plain functions of sizes and alignment, without
// CUDA, so that the CPU tests compile and check them.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define TRV_HOST_DEVICE __host__ __device__
#else
#define TRV_HOST_DEVICE
#endif

namespace trv {

// ---- structs per lane --------------------------------------------------------

// Heuristic unroll when the caller gives none: about 16 words in flight per
// lane (tuned by the autotuner when a cache entry exists).
inline int default_unroll(uint32_t width) {
    const uint32_t words = width / 4;
    if (words <= 2) return 8;
    if (words <= 4) return 4;
    if (words <= 8) return 2;
    return 1;
}

// Structs per lane of the row-form kernels when the caller gives neither them nor a
// grid (a grid's few warps want more in flight, default_unroll: 2^22 rows of 12 bytes
// scattered by 152 blocks 113 us at 4, 146 at 1).  A call
// of at most 2^16 structs does not fill the GPU (2048 warps at one struct per
// lane): more structs per lane only lengthen each warp (4096 structs of 28
// bytes: 1.79 us at 1, 1.93 at 2, 2.43 at 4).  Above, one or two 4- or 8-byte
// words in flight per lane are too few (2^24 structs of 4 bytes: gather 99 us
// at 1, 80 at 2, 79 at 4; 2^20 of 8 bytes: 8.7 / 8.1 / 8.0 us; 2^20 of 12 to
// 24 bytes: 2-6 % faster at 2 than at 1), while from 28 bytes up one struct
// per lane is as fast or faster (2^20 of 36 bytes: 16.1 us at 1, 17.0 at 2).
// Scatters gain from 2 up to 8 bytes only (2^20 of 8 bytes: 8.8 / 7.8 us; of
// 24 bytes: 23.3 / 23.8).
inline int rows_unroll(bool gather, uint32_t width, uint64_t n) {
    if (n <= (uint64_t(1) << 16)) return 1;
    if (gather) return width <= 8 ? 4 : width <= 24 ? 2 : 1;
    return width <= 8 ? 2 : 1;
}

// The same for coalesced_ptr access, whose loads and stores go through a struct to a
// lane: 2^23 structs of 4 bytes 48.7 us at 1, 42.3 at 2, 41.1 at 4, 40.7 at 8;
// contiguous indices of 16 bytes 53.1 / 48.2 / 45.1 at 1 / 2 / 4; of 12 bytes 58.1 /
// 49.9 / 48.3, but random ones 86.9 / 86.3 / 90.2.  Scatters of 8 bytes in order gain
// up to 8 (2^24: 51.1 at 4, 49.1 at 8); from 28 bytes up 1 is as fast or faster, but
// for gathers of many 32-byte structs in runs (2^24: 196 us at 1, 190 at 2).
// Compiler-generated access (DIRECT) stays with default_unroll: 2^24 sorted structs
// of 28 bytes scattered in 298 us at 2, 344 at 1.
inline int struct_unroll(bool gather, uint32_t width, uint64_t n) {
    if (n <= (uint64_t(1) << 16)) return 1;
    if (width <= 8) return width == 4 || !gather ? 8 : 4;
    if (width == 32) return gather && n >= (uint64_t(1) << 22) ? 2 : 1;
    return width == 16 ? 4 : width <= 24 ? 2 : 1;
}

// Structs per lane of the early-exit copy when the caller gives none.  Up to 4
// MiB the GPU is not full and more to a lane only lengthens each warp (1 MiB of
// 12 bytes 1.74 us at 1, 1.94 at 2, 2.16 at 4).  Above, narrow structs need
// several in flight (1 GiB of 4 bytes 770 / 446 / 326 / 305 us at 1 / 2 / 4 / 8;
// of 8 bytes 442 / 324 / 304 / 306; of 12 bytes 380 / 351 / 309 / 322; of 16 bytes
// 315 / 303 / 304, but 16 MiB 5.9 / 5.6 / 5.3) and from 24 bytes up one is as good as
// two or better (24 bytes 298 / 302, 28 bytes 300 / 305).  20 bytes change over: 16
// MiB 7.4 / 8.0, 128 MiB 41.8 / 41.5, 1 GiB 315 / 307.
inline int exit_unroll(uint32_t width, uint64_t bytes) {
    if (bytes <= (uint64_t(4) << 20)) return width == 4 ? 2 : 1;
    if (width == 20) return bytes >= (uint64_t(128) << 20) ? 2 : 1;
    if (width == 16) return bytes < (uint64_t(64) << 20) ? 4 : 2;
    return width == 4 ? 8 : width <= 12 ? 4 : 1;
}

// The same for the layout conversions, in us at 1 / 2 / 4 / 8.  To SoA, 512 MiB of 4
// bytes 366 / 214 / 159 / 153, of 8 bytes 216 / 161 / 154 / 154, of 12 bytes 183 / 179 /
// 177 / 254 (32 MiB 13.9 / 13.9 / 14.6), 32 MiB of 16 bytes 11.7 / 10.7 / 10.3 / 10.7;
// 1 GiB of 20 bytes 1 % faster at 2, shorter ones as fast or slower; 24 and 28 bytes
// fastest at 1.  From 32 bytes on 1 too where the fields' arrays are aligned to
// sectors (1 GiB of 32 / 36 / 44 / 48 / 64 bytes 307 / 304 / 324 / 322 / 311 at 1, 306
// / 304 / 331 / 327 / 319 at 2).  Where they are not, a warp's 128 bytes of a field end
// in a sector that the next warp's begin, and a warp of two such pieces saves one of
// the two (352 / 320 / 344 / 364 / 398 at 1, 327 / 323 / 350 / 346 / 353 at 2; 40 / 52
// / 56 / 60 bytes 325 / 335 / 345 / 350 and 317 / 331 / 323 / 336): from 64 MiB on, but
// for 36 and 44 bytes, whose transpose holds more registers than it saves.  From SoA:
// 512 MiB of 12 bytes 190 / 158 / 156, of 24 bytes 159 / 159 / 157, of 28 bytes 156 /
// 157, but 16 MiB 5.1 / 4.7, of 32 bytes 5.1 / 4.6.
inline int layout_unroll(bool to_soa, uint32_t width, uint64_t n) {
    const uint64_t bytes = n * width, MiB = uint64_t(1) << 20;
    if (bytes < 4 * MiB) return width == 4 ? 2 : 1;
    if (width == 4) return 8;
    if (!to_soa) return width <= 12 ? 4 : width <= 24 ? 2 : width <= 32 && bytes < 24 * MiB ? 2 : 1;
    if (width == 8 || width == 16) return width == 8 ? 8 : 4;
    if (width == 12) return bytes >= 256 * MiB ? 4 : 2;
    if (width <= 28) return width == 20 && bytes >= 256 * MiB ? 2 : 1;
    return n % 8 != 0 && bytes >= 64 * MiB && width != 36 && width != 44 ? 2 : 1;
}

// ---- scatters in parts (scatter_parts.cu) ----------------------------------

// In how many parts a scatter writes its destination: 0, as one plain pass; 1,
// one pass after the destination has been fetched into L2; more, a pass for each
// part.  This is policy 6, asked for, tuned or by default.  `sectors`: the
// destination is 32-byte aligned.  Measured on GB300 with random permutations:
//  - rows that fill whole 32-byte sectors need no fill: one plain pass;
//  - up to 40 MiB of destination L2 absorbs the partial sectors of a destination
//    that it may still hold from its last use: plain / with the fetch in us, three
//    destinations in turn and one that is not in L2, of 24 bytes 24 MiB 12 / 18 and
//    29 / 25, 32 MiB 16 / 24 and 39 / 29, 40 MiB 26 / 29 and 47 / 33, 48 MiB 48 / 32
//    and 57 / 43; of 8 bytes 32 MiB 25 / 32, 40 MiB 39 / 41, 48 MiB 69 / 46; of 48
//    bytes 32 MiB 15 / 22, 40 MiB 24 / 25, 48 MiB 32 / 28.  The fetch costs rows in
//    order 2 us.  4-byte rows gain nothing from it (2^24: 103 against 104 us);
//  - up to 64 MiB one pass is still best (2^24 rows of 4 bytes, 64 MiB: 104 us,
//    114 in two; 3 * 2^20 of 20 bytes, 60 MiB: 49.4 and 55.0);
//  - parts of 48, 56 and 64 MiB: 2^24 rows of 24 bytes 406 / 409 / 429 us, of 60
//    bytes 931 / 916 / 927, 5 * 2^24 of 16 bytes 2921 / 2820 / 2848;
//  - a pass costs about 1 ns per index whatever it writes, so many parts lose
//    again: 5 * 2^24 rows of 20 bytes in 29 parts 3548 us against 3812 plain, of
//    24 bytes in 35 parts 4053 against 3853;
//  - a destination most of whose rows are not written would be fetched for
//    nothing;
//  - of rows wider than 64 bytes only the two sectors at the ends are filled, and
//    the passes pay later: plain / in parts in us, 2^20 rows of 80 bytes 47 / 53,
//    2^21 121 / 104; 2^20 of 120 bytes 77 / 87, 2^21 180 / 149; 400 MiB of 132 bytes
//    337 / 276, of 200 bytes 241 / 225 and, where half of them lie in order, 185 /
//    225: wider than 136 bytes they stay plain.  The fetch alone they never take
//    (kWideRows);
//  - packed rows (packed.cu), whose plain pass is slower, gain from the fetch from 22
//    MiB on (2^22 rows of 10 bytes 95 us, 107 without).
enum RowKind { kStructRows, kWideRows, kPackedRows };
constexpr uint64_t kPlainPackedBytes = uint64_t(22) << 20;
constexpr uint64_t kPlainScatterBytes = uint64_t(40) << 20;
constexpr uint64_t kOnePassBytes = uint64_t(64) << 20;
constexpr uint64_t kPartBytes = uint64_t(56) << 20;
constexpr uint64_t kMostParts = 24;
constexpr uint32_t kWidestInParts = 136;

inline int scatter_parts(uint32_t width, uint64_t n, uint64_t dst_n, bool sectors, RowKind kind) {
    const bool wide = kind == kWideRows;
    const uint64_t bytes = dst_n * width;
    if (n < 2 || bytes <= (kind == kPackedRows ? kPlainPackedBytes : kPlainScatterBytes) || 2 * n < dst_n) return 0;
    if (width % 32 == 0 && sectors) return 0;
    if (wide && (width > kWidestInParts || n < (uint64_t(1) << 21))) return 0;
    const uint64_t parts = bytes <= kOnePassBytes ? 1 : (bytes + kPartBytes - 1) / kPartBytes;
    if (parts > kMostParts || (parts == 1 && (width < 8 || wide))) return 0;
    return int(parts);
}

// The sample that tells scatters onto large destinations how their indices lie
// (fetch.cuh): lane k of a warp takes the indices at this position of n >= 2 and
// at the next one.  32 positions spread over the array, each seven further off a
// multiple of the array's 32nd than the one before: without that, in an array of a
// power of two all pairs lay across the same place of every run of 32 (2^24 rows of
// 48 bytes in shuffled runs of 32 were taken for random, 513 us against 268 plain).
constexpr int kSamples = 32;
TRV_HOST_DEVICE inline long long sample_position(int lane, long long n) {
    const long long p = (long long)lane * (n - 1) / kSamples, back = 7ll * lane;
    return p >= back ? p - back : p;
}

// Rows so near each other that their writes meet in L2 by themselves, and how
// many of the pairs have to be near: of wide rows fewer, since parts give them less
// (2^21 rows of 120 bytes of which half lie in order 126 us plain, 143 in parts).
constexpr int kNearBytes = 4096;
TRV_HOST_DEVICE inline int near_pairs(int row_bytes) { return row_bytes > 64 ? 12 : 20; }
TRV_HOST_DEVICE inline bool sample_near(int a, int b, int row_bytes) {
    const long long d = (long long)b - a;
    return (d < 0 ? -d : d) * row_bytes <= kNearBytes;
}

// ---- tiles of a batch (batch.cu) -----------------------------------------------

// Staging memory of a block of the batch kernel, by its resident blocks per SM, and
// the rows of one staged piece: of 16-byte words two pieces and their indices fit it,
// of 4- and 8-byte words three and four index arrays.  A piece of 16-byte words is at
// most a whole number of words for each of 256 threads, four or eight (2^24 rows of 32
// bytes in order 173 us in pieces of 512, 189 in pieces of 544).
constexpr int kPieces = 3, kIndexSlots = 4, kWidePieces = 2;
TRV_HOST_DEVICE constexpr int stage_bytes(int blocks_per_sm) { return blocks_per_sm == 2 ? 81408 : 40704; }
TRV_HOST_DEVICE constexpr int piece_rows(int stage, bool wide, int row_bytes) {
    const int fit = wide ? stage / (kWidePieces * (row_bytes + 4)) : stage / (kPieces * row_bytes + kIndexSlots * 4);
    const int even = stage / stage_bytes(4) * 4 * 256 * 16 / row_bytes;
    return (wide && even < fit ? even : fit) / 32 * 32;
}

// The largest tile of copies, gathers and scatters (by trv_op): big enough to amortise
// the queue step and the filling of the pieces, small enough that the tiles in flight,
// and with them the sources and destinations in use, stay in L2, and that the last
// ones balance across 152 SMs.  512 arrays of 1 K-4 M structs (14.9 GB) in us at 24 /
// 32 / 48 / 64 / 128 KiB: copies 1013 / 1015 / 1020 / 1026 / 1032, gathers 1479 / 1390 /
// 1356 / 1370 / 1508, scatters 510 / 513 / 523 / 538 / 672.  220 scatters of 1 K-1 M
// rows (1 GB) at 24 / 48 / 64 KiB: at random 501 / 477 / 479, in order 373 / 341 / 339.
// 24 gathers of 2^19 rows of 64 bytes in order: 257 at 48 KiB, 251 at 64.  A tile
// that is a little longer than whole pieces is cut to them (plan_task): of 16-byte rows
// 64 KiB are 4096, four pieces of 992 and a fifth of 128.
constexpr int kLargestTile[3] = {128 << 10, 64 << 10, 48 << 10};

struct TileTask {
    bool copy;
    uint32_t width;
    uint64_t n;
};

// Tile sizes of a batch where nothing else chooses them.  A tile takes a block about
// 8 us before its first rows arrive, then 1.2 ns a row and 23 ps a byte (one array a
// block, us: 16384 rows of 4 bytes 28, 1024 rows of 64 bytes 10), so rows of w bytes
// weigh w + 48, and a batch of mixed widths is dealt out by weight: in bytes alone a
// tile of narrow rows takes three times as long as one of wide rows.
//
// A batch that fits the resident blocks in one wave of tiles of at most 64 KiB gets
// tiles that just do so, whatever is left over of each array counted: a second wave
// of a few tiles costs as much as the first (256 arrays of 8192 rows of 16 bytes 24.7
// us in one wave of 512 tiles, 28.8 in 1024 and 31.4 in 2560).  A larger one gets four
// to a block, gathers two, up to the largest, so that the last ones are short (87
// arrays of 2-64 K structs, 46 MB of gathers 57 us with the largest tile, 43 so);
// copies, which take time by their bytes, not below 48 KiB.
class TileRule {
public:
    static constexpr int kRowWeight = 48;
    static constexpr double kOneWaveBytes = 64 << 10;
    // A shorter tile loses more in the queue step than it gains (256 arrays of 512 rows
    // 8.4 us in one tile each, 10.4 in two).
    static constexpr uint32_t kLeastRows = 512, kLeastCopyBytes = 8 << 10;

    template <typename TaskAt>  // TileTask TaskAt(k), k < count
    TileRule(TaskAt&& at, uint64_t count, int blocks) {
        double total = 0, most = 0;  // work, and the largest share of bytes in it
        uint64_t arrays = 0;
        for (uint64_t k = 0; k < count; ++k) {
            const TileTask t = at(k);
            if (!t.n) continue;
            const double w = weight(t.copy, t.width);
            total += double(t.n) * w;
            most = most < t.width / w ? t.width / w : most;
            ++arrays;
        }
        work_ = total / blocks;
        if (!arrays) one_wave_ = true;
        while (!one_wave_ && arrays <= uint64_t(blocks) && work_ * most <= kOneWaveBytes) {
            double tiles = 0;
            for (uint64_t k = 0; k < count; ++k) {
                const TileTask t = at(k);
                const uint64_t each = structs(work_, t.copy, t.width);
                tiles += double(t.n / each + (t.n % each != 0));
            }
            if (tiles <= blocks) {
                one_wave_ = true;
                return;
            }
            const double over = tiles / blocks, limit = kOneWaveBytes / most;
            if (work_ == limit) break;
            work_ *= over > 1.25 ? 1.25 : over < 1.05 ? 1.05 : over;
            if (work_ > limit) work_ = limit;  // the last try
        }
        work_ = total / blocks;
    }

    bool one_wave() const { return one_wave_; }

    // With a tuned size (0: none), which was tuned on some batch of such tasks: a batch
    // too small for the largest tiles takes no larger ones than its own (16 gathers of
    // 4-32 K rows 14 us, 27 with a tuned 64 KiB).
    int tile_bytes(int op, uint32_t width, int tuned) const {
        const int own = tile_bytes(op, width);
        if (tuned <= 0) return own;
        return (one_wave_ || own < kLargestTile[op]) && own < tuned ? own : tuned;
    }

    int tile_bytes(int op, uint32_t width) const {
        const bool copy = op == 0;
        if (one_wave_) return int(structs(work_, copy, width) * width);
        const double bytes = work_ / (op == 1 ? 2 : 4) * width / weight(copy, width);
        const double most = kLargestTile[op], least = copy ? 48 << 10 : kLeastRows * width;
        return int(bytes >= most ? most : bytes <= least ? least : bytes);
    }

private:
    static double weight(bool copy, uint32_t width) { return copy ? width : width + kRowWeight; }
    static uint64_t structs(double work, bool copy, uint32_t width) {  // of a tile: whole warps, as plan_task rounds
        const uint64_t s = uint64_t(work / weight(copy, width)), least = copy ? kLeastCopyBytes / width : kLeastRows;
        return (s < least ? least : s) / 32 * 32;
    }
    double work_ = 0;  // of a tile
    bool one_wave_ = false;
};

// Rows of any width and alignment move in 4-byte words (packed.cu) where that
// beats a thread per row moving bytes (flat.cu).  A word takes its bytes from at
// most two rows, and words read past a row from at most two more: rows have at least
// kLeastPackedWidth bytes, whatever pays.
//
// What pays, bytes / words in us.  Random rows: gathers of 29 bytes 6.5 / 2.8 for
// 2^12, of 13 bytes 4.8 / 3.9 for 2^16, of 6 bytes 5.1 / 5.6 for 2^18 and 16.4 / 9.5
// for 2^20; scatters of 13 bytes 4.9 / 2.4 for 2^12, of 6 / 8 / 10 bytes 5.9 / 4.3,
// 7.0 / 3.6 and 8.1 / 4.3 for 2^16, 50 / 24, 68 / 12 and 84 / 24 for 2^20.  In order:
// of 13 bytes 29.7 / 18.9 and 29.9 / 20.5 for 2^20, but the bytes of narrow rows meet
// in the same sectors by themselves: gathers of 6 bytes 8.0 / 8.5 for 2^20, scatters
// of 6 / 8 / 10 bytes 2.5 / 3.3, 2.2 / 3.4 and 2.8 / 3.8 for 2^16, 24 / 41, 29 / 44
// and 51 / 56 for 2^22.  Long scatters of up to 8 bytes so go by words only where a
// sample of the indices does not find them in order: both kernels are launched and
// one leaves, which takes 2 to 3 us, more than shorter ones lose.
enum PackedForm { kByBytes, kByWords, kBySample };
constexpr uint32_t kLeastPackedWidth = 4, kMostPackedWidth = 1u << 20;
inline PackedForm packed_form(bool gather, uint32_t width, uint64_t n) {
    if (width < kLeastPackedWidth || width > kMostPackedWidth) return kByBytes;  // words would come out wrong
    if (width < 6) return kByBytes;                                              // most words straddle rows
    if (width >= 13) return kByWords;
    if (gather) return n >= (1u << 19) ? kByWords : kByBytes;
    if (n < (1u << 16)) return kByBytes;
    return width <= 8 && n >= (1u << 20) ? kBySample : kByWords;
}

// Rows that a warp of the parts kernel takes at a time: its offsets inside such a
// slab have 32 bits.
constexpr int kSlabRounds = 16;
constexpr int kSlab = 32 * kSlabRounds;
constexpr uint32_t kMostPassWords = (1u << 30) / kSlab;
static_assert(kWidestInParts / 4 <= kMostPassWords, "a slab of the widest rows that go in parts");

}  // namespace trv
