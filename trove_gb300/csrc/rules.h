// The rules by which the C ABI chooses among its kernels where the caller and the
// autotuner leave the choice open: plain functions of sizes and alignment, without
// CUDA, so that the CPU tests compile and check them.
#pragma once

#include <cstdint>

namespace trv {

// ---- scatters in parts (scatter_parts.cu) ----------------------------------

// Rows that a warp of the parts kernel takes at a time, and the widest rows, in
// words moved, for which its offsets inside such a slab stay below 2^30 and so
// within 32 bits.  Wider rows are scattered in one pass of the row kernels, whose
// row offsets have 64 bits; with 8 MiB and more to a row there are no partial
// sectors worth saving.
constexpr int kSlabRounds = 16;
constexpr int kSlab = 32 * kSlabRounds;
constexpr uint32_t kMostPassWords = (1u << 30) / kSlab;

}  // namespace trv
