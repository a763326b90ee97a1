// Instantiations of the run-time-width row-form gather / scatter kernels.
#include "kernels.cuh"
#include "ops.h"

namespace trv {

namespace {
template <typename V, int G, bool GATHER>
void launch_rt(const IndexArgs& a, int m, int grid, cudaStream_t st) {
    index_rows_rt_kernel<V, G, GATHER><<<grid, 256, 0, st>>>(static_cast<const V*>(a.src), a.idx,
                                                            static_cast<V*>(a.dst), a.bound, a.n, m, a.policy);
}

template <typename V, int R, int G, int POL, bool GATHER>
void launch_wide(const IndexArgs& a, int m, cudaStream_t st) {
    const unsigned bound = a.bound > 0x80000000ll ? 0x80000000u : unsigned(a.bound);
    const unsigned grid = unsigned((a.n + 8 * R - 1) / (8 * R));
    wide_rows_kernel<V, R, G, POL, GATHER><<<grid, 256, 0, st>>>(static_cast<const V*>(a.src), a.idx,
                                                                 static_cast<V*>(a.dst), bound, a.n, m);
}

template <typename V, int R, int G>
void launch_wide_op(bool gather, const IndexArgs& a, int m, cudaStream_t st) {
    if (!gather)
        launch_wide<V, R, G, 1, false>(a, m, st);
    else if (a.policy == 4)
        launch_wide<V, R, G, 4, true>(a, m, st);
    else
        launch_wide<V, R, G, 5, true>(a, m, st);
}

template <typename V, int G>
void launch_wide_short(bool gather, const IndexArgs& a, int m, cudaStream_t st) {
    if (a.n <= (1 << 13))
        launch_wide_op<V, 4, G>(gather, a, m, st);
    else if (a.n <= (1 << 15))
        launch_wide_op<V, 8, G>(gather, a, m, st);
    else
        launch_wide_op<V, 16, G>(gather, a, m, st);
}
}  // namespace

// Rows to a warp by the length: gathers in us at 4 / 8 / 16 / 32 rows, 2^12 rows
// of 100 bytes 2.0 / 2.1 / 2.8 / 4.0; 2^15 3.8 / 3.1 / 3.1 / 4.0; 2^16 6.0 / 4.2 /
// 4.1; 2^18 22.5 / 16.2 / 16.1 / 13.2.  Beyond 2^16 rows (scatters 2^17), words of
// 8 and 16 bytes stay with the grid-stride form, whose 30 registers keep more
// warps resident (2^18 rows of 200 bytes 20.6 us, 26.5 here).
bool launch_wide_rows(bool gather, int word_bytes, const IndexArgs& a, int m, cudaStream_t st) {
    if (a.n <= (gather && word_bytes != 4 ? 1 << 16 : 1 << 17)) {
        if (word_bytes == 16)
            launch_wide_short<uint4, 4>(gather, a, m, st);
        else if (word_bytes == 8)
            launch_wide_short<uint2, 6>(gather, a, m, st);
        else
            launch_wide_short<unsigned, 8>(gather, a, m, st);
        return true;
    }
    if (word_bytes != 4 || a.n > 0x7FFFFFFFll * 256) return false;
    launch_wide_op<unsigned, 32, 4>(gather, a, m, st);
    return true;
}

void launch_index_rows_rt(bool gather, int word_bytes, const IndexArgs& a, int m, int grid, cudaStream_t st) {
    if (word_bytes == 16)
        gather ? launch_rt<uint4, 2, true>(a, m, grid, st) : launch_rt<uint4, 2, false>(a, m, grid, st);
    else if (word_bytes == 8)
        gather ? launch_rt<uint2, 4, true>(a, m, grid, st) : launch_rt<uint2, 4, false>(a, m, grid, st);
    else
        gather ? launch_rt<unsigned, 4, true>(a, m, grid, st) : launch_rt<unsigned, 4, false>(a, m, grid, st);
}

const void* index_rows_rt_func(bool gather, int word_bytes) {
    if (word_bytes == 16)
        return gather ? (const void*)&index_rows_rt_kernel<uint4, 2, true> : (const void*)&index_rows_rt_kernel<uint4, 2, false>;
    if (word_bytes == 8)
        return gather ? (const void*)&index_rows_rt_kernel<uint2, 4, true> : (const void*)&index_rows_rt_kernel<uint2, 4, false>;
    return gather ? (const void*)&index_rows_rt_kernel<unsigned, 4, true>
                  : (const void*)&index_rows_rt_kernel<unsigned, 4, false>;
}

}  // namespace trv
