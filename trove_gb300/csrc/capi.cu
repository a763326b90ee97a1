// C ABI entry points (include/trove_gb300.h): argument checks, path choice
// and launch shape, then one kernel launch on the caller's stream.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <map>
#include <mutex>
#include <new>
#include <utility>
#include <vector>

#include "autotune.h"
#include "bulk.h"
#include "flat.h"
#include "ops.h"
#include "rules.h"
#include "runtime.h"
#include "trove_gb300.h"

namespace trv {

thread_local int g_last_cuda_error = 0;

int cuda_fail(cudaError_t e) {
    g_last_cuda_error = int(e);
    return TRV_ERR_CUDA;
}

int check_launch() {
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TRV_OK : cuda_fail(e);
}

DeviceInfo& device_info() {
    static std::mutex mu;
    static DeviceInfo infos[64];
    static std::map<int, DeviceInfo> more;  // devices past the array (map nodes never move)
    int dev = 0;
    cudaGetDevice(&dev);
    DeviceInfo* dp;
    if (dev >= 0 && dev < 64) {
        dp = &infos[dev];
    } else {
        std::lock_guard<std::mutex> g(mu);
        dp = &more[dev];
    }
    DeviceInfo& d = *dp;
    if (!d.ready.load(std::memory_order_acquire)) {
        std::lock_guard<std::mutex> g(mu);
        if (!d.ready.load(std::memory_order_relaxed)) {
            cudaDeviceGetAttribute(&d.sm_count, cudaDevAttrMultiProcessorCount, dev);
            if (d.sm_count <= 0) d.sm_count = 1;
            d.device = dev;
            d.ready.store(true, std::memory_order_release);
        }
    }
    return d;
}

// The error flag is a module-scope device variable (one per device, zero at
// load), so finding it allocates nothing: callers that must not allocate
// (trv_batch_run_static) and stream capture can use it.  Resolve it outside
// a capture the first time (trv_batch_create and trv_server_create do).
__device__ int g_device_flag;

int* device_flag() {
    static std::mutex mu;
    DeviceInfo& d = device_info();
    std::lock_guard<std::mutex> g(mu);
    if (!d.flag) {
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_device_flag) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        d.flag = static_cast<int*>(p);
    }
    return d.flag;
}

int resident_blocks(const void* func, int block) {
    static std::mutex mu;
    static std::map<std::pair<int, const void*>, int> cache;  // (device, kernel) at 256 threads
    DeviceInfo& d = device_info();
    const std::pair<int, const void*> key(d.device, func);
    {
        std::lock_guard<std::mutex> g(mu);
        auto it = cache.find(key);
        if (it != cache.end() && block == 256) return it->second;
    }
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, func, block, 0) != cudaSuccess || per_sm < 1)
        per_sm = 1;
    const int r = per_sm * d.sm_count;
    if (block == 256) {
        std::lock_guard<std::mutex> g(mu);
        cache[key] = r;
    }
    return r;
}

int grid_for(const void* func, long long work_items, int items_per_block, int block, int requested) {
    if (requested > 0) return requested;
    long long need = (work_items + items_per_block - 1) / items_per_block;
    if (need < 1) need = 1;
    if (requested < 0) {  // persistent: no more blocks than can be resident at once
        const int cap = resident_blocks(func, block);
        return need < cap ? int(need) : cap;
    }
    return need < 0x7FFFFFFFll ? int(need) : 0x7FFFFFFF;  // one pass per warp
}

// True (and the grid) when the default launch applies: no grid requested and
// one 32*unroll-struct chunk per warp fits in a grid of 256-thread blocks.
bool one_chunk_per_warp(long long n, int unroll, int requested, int* grid) {
    if (requested != 0) return false;
    const long long per_block = 256ll * unroll;
    const long long need = (n + per_block - 1) / per_block;
    if (need < 1 || need > 0x7FFFFFFFll) return false;
    *grid = int(need);
    return true;
}

int unroll_slot(int unroll) {
    switch (unroll) {
        case 1: return 0;
        case 2: return 1;
        case 4: return 2;
        case 8: return 3;
    }
    return -1;
}

}  // namespace trv

using namespace trv;

namespace {

bool aligned(const void* p, uintptr_t a) { return (reinterpret_cast<uintptr_t>(p) & (a - 1)) == 0; }

// Whether p lies in this GPU's own memory: what is read or written again and again,
// or counts on L2, is not worth it over the link to host memory or another GPU.
// (The question takes about 0.1 us; only calls of tens of microseconds ask it.)
bool on_this_gpu(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeDevice && a.device == device_info().device;
}

bool size_ok(uint64_t n, uint32_t width) { return width != 0 && n <= (uint64_t(1) << 62) / width; }

bool struct_width(uint32_t width) { return width % 4 == 0 && width >= 4 && width <= 64; }

// Copies between different alignments are joined from aligned vectors (flat.cu)
// from this length on: 1 MiB shared 4-byte alignment 1.73 us by words and 1.81
// joined, odd addresses 2.6 by bytes and 1.8 joined; 64 KiB 1.6 and 1.7.  Short
// ones take one vector to a thread (1 MiB: 1.8 us at 1, 2.07 at 4; 16 MiB: 7.6
// and 7.1).  Host memory is written faster by words than by joined vectors (144 MB
// that share 4-byte alignment 391 us by words, 440 joined), but not by bytes (524
// and 438).
constexpr uint64_t kShiftCopyBytes = uint64_t(512) << 10;
constexpr uint64_t kShortShiftBytes = uint64_t(4) << 20;

// Copies of 16-byte vectors take one to a thread up to this length, which do not
// fill the GPU: in us at 1 / 4, 64 KiB 1.63 / 1.79, 512 KiB 1.63 / 1.84, 1 MiB 1.73 /
// 1.87, 1.5 MiB 1.93 / 1.86, 8 MiB 4.94 / 4.31, 1 GiB 371 / 301.
constexpr uint64_t kShortFlatBytes = uint64_t(1) << 20;

int copy_flat(void* dst, const void* src, uint64_t nbytes, int unroll, int grid_req, cudaStream_t st) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(src), b = reinterpret_cast<uintptr_t>(dst);
    int vec = 16;
    while (vec > 1 && ((a ^ b) & uintptr_t(vec - 1)) != 0) vec >>= 1;
    long long head = (long long)((vec - (a & uintptr_t(vec - 1))) & uintptr_t(vec - 1));
    if ((uint64_t)head > nbytes) head = (long long)nbytes;
    const int asked = unroll;
    if (unroll <= 0) unroll = vec == 16 && nbytes <= kShortFlatBytes ? 1 : 4;
    if (unroll_slot(unroll) < 0) return TRV_ERR_INVALID_ARGUMENT;
    if (vec < 16 && nbytes >= kShiftCopyBytes && (vec < 4 || on_this_gpu(dst))) {
        const ShiftPlan p = plan_shift_copy(src, dst, (long long)nbytes);
        const int u = asked > 0 ? std::min(asked, 4) : nbytes < kShortShiftBytes ? 1 : 4;
        launch_shift_copy(src, dst, (long long)nbytes, p, u,
                          grid_for(shift_copy_func(), p.body, 256 * u, 256, grid_req), st);
        return check_launch();
    }
    const void* func = flat_copy_func(vec, unroll);
    const long long body = ((long long)nbytes - head) / vec;
    const int grid = grid_for(func, body, 256 * unroll, 256, grid_req);
    launch_flat_copy(src, dst, (long long)nbytes, vec, int(head), unroll, grid, st);
    return check_launch();
}

int copy_bulk(void* dst, const void* src, uint64_t nbytes, int chunk, int grid_req, cudaStream_t st) {
    if (!bulk_copy_supported(src, dst)) return TRV_ERR_MISALIGNED;
    if (chunk <= 0) chunk = 32 << 10;
    // chunk is bounded before the ring size is computed, which would overflow
    if (chunk % 16 != 0 || chunk > (227 << 10) || bulk_copy_smem_bytes(chunk) > (227 << 10))
        return TRV_ERR_INVALID_ARGUMENT;
    int* flag = device_flag();
    if (!flag) return TRV_ERR_OUT_OF_MEMORY;
    const long long nchunks = (long long)((nbytes + chunk - 1) / chunk);
    int grid = grid_req > 0 ? grid_req : device_info().sm_count;
    if (grid > nchunks) grid = nchunks > 0 ? int(nchunks) : 1;
    const cudaError_t e = launch_bulk_copy(src, dst, (long long)nbytes, chunk, grid, flag, st);
    return e == cudaSuccess ? TRV_OK : cuda_fail(e);
}

// Copy path without a tuned entry: the flat vector copy, one pass per warp.
// It needs no alignment beyond the bytes themselves and measured 7.0-7.1 TB/s
// on 2 GiB arrays at every width on GB300 (TMA bulk 6.8 TB/s; the device-API
// kernels 6.85-7.18 TB/s once tuned).
constexpr int kDefaultCopyPath = TRV_PATH_VECTOR;

}  // namespace

extern "C" {

const char* trv_status_string(int32_t status) {
    switch (status) {
        case TRV_OK: return "ok";
        case TRV_ERR_INVALID_ARGUMENT: return "invalid argument";
        case TRV_ERR_UNSUPPORTED: return "unsupported path/width combination";
        case TRV_ERR_MISALIGNED: return "pointer alignment not supported by the requested path";
        case TRV_ERR_CUDA: return "CUDA error";
        case TRV_ERR_OUT_OF_MEMORY: return "out of device memory";
        case TRV_ERR_BUDGET: return "request exceeds the HBM budget";
        case TRV_ERR_TIMEOUT: return "timed out";
        case TRV_ERR_NOT_FOUND: return "not found";
        case TRV_ERR_BUSY: return "busy";
        case TRV_ERR_CANCELLED: return "cancelled";
        case TRV_ERR_DEVICE_FLAG: return "a kernel reported an error";
    }
    return "unknown status";
}

int32_t trv_version(void) { return 100; }

int32_t trv_last_cuda_error(void) { return g_last_cuda_error; }

int32_t trv_set_l2_fetch_granularity(int32_t bytes, int32_t* previous) {
    if (bytes != 32 && bytes != 64 && bytes != 128) return TRV_ERR_INVALID_ARGUMENT;
    size_t old = 0;
    cudaError_t e = cudaDeviceGetLimit(&old, cudaLimitMaxL2FetchGranularity);
    if (e != cudaSuccess) return cuda_fail(e);
    e = cudaDeviceSetLimit(cudaLimitMaxL2FetchGranularity, size_t(bytes));
    if (e != cudaSuccess) return cuda_fail(e);
    if (previous) *previous = int32_t(old);
    return TRV_OK;
}

int32_t trv_debug_set_bulk_wait_polls(uint32_t polls) {
    set_bulk_wait_polls(polls);
    return TRV_OK;
}

int32_t trv_check_device(void* stream) {
    cudaError_t e = cudaStreamSynchronize(static_cast<cudaStream_t>(stream));
    if (e != cudaSuccess) return cuda_fail(e);
    int* flag = device_flag();
    if (!flag) return TRV_ERR_OUT_OF_MEMORY;
    int h = 0;
    e = cudaMemcpy(&h, flag, sizeof(int), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return cuda_fail(e);
    if (h != 0) {
        e = cudaMemset(flag, 0, sizeof(int));
        if (e != cudaSuccess) return cuda_fail(e);
        return TRV_ERR_DEVICE_FLAG;
    }
    return TRV_OK;
}

int32_t trv_copy_ex(void* dst, const void* src, uint64_t n, uint32_t width, const trv_launch* cfg, void* stream) {
    if (!size_ok(n, width)) return TRV_ERR_INVALID_ARGUMENT;
    if (n == 0) return TRV_OK;
    if (!dst || !src) return TRV_ERR_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    trv_launch c = cfg ? *cfg : trv_launch{TRV_PATH_AUTO, 0, 0, 0, 0};
    if (c.block_threads != 0 && c.block_threads != 256) return TRV_ERR_UNSUPPORTED;
    if (c.path == TRV_PATH_AUTO) {
        TuneChoice t;
        if (tune_lookup(TuneKey{SCOPE_CALL, TRV_OP_COPY, int(width), len_bucket(n)}, &t) &&
            (t.path != TRV_PATH_BULK || bulk_copy_supported(src, dst)) &&
            (t.path != TRV_PATH_WARP || (struct_width(width) && aligned(dst, 4) && aligned(src, 4))))
            c = trv_launch{t.path, t.unroll, 0, t.grid, t.chunk, 0};
        else
            c.path = kDefaultCopyPath;
    }
    int path = c.path;
    const int unroll = c.unroll;
    const int grid_req = c.grid_blocks;
    if (path == TRV_PATH_VECTOR) return copy_flat(dst, src, n * width, unroll, grid_req, st);
    if (path == TRV_PATH_BULK) return copy_bulk(dst, src, n * width, c.chunk_bytes, grid_req, st);
    if (path != TRV_PATH_WARP && path != TRV_PATH_BLOCK && path != TRV_PATH_DIRECT) return TRV_ERR_UNSUPPORTED;
    if (!struct_width(width)) return TRV_ERR_UNSUPPORTED;
    if (!aligned(dst, 4) || !aligned(src, 4)) return TRV_ERR_MISALIGNED;
    const int u = unroll > 0 ? unroll : default_unroll(width);
    const int slot = unroll_slot(u);
    if (slot < 0) return TRV_ERR_INVALID_ARGUMENT;
    const int api = path == TRV_PATH_WARP ? 0 : path == TRV_PATH_BLOCK ? 1 : 2;
    const WidthOps* ops = ops_for_words(int(width / 4));
    const int ub = ops->built_unroll[slot];
    int grid = 0;
    const bool once = one_chunk_per_warp((long long)n, ub, grid_req, &grid);
    const CopyKernel& k = once ? ops->copy[api][slot] : ops->copy_grid[api][slot];
    if (!once) grid = grid_for(k.func, (long long)n, 256 * ub, 256, grid_req);
    k.launch(CopyArgs{src, dst, (long long)n, {}}, grid, 256, st);
    return check_launch();
}

int32_t trv_copy(void* dst, const void* src, uint64_t n, uint32_t width, void* stream) {
    return trv_copy_ex(dst, src, n, width, nullptr, stream);
}

int32_t trv_copy_exit_ex(void* dst, const void* src, uint64_t n, uint32_t width, uint32_t modulus,
                         const trv_launch* cfg, void* stream) {
    if (!size_ok(n, width) || !cfg) return TRV_ERR_INVALID_ARGUMENT;
    if (n == 0) return TRV_OK;
    if (!dst || !src) return TRV_ERR_INVALID_ARGUMENT;
    if (!struct_width(width)) return TRV_ERR_UNSUPPORTED;
    if (cfg->path != TRV_PATH_WARP && cfg->path != TRV_PATH_BLOCK) return TRV_ERR_UNSUPPORTED;
    if (cfg->block_threads != 0 && cfg->block_threads != 256) return TRV_ERR_UNSUPPORTED;
    if (!aligned(dst, 4) || !aligned(src, 4)) return TRV_ERR_MISALIGNED;
    int u = cfg->unroll, grid_req = cfg->grid_blocks;
    if (u == 0) {
        TuneChoice t;
        const int op = cfg->path == TRV_PATH_WARP ? TRV_OP_COPY_EXIT_WARP : TRV_OP_COPY_EXIT_BLOCK;
        if (tune_lookup(TuneKey{SCOPE_CALL, op, int(width), len_bucket(n)}, &t)) {
            u = t.unroll;
            if (grid_req == 0) grid_req = t.grid;
        } else {
            u = exit_unroll(width, n * width);
        }
    }
    const int slot = unroll_slot(u);
    if (slot < 0) return TRV_ERR_INVALID_ARGUMENT;
    const int api = cfg->path == TRV_PATH_WARP ? 0 : 1;
    const WidthOps* ops = ops_for_words(int(width / 4));
    const int ub = ops->built_unroll[slot];
    int grid = 0;
    const bool once = one_chunk_per_warp((long long)n, ub, grid_req, &grid);
    const CopyKernel& k = modulus == 0 ? (once ? ops->copy[api][slot] : ops->copy_grid[api][slot])  // no struct leaves
                          : once       ? ops->copy_exit[api][slot]
                                       : ops->copy_exit_grid[api][slot];
    if (!once) grid = grid_for(k.func, (long long)n, 256 * ub, 256, grid_req);
    k.launch(CopyArgs{src, dst, (long long)n, modulus == 0 ? ExitTest() : ExitTest(modulus)}, grid, 256,
             static_cast<cudaStream_t>(stream));
    return check_launch();
}

int32_t trv_copy_exit(void* dst, const void* src, uint64_t n, uint32_t width, uint32_t modulus, int32_t path,
                      void* stream) {
    trv_launch cfg = {path, 0, 0, 0, 0, 0};
    return trv_copy_exit_ex(dst, src, n, width, modulus, &cfg, stream);
}

// L2 fetch hint of a gather's random loads.  A source larger than L2 is
// fetched by 64-byte halves (policy 4): the rest of a 128-byte line would leave
// L2 before another row of it is asked for.  A source that fits (112 MiB of 126)
// and most of whose rows are read is fetched by whole lines (policy 5), which
// brings the neighbouring rows in early: in us at 64 / 128-byte fetches, 2^20
// rows of 64 bytes 28.6 / 25.5, 2^22 of 28 bytes 77.3 / 69.0, 2^23 of 12 bytes
// 94.7 / 81.9.  8-byte rows and narrower do not care, and between 112 and 256
// MiB GB300s differ (2^24 of 12 bytes 282 / 257 on one, 220 / 244 on another).
constexpr uint64_t kL2SourceBytes = uint64_t(112) << 20;
static int gather_policy(uint32_t width, uint64_t n, uint64_t src_n) {
    return width >= 12 && src_n * width <= kL2SourceBytes && 2 * n >= src_n ? 5 : 4;
}

// Without a tuned entry, struct gathers and scatters take the row-form path,
// streaming the index and contiguous side; scatters onto large destinations
// run in parts (policy 6).
static int32_t index_op(bool gather, void* dst, const void* src, uint64_t bound, const int32_t* idx, uint64_t n,
                        uint32_t width, const trv_launch* cfg, void* stream) {
    if (!size_ok(n, width) || !size_ok(bound, width)) return TRV_ERR_INVALID_ARGUMENT;
    if (n == 0) return TRV_OK;
    if (!dst || !src || !idx) return TRV_ERR_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    trv_launch c = cfg ? *cfg : trv_launch{TRV_PATH_AUTO, 0, 0, 0, 0};
    if (c.block_threads != 0 && c.block_threads != 256) return TRV_ERR_UNSUPPORTED;
    if (!aligned(idx, 4)) return TRV_ERR_MISALIGNED;
    const bool structs = struct_width(width) && aligned(dst, 4) && aligned(src, 4);
    const bool wide_words = width % 4 == 0 && width > 64 && aligned(dst, 4) && aligned(src, 4);
    if (c.path == TRV_PATH_AUTO) {
        TuneChoice t;
        if (structs && tune_lookup(TuneKey{SCOPE_CALL, gather ? TRV_OP_GATHER : TRV_OP_SCATTER, int(width),
                                           len_bucket(n)},
                                   &t))
            c = trv_launch{t.path, t.unroll, 0, t.grid, 0, t.cache_policy};
        else if (structs)
            c = gather                                    ? trv_launch{TRV_PATH_WARP, 0, 0, 0, 0, gather_policy(width, n, bound)}
                                                          : trv_launch{TRV_PATH_WARP, 0, 0, 0, 0, 6};
        else if (wide_words)
            c = trv_launch{TRV_PATH_WARP, 0, 0, 0, 0, gather ? gather_policy(width, n, bound) : 6};
        else
            c.path = TRV_PATH_VECTOR;
    }
    if (c.cache_policy < 0 || c.cache_policy > 6 || (gather && c.cache_policy == 6)) return TRV_ERR_INVALID_ARGUMENT;
    const int path = c.path;
    const int grid_req = c.grid_blocks;
    // Policy 6 asks for parts where they pay on the destination at hand: a tuned
    // entry does not know the destination's length.
    // Each part reads the indices and much of the source again, which host memory is
    // too far away for (3 * 2^20 rows of 24 bytes from there 361 us, 652 in parts).
    const RowKind kind = path == TRV_PATH_VECTOR ? kPackedRows : width > 64 ? kWideRows : kStructRows;
    int parts = gather ? 0 : scatter_parts(width, n, bound, aligned(dst, 32), kind);
    if (parts && !(on_this_gpu(dst) && on_this_gpu(src) && on_this_gpu(idx))) parts = 0;
    if (c.cache_policy == 6 && parts == 0) c.cache_policy = width > 64 ? 0 : 1;
    if (path == TRV_PATH_VECTOR) {  // any width, any alignment
        const long long blocks = (long long)((n + 255) / 256);
        const int cap = device_info().sm_count * 8;
        const int g = grid_req > 0 ? grid_req : (blocks < cap ? int(blocks) : cap);
        const PackedForm form = packed_form(gather, width, n);
        const bool sampled = form == kBySample;
        if (form != kByBytes) {
            if (parts == 1)
                launch_fetch_destination(IndexArgs{src, dst, idx, (long long)n, (long long)bound, 1}, int(width),
                                         kPlainPackedBytes, st);
            launch_index_packed(gather, src, idx, dst, (long long)bound, (long long)n, int(width),
                                grid_req > 0 ? grid_req : grid_req < 0 ? cap : 0, sampled, st);
        }
        if (form != kByWords) {
            if (gather)
                launch_gather_bytes(src, (long long)bound, idx, dst, (long long)n, width, g, st);
            else
                launch_scatter_bytes(src, idx, dst, (long long)bound, (long long)n, width, g, sampled, st);
        }
        return check_launch();
    }
    if (path != TRV_PATH_COALESCED && path != TRV_PATH_DIRECT && path != TRV_PATH_WARP) return TRV_ERR_UNSUPPORTED;
    if (path == TRV_PATH_WARP && width % 4 == 0 && width > 64) {  // run-time word count
        if (!aligned(dst, 4) || !aligned(src, 4)) return TRV_ERR_MISALIGNED;
        int wb = 16;
        while (wb > 4 && (width % uint32_t(wb) != 0 || !aligned(dst, uintptr_t(wb)) || !aligned(src, uintptr_t(wb))))
            wb >>= 1;
        const int m = int(width / uint32_t(wb));
        IndexArgs a{src, dst, idx, (long long)n, (long long)bound, c.cache_policy};
        if (c.cache_policy == 6 && grid_req == 0) {
            launch_scatter_passes(wb, a, m, parts, st);
            return check_launch();
        }
        if (grid_req == 0 && (gather ? c.cache_policy == 4 || c.cache_policy == 5 : c.cache_policy != 2 && c.cache_policy != 3) &&
            launch_wide_rows(gather, wb, a, m, st))
            return check_launch();
        const long long warps = (long long)((n + 31) / 32);
        const int grid = grid_for(index_rows_rt_func(gather, wb), warps, 8, 256, grid_req);
        launch_index_rows_rt(gather, wb, a, m, grid, st);
        return check_launch();
    }
    if (!struct_width(width)) return TRV_ERR_UNSUPPORTED;
    if (!aligned(dst, 4) || !aligned(src, 4)) return TRV_ERR_MISALIGNED;
    const int u = c.unroll > 0                ? c.unroll
                  : path == TRV_PATH_DIRECT || (path == TRV_PATH_WARP && grid_req != 0)
                      ? default_unroll(width)
                  : path == TRV_PATH_WARP ? rows_unroll(gather, width, n)
                                          : struct_unroll(gather, width, n);
    const int slot = unroll_slot(u);
    if (slot < 0) return TRV_ERR_INVALID_ARGUMENT;
    const WidthOps* ops = ops_for_words(int(width / 4));
    const IndexKernel* kp;
    if (path == TRV_PATH_WARP) {
        const uintptr_t wb = uintptr_t(ops->rows_word_bytes);
        const int var = (aligned(dst, wb) && aligned(src, wb)) ? 0 : 1;
        kp = gather ? &ops->gather_rows[var][slot] : &ops->scatter_rows[var][slot];
    } else {
        const int mode = path == TRV_PATH_COALESCED ? 0 : 1;
        kp = gather ? &ops->gather[mode][slot] : &ops->scatter[mode][slot];
    }
    const IndexKernel& k = *kp;
    int grid = 0;
    const bool once = one_chunk_per_warp((long long)n, ops->built_unroll[slot], grid_req, &grid);
    if (!once) grid = grid_for(k.func, (long long)n, 256 * ops->built_unroll[slot], 256, grid_req);
    if (path == TRV_PATH_WARP && c.cache_policy == 6 && grid_req != 0) {
        // a requested grid is each part's, and the requested structs per lane too
        for (int p = 0; p < parts; ++p) {
            IndexArgs a{src, dst, idx, (long long)n, (long long)bound * (p + 1) / parts, 1};
            a.lo = (long long)bound * p / parts;
            k.launch(a, grid, 256, st);
        }
        return check_launch();
    }
    if (path == TRV_PATH_WARP && c.cache_policy == 6) {
        const IndexArgs a{src, dst, idx, (long long)n, (long long)bound, 1, 0, once};
        if (parts > 1) {
            const int wb = kp == &ops->scatter_rows[0][slot] ? ops->rows_word_bytes : 4;
            launch_scatter_passes(wb, a, int(width) / wb, parts, st);
        } else {
            launch_fetch_destination(a, int(width), kPlainScatterBytes, st);
            k.launch(a, grid, 256, st);
        }
        return check_launch();
    }
    k.launch(IndexArgs{src, dst, idx, (long long)n, (long long)bound, c.cache_policy, 0, once}, grid, 256, st);
    return check_launch();
}

int32_t trv_gather_ex(void* dst, const void* src, uint64_t src_n, const int32_t* idx, uint64_t n, uint32_t width,
                      const trv_launch* cfg, void* stream) {
    return index_op(true, dst, src, src_n, idx, n, width, cfg, stream);
}

int32_t trv_gather(void* dst, const void* src, uint64_t src_n, const int32_t* idx, uint64_t n, uint32_t width,
                   void* stream) {
    return index_op(true, dst, src, src_n, idx, n, width, nullptr, stream);
}

int32_t trv_scatter_ex(void* dst, uint64_t dst_n, const void* src, const int32_t* idx, uint64_t n, uint32_t width,
                       const trv_launch* cfg, void* stream) {
    return index_op(false, dst, src, dst_n, idx, n, width, cfg, stream);
}

int32_t trv_scatter(void* dst, uint64_t dst_n, const void* src, const int32_t* idx, uint64_t n, uint32_t width,
                    void* stream) {
    return index_op(false, dst, src, dst_n, idx, n, width, nullptr, stream);
}

static int32_t layout_op(bool to_soa, void* dst, const void* src, uint64_t n, uint32_t width, const trv_launch* cfg,
                         void* stream) {
    if (!size_ok(n, width)) return TRV_ERR_INVALID_ARGUMENT;
    if (n == 0) return TRV_OK;
    if (!dst || !src) return TRV_ERR_INVALID_ARGUMENT;
    if (!struct_width(width)) return TRV_ERR_UNSUPPORTED;
    if (!aligned(dst, 4) || !aligned(src, 4)) return TRV_ERR_MISALIGNED;
    if (cfg && cfg->block_threads != 0 && cfg->block_threads != 256) return TRV_ERR_UNSUPPORTED;
    int u = cfg ? cfg->unroll : 0;
    int grid_req = cfg ? cfg->grid_blocks : 0;
    if (u == 0) {
        TuneChoice t;
        if (tune_lookup(TuneKey{SCOPE_CALL, to_soa ? TRV_OP_AOS_TO_SOA : TRV_OP_SOA_TO_AOS, int(width), len_bucket(n)},
                        &t)) {
            u = t.unroll;
            if (grid_req == 0) grid_req = t.grid;
        } else {
            u = layout_unroll(to_soa, width, n);
        }
    }
    const int slot = unroll_slot(u);
    if (slot < 0) return TRV_ERR_INVALID_ARGUMENT;
    const WidthOps* ops = ops_for_words(int(width / 4));
    const int ub = ops->built_unroll[slot];
    int grid = 0;
    const bool once = one_chunk_per_warp((long long)n, ub, grid_req, &grid);
    const CopyKernel& k = once ? (to_soa ? ops->aos_to_soa[slot] : ops->soa_to_aos[slot])
                               : (to_soa ? ops->aos_to_soa_grid[slot] : ops->soa_to_aos_grid[slot]);
    if (!once) grid = grid_for(k.func, (long long)n, 256 * ub, 256, grid_req);
    k.launch(CopyArgs{src, dst, (long long)n, {}}, grid, 256, static_cast<cudaStream_t>(stream));
    return check_launch();
}

int32_t trv_aos_to_soa(void* dst_soa, const void* src_aos, uint64_t n, uint32_t width, void* stream) {
    return layout_op(true, dst_soa, src_aos, n, width, nullptr, stream);
}

int32_t trv_soa_to_aos(void* dst_aos, const void* src_soa, uint64_t n, uint32_t width, void* stream) {
    return layout_op(false, dst_aos, src_soa, n, width, nullptr, stream);
}

int32_t trv_aos_to_soa_ex(void* dst_soa, const void* src_aos, uint64_t n, uint32_t width, const trv_launch* cfg,
                          void* stream) {
    return layout_op(true, dst_soa, src_aos, n, width, cfg, stream);
}

int32_t trv_soa_to_aos_ex(void* dst_aos, const void* src_soa, uint64_t n, uint32_t width, const trv_launch* cfg,
                          void* stream) {
    return layout_op(false, dst_aos, src_soa, n, width, cfg, stream);
}

int32_t trv_fill_uniform_indices(int32_t* idx, uint64_t n, uint32_t bound, uint64_t seed, void* stream) {
    if (n == 0) return TRV_OK;
    if (!idx || bound == 0 || bound > 0x7FFFFFFFu || n > (uint64_t(1) << 61)) return TRV_ERR_INVALID_ARGUMENT;
    if (!aligned(idx, 4)) return TRV_ERR_MISALIGNED;
    launch_uniform_indices(idx, (long long)n, bound, seed, device_info().sm_count * 8,
                           static_cast<cudaStream_t>(stream));
    return check_launch();
}

int32_t trv_fill_run_indices(int32_t* idx, uint64_t n, uint64_t seed, void* stream) {
    if (n == 0) return TRV_OK;
    if (!idx || n < 32 || n > 0x7FFFFFFFull) return TRV_ERR_INVALID_ARGUMENT;
    if (!aligned(idx, 4)) return TRV_ERR_MISALIGNED;
    launch_run_indices(idx, (long long)n, seed, device_info().sm_count * 8, static_cast<cudaStream_t>(stream));
    return check_launch();
}

int32_t trv_fill_permutation(int32_t* idx, uint64_t n, uint64_t seed, void* stream) {
    if (n == 0) return TRV_OK;
    if (!idx || n > 0x7FFFFFFFull) return TRV_ERR_INVALID_ARGUMENT;
    if (!aligned(idx, 4)) return TRV_ERR_MISALIGNED;
    // Fisher-Yates from the top: step i (i = n .. 2) swaps slot i - 1 with a
    // slot drawn from word i over [0, i).  Inherently sequential, so it runs
    // on the host and the result is copied once.
    std::vector<int32_t> h;
    try {
        h.resize(n);
    } catch (const std::bad_alloc&) {
        return TRV_ERR_OUT_OF_MEMORY;
    }
    for (uint64_t i = 0; i < n; ++i) h[i] = int32_t(i);
    for (uint64_t i = n; i > 1; --i) std::swap(h[i - 1], h[stream_bounded(seed, i, unsigned(i))]);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    cudaError_t e = cudaMemcpyAsync(idx, h.data(), n * sizeof(int32_t), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);  // h is freed on return
    return e == cudaSuccess ? TRV_OK : cuda_fail(e);
}

int32_t trv_fill_random_u32(uint32_t* dst, uint64_t nwords, uint64_t seed, void* stream) {
    if (nwords == 0) return TRV_OK;
    if (!dst || nwords > (uint64_t(1) << 61)) return TRV_ERR_INVALID_ARGUMENT;
    const int grid = device_info().sm_count * 8;
    launch_fill_u32(dst, (long long)nwords, seed, grid, static_cast<cudaStream_t>(stream));
    return check_launch();
}

}  // extern "C"
