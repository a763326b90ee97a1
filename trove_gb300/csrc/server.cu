// Serving: a request loop that admits copy / gather requests against an HBM
// budget and folds them into the batched persistent kernel (batch.cu).
//
// One dispatcher thread per server repeats:
//   1. completion — every in-flight batch whose event has fired marks its
//      requests done (latency = submit -> observed completion);
//   2. admission — queued requests, in arrival order, get their output carved
//      from the budget arena (first fit, 256-byte granules) while it fits;
//   3. launch — while a batch slot is free, up to max_batch_requests admitted
//      requests become one batch: its task table and tile prefixes are written
//      to the slot's pinned staging, copied to the slot's device table, and
//      the persistent kernel runs on the slot's stream, once for the batch's
//      small requests and once for its large ones, each followed by its own
//      completion event, so small requests do not wait for the largest one.
// With several slots, batches overlap on the GPU and requests that arrive
// while others run join the next batch: continuous batching, not a queue in
// front of a single launch.  Sources and index arrays stay device-resident
// (the caller owns them); the server owns only outputs and its tables.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdint>
#include <deque>
#include <map>
#include <mutex>
#include <new>
#include <thread>
#include <unordered_map>
#include <utility>
#include <vector>

#include "autotune.h"
#include "batch.h"
#include "rules.h"
#include "runtime.h"
#include "trove_gb300.h"

namespace trv {
namespace {

using clock_type = std::chrono::steady_clock;

constexpr uint64_t kGranule = 256;
// Register budget of the server's batch kernel: 4 resident blocks per SM, the
// batch default (the staged movers and TMA copy tiles need few registers).
constexpr int kServerBlocksPerSm = 4;

// First-fit allocator over one device allocation.
class Arena {
public:
    bool init(uint64_t bytes) {
        size_ = (bytes + kGranule - 1) / kGranule * kGranule;
        if (size_ == 0) return false;
        if (cudaMalloc(&base_, size_) != cudaSuccess) {
            cudaGetLastError();
            base_ = nullptr;
            return false;
        }
        free_[0] = size_;
        return true;
    }
    ~Arena() {
        if (base_) cudaFree(base_);
    }
    // Offset of a block of `bytes`, or UINT64_MAX if none fits.
    uint64_t alloc(uint64_t bytes) {
        bytes = (bytes + kGranule - 1) / kGranule * kGranule;
        for (auto it = free_.begin(); it != free_.end(); ++it) {
            if (it->second >= bytes) {
                const uint64_t off = it->first, left = it->second - bytes;
                free_.erase(it);
                if (left) free_[off + bytes] = left;
                used_ += bytes;
                return off;
            }
        }
        return UINT64_MAX;
    }
    void release(uint64_t off, uint64_t bytes) {
        bytes = (bytes + kGranule - 1) / kGranule * kGranule;
        used_ -= bytes;
        auto it = free_.emplace(off, bytes).first;
        auto next = std::next(it);
        if (next != free_.end() && it->first + it->second == next->first) {
            it->second += next->second;
            free_.erase(next);
        }
        if (it != free_.begin()) {
            auto prev = std::prev(it);
            if (prev->first + prev->second == it->first) {
                prev->second += it->second;
                free_.erase(it);
            }
        }
    }
    unsigned char* base() const { return static_cast<unsigned char*>(base_); }
    uint64_t size() const { return size_; }
    uint64_t used() const { return used_; }

private:
    void* base_ = nullptr;
    uint64_t size_ = 0, used_ = 0;
    std::map<uint64_t, uint64_t> free_;
};

enum ReqPhase { QUEUED, ADMITTED, LAUNCHED, DONE };

struct Req {
    trv_request r;
    ReqPhase phase = QUEUED;
    bool released = false;
    uint64_t off = 0, bytes = 0;
    int batch = -1;
    double submit_ms = 0, launch_ms = 0, done_ms = 0;
};

struct Slot {
    cudaStream_t stream = nullptr;
    cudaEvent_t done = nullptr;
    cudaEvent_t done_small = nullptr;  // after the small requests' launch, when the batch has two
    size_t n_small = 0;                // ids[0, n_small) complete at done_small (0: one launch)
    bool small_done = false;
    cudaError_t small_q = cudaErrorNotReady, done_q = cudaErrorNotReady;  // what the last poll saw
    unsigned char* d_tables = nullptr;
    unsigned char* h_tables = nullptr;  // pinned staging
    std::vector<uint64_t> ids;
    std::vector<std::pair<trv_request, uint64_t>> todo;  // the batch's requests, offset of each one's output
    bool busy = false;
};

// A batch's tables lie in one block, so that one copy brings them to the
// device: two work counters (zero), the small and the large requests' tile
// prefixes, the task table.
struct Tables {
    unsigned long long* counter;
    long long* prefix;  // of the small requests; the large ones' follows
    BatchTask* tasks;
    static size_t tasks_at(size_t take) { return (16 + (take + 2) * sizeof(long long) + 15) / 16 * 16; }
    static size_t bytes(size_t take) { return tasks_at(take) + take * sizeof(BatchTask); }
    Tables(unsigned char* p, size_t take)
        : counter(reinterpret_cast<unsigned long long*>(p)),
          prefix(reinterpret_cast<long long*>(p + 16)),
          tasks(reinterpret_cast<BatchTask*>(p + tasks_at(take))) {}
};

uint64_t request_bytes(const trv_request& r) {
    return 2 * r.n * r.width + (r.op == TRV_OP_GATHER ? 4 * r.n : 0);
}

// A batch's requests that move at most this many bytes run in a launch of
// their own ahead of the larger ones and complete at their own event.  On the
// serving stream of 50 k requests/s (lengths log-uniform up to 2^23 structs),
// thresholds of 4 / 16 / 64 / 128 / 256 / 512 MB gave p50 0.161 / 0.154 /
// 0.155 / 0.159 / 0.176 / 0.193 ms and p99 0.92 / 0.88 / 0.82 / 0.77 / 0.78 /
// 0.88 ms, against 0.206 / 1.02 ms with one launch per batch.
constexpr uint64_t kSmallRequestBytes = uint64_t(128) << 20;

// Upper limits of the slot count and of a slot's task table (every slot
// holds a device and a pinned copy of its table).
constexpr int kMaxInflight = 64;
constexpr int kMaxBatchRequests = 1 << 16;

}  // namespace
}  // namespace trv

using namespace trv;

struct trv_server {
    trv_server_config cfg{};
    int device = 0;
    int grid = 1;        // blocks of a small-request launch: an equal share of the GPU per slot
    int grid_large = 1;  // blocks of a large-request launch: every resident block
    Arena arena;
    std::vector<Slot> slots;
    std::mutex mu;
    std::condition_variable wake, finished;
    std::deque<uint64_t> queue;
    std::deque<uint64_t> admitted;
    std::unordered_map<uint64_t, Req> reqs;
    uint64_t next_id = 1;
    int batches = 0;
    bool stop = false;
    std::atomic<bool> kick{false};  // something to admit, or the stop: set under the lock
    int error = TRV_OK;
    trv_server_stats st{};
    std::vector<double> latencies;
    clock_type::time_point t0 = clock_type::now();
    std::thread dispatcher;

    double now_ms() const {
        return std::chrono::duration<double, std::milli>(clock_type::now() - t0).count();
    }

    void mark_done(uint64_t id, double t) {  // lock held
        Req& r = reqs[id];
        r.phase = DONE;
        r.done_ms = t;
        ++st.completed;
        st.bytes += request_bytes(r.r);
        latencies.push_back(r.done_ms - r.submit_ms);
        if (cfg.release_when_done && !r.released) {
            arena.release(r.off, r.bytes);
            r.released = true;
        }
    }

    // Asks the events of the in-flight batches, without the lock: a slot's
    // fields belong to the dispatcher alone.  True if any has fired.
    bool poll_events() {
        bool any = false;
        for (Slot& s : slots) {
            if (!s.busy) continue;
            if (s.n_small && !s.small_done) {
                s.small_q = cudaEventQuery(s.done_small);
                any |= s.small_q != cudaErrorNotReady;
            }
            s.done_q = cudaEventQuery(s.done);
            any |= s.done_q != cudaErrorNotReady;
        }
        return any;
    }

    void complete_fired() {  // lock held
        for (Slot& s : slots) {
            if (!s.busy) continue;
            if (s.n_small && !s.small_done && s.small_q != cudaErrorNotReady) {
                if (s.small_q == cudaSuccess) {
                    const double t = now_ms();
                    st.last_done_ms = t;
                    for (size_t k = 0; k < s.n_small; ++k) mark_done(s.ids[k], t);
                    s.small_done = true;
                } else if (error == TRV_OK) {
                    error = cuda_fail(s.small_q);
                }
            }
            if (s.done_q == cudaErrorNotReady) continue;
            if (s.done_q != cudaSuccess && error == TRV_OK) error = cuda_fail(s.done_q);
            const double t = now_ms();
            st.last_done_ms = t;
            for (size_t k = (s.n_small && s.small_done) ? s.n_small : 0; k < s.ids.size(); ++k) mark_done(s.ids[k], t);
            s.ids.clear();
            s.n_small = 0;
            s.small_done = false;
            s.small_q = s.done_q = cudaErrorNotReady;
            s.busy = false;
        }
    }

    void admit() {  // lock held
        while (!queue.empty()) {
            Req& r = reqs[queue.front()];
            const uint64_t off = arena.alloc(r.bytes);
            if (off == UINT64_MAX) break;  // FIFO: wait for budget to free up
            r.off = off;
            r.phase = ADMITTED;
            admitted.push_back(queue.front());
            queue.pop_front();
            ++st.admitted;
        }
    }

    // Fills the free slots.  The lock is held while a batch is taken, not while
    // its tables are written and its copies and kernels are launched (about 20
    // microseconds that every submission used to wait for).
    void launch_ready() {
        for (Slot& s : slots) {
            if (s.busy) continue;
            size_t take, ns;
            {
                std::lock_guard<std::mutex> g(mu);
                if (admitted.empty()) return;
                take = std::min<size_t>(admitted.size(), size_t(cfg.max_batch_requests));
                s.ids.assign(admitted.begin(), admitted.begin() + take);
                admitted.erase(admitted.begin(), admitted.begin() + take);
                // Small requests run in a launch of their own ahead of the large
                // ones, with their own completion event: they complete without
                // waiting for the largest request of the batch.  Each group keeps
                // its arrival order.
                const uint64_t small = kSmallRequestBytes;
                ns = size_t(std::stable_partition(s.ids.begin(), s.ids.end(),
                                                  [&](uint64_t id) { return request_bytes(reqs[id].r) <= small; }) -
                            s.ids.begin());
                const double t = now_ms();
                s.todo.clear();
                for (uint64_t id : s.ids) {
                    Req& r = reqs[id];
                    s.todo.emplace_back(r.r, r.off);
                    r.phase = LAUNCHED;
                    r.batch = batches;
                    r.launch_ms = t;
                }
                ++batches;
            }
            const Tables h(s.h_tables, take), d(s.d_tables, take);
            long long tiles[2] = {0, 0};
            const auto task_at = [&](uint64_t k) {
                const trv_request& r = s.todo[k].first;
                return TileTask{r.op == TRV_OP_COPY, r.width, r.n};
            };
            const TileRule rule[2] = {TileRule(task_at, ns, grid),
                                      TileRule([&](uint64_t k) { return task_at(ns + k); }, take - ns, grid_large)};
            for (size_t k = 0; k < take; ++k) {
                const trv_request& r = s.todo[k].first;
                const int grp = k < ns ? 0 : 1;
                TuneChoice c;
                const bool tuned = tune_lookup(TuneKey{SCOPE_BATCH, r.op, int(r.width), len_bucket(r.n)}, &c);
                const int tb = cfg.tile_bytes > 0 ? cfg.tile_bytes
                                                  : rule[grp].tile_bytes(r.op, r.width, tuned ? c.tile_bytes : 0);
                TaskPlan p;
                p.tile_bytes = tb;
                p.gather_policy = 7;  // rows staged through shared memory, 128-byte L2 fetches
                p.scatter_policy = 5;
                p.copy_bulk = 1;
                if (cfg.tile_bytes <= 0 && !(tuned && c.tile_bytes > 0) && !rule[grp].one_wave())
                    p.stage = stage_bytes(kServerBlocksPerSm);
                const long long nt = plan_task(r.op, r.width, r.n, r.src_n, r.src, arena.base() + s.todo[k].second,
                                               r.idx, p, &h.tasks[k]);
                h.prefix[k + size_t(grp)] = tiles[grp];
                tiles[grp] += nt;
            }
            h.prefix[ns] = tiles[0];
            h.prefix[take + 1] = tiles[1];
            h.counter[0] = h.counter[1] = 0;
            cudaError_t e = cudaMemcpyAsync(s.d_tables, s.h_tables, Tables::bytes(take), cudaMemcpyHostToDevice,
                                            s.stream);
            const bool two = ns > 0 && ns < take;
            int launches = 0;
            if (e == cudaSuccess && ns > 0 && tiles[0] > 0) {
                const int g = tiles[0] < grid ? int(tiles[0]) : grid;
                e = launch_batch_kernel(d.tasks, int(ns), d.prefix, d.counter, g, kServerBlocksPerSm, s.stream);
                ++launches;
            }
            if (e == cudaSuccess && two) e = cudaEventRecord(s.done_small, s.stream);
            if (e == cudaSuccess && ns < take && tiles[1] > 0) {
                const int g = tiles[1] < grid_large ? int(tiles[1]) : grid_large;
                e = launch_batch_kernel(d.tasks + ns, int(take - ns), d.prefix + ns + 1, d.counter + 1, g,
                                        kServerBlocksPerSm, s.stream);
                ++launches;
            }
            if (e == cudaSuccess) e = cudaEventRecord(s.done, s.stream);
            s.n_small = two ? ns : 0;
            s.small_done = false;
            s.busy = true;
            std::lock_guard<std::mutex> g(mu);
            if (e != cudaSuccess && error == TRV_OK) error = cuda_fail(e);
            st.batches += uint64_t(launches);
        }
    }

    bool any_busy() const {
        for (const Slot& s : slots)
            if (s.busy) return true;
        return false;
    }

    // While batches are in flight the dispatcher polls their events with a
    // yield between rounds, so it holds one host core busy; idle, it blocks
    // until a submission or a release wakes it.  A 20-microsecond sleep between
    // polls (which the kernel's timer slack stretches further) measured p50
    // 0.094 / 0.165 ms and p99 0.24 / 0.59 ms at 2 k / 50 k requests per
    // second, against 0.042 / 0.068 ms and 0.16 / 0.42 ms with the yield.
    // It takes the lock only when an event has fired or `kick` says that there
    // is something to admit: polling and launching under the lock made a
    // submission wait 17 us for it (submitting a burst of 64 requests: 1120 us,
    // 105 us since; the whole burst with its results copied out 1515 -> 636 us).
    void run() {
        cudaSetDevice(device);
        for (;;) {
            if (poll_events() | kick.exchange(false)) {
                {
                    std::lock_guard<std::mutex> g(mu);
                    complete_fired();
                    admit();
                    if (stop && queue.empty() && admitted.empty() && !any_busy()) break;
                }
                finished.notify_all();
                launch_ready();
            } else if (any_busy()) {
                std::this_thread::yield();
            } else {
                std::unique_lock<std::mutex> lk(mu);
                wake.wait_for(lk, std::chrono::milliseconds(1), [&] { return kick.load(); });
            }
        }
        finished.notify_all();
    }
};

namespace {

void free_slot(Slot& s) {
    if (s.stream) cudaStreamDestroy(s.stream);
    if (s.done) cudaEventDestroy(s.done);
    if (s.done_small) cudaEventDestroy(s.done_small);
    if (s.d_tables) cudaFree(s.d_tables);
    if (s.h_tables) cudaFreeHost(s.h_tables);
    s = Slot();
}

int validate_request(const trv_request& r, uint64_t budget) {
    if (r.op != TRV_OP_COPY && r.op != TRV_OP_GATHER) return TRV_ERR_INVALID_ARGUMENT;
    if (r.width == 0 || r.n == 0 || r.n > (uint64_t(1) << 40) / r.width) return TRV_ERR_INVALID_ARGUMENT;
    if (r.width % 4 != 0 || r.width > 64) return TRV_ERR_UNSUPPORTED;
    if (!r.src || (reinterpret_cast<uintptr_t>(r.src) & 3u)) return TRV_ERR_INVALID_ARGUMENT;
    if (r.op == TRV_OP_GATHER && (!r.idx || (reinterpret_cast<uintptr_t>(r.idx) & 3u) || r.src_n == 0))
        return TRV_ERR_INVALID_ARGUMENT;
    if (r.n * r.width > budget) return TRV_ERR_BUDGET;
    return TRV_OK;
}

void fill_stats(const std::vector<double>& lat, trv_server_stats* out) {
    if (lat.empty()) return;
    std::vector<double> v(lat);
    std::sort(v.begin(), v.end());
    auto q = [&](double p) { return v[std::min(v.size() - 1, size_t(p * double(v.size() - 1) + 0.5))]; };
    out->p50_ms = q(0.50);
    out->p99_ms = q(0.99);
    out->max_ms = v.back();
    double sum = 0;
    for (double x : v) sum += x;
    out->mean_ms = sum / double(v.size());
}

}  // namespace

extern "C" {

static int32_t server_create_impl(const trv_server_config* cfg, trv_server** out) {
    if (!cfg || !out) return TRV_ERR_INVALID_ARGUMENT;
    *out = nullptr;
    if (cfg->hbm_budget_bytes == 0 || cfg->max_inflight < 0 || cfg->max_inflight > kMaxInflight ||
        cfg->max_batch_requests < 0 || cfg->max_batch_requests > kMaxBatchRequests || cfg->tile_bytes < 0)
        return TRV_ERR_INVALID_ARGUMENT;
    // the batch kernel's error flag and set-up, resolved before the dispatcher runs
    if (!device_flag()) return TRV_ERR_CUDA;
    const int resident = batch_grid(kServerBlocksPerSm);
    if (resident < 1) return TRV_ERR_CUDA;
    trv_server* s = new (std::nothrow) trv_server;
    if (!s) return TRV_ERR_OUT_OF_MEMORY;
    s->cfg = *cfg;
    if (s->cfg.max_inflight == 0) s->cfg.max_inflight = 4;
    if (s->cfg.max_batch_requests == 0) s->cfg.max_batch_requests = 1024;
    cudaGetDevice(&s->device);
    if (!s->arena.init(cfg->hbm_budget_bytes)) {
        delete s;
        return TRV_ERR_OUT_OF_MEMORY;
    }
    try {
        s->slots.resize(size_t(s->cfg.max_inflight));
    } catch (...) {
        delete s;
        return TRV_ERR_OUT_OF_MEMORY;
    }
    const size_t nt = size_t(s->cfg.max_batch_requests);
    for (Slot& sl : s->slots) {
        cudaError_t e = cudaStreamCreateWithFlags(&sl.stream, cudaStreamNonBlocking);
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&sl.done, cudaEventDisableTiming);
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&sl.done_small, cudaEventDisableTiming);
        if (e == cudaSuccess) e = cudaMalloc(&sl.d_tables, Tables::bytes(nt));
        if (e == cudaSuccess) e = cudaMallocHost(&sl.h_tables, Tables::bytes(nt));
        if (e != cudaSuccess) {
            cudaGetLastError();
            for (Slot& x : s->slots) free_slot(x);
            delete s;
            return e == cudaErrorMemoryAllocation ? TRV_ERR_OUT_OF_MEMORY : cuda_fail(e);
        }
    }
    // Concurrent batches share the GPU: a small-request launch gets an equal
    // part of it.  A large-request launch gets every resident block: its
    // blocks take the SMs as other batches' blocks leave them, and a large
    // request running alone is not held to a fraction of the GPU (on the
    // serving stream at 50 k requests/s, p99 0.58 ms against 0.77 ms with
    // the equal part; 2 k requests/s: 0.23 against 0.32 ms; p50 unchanged).
    s->grid = std::max(1, resident / s->cfg.max_inflight);
    s->grid_large = std::max(1, resident);
    s->t0 = clock_type::now();
    try {
        s->dispatcher = std::thread([s] { s->run(); });
    } catch (...) {  // no thread to be had: undo everything above
        for (Slot& x : s->slots) free_slot(x);
        delete s;
        return TRV_ERR_OUT_OF_MEMORY;
    }
    *out = s;
    return TRV_OK;
}

int32_t trv_server_create(const trv_server_config* cfg, trv_server** out) {
    return no_throw([&] { return server_create_impl(cfg, out); });
}

static int32_t server_submit_impl(trv_server* s, const trv_request* req, uint64_t* id) {
    if (!s || !req) return TRV_ERR_INVALID_ARGUMENT;
    std::lock_guard<std::mutex> g(s->mu);
    ++s->st.submitted;
    const int rc = validate_request(*req, s->arena.size());
    if (rc != TRV_OK) {
        ++s->st.rejected;
        return rc;
    }
    if (s->stop) return TRV_ERR_CANCELLED;
    const uint64_t k = s->next_id++;
    Req& r = s->reqs[k];
    r.r = *req;
    r.bytes = req->n * req->width;
    r.submit_ms = s->now_ms();
    if (s->st.first_submit_ms == 0 && s->st.submitted == 1) s->st.first_submit_ms = r.submit_ms;
    s->queue.push_back(k);
    if (s->queue.size() > s->st.max_queued) s->st.max_queued = s->queue.size();
    if (id) *id = k;
    s->kick = true;
    s->wake.notify_one();
    return TRV_OK;
}

int32_t trv_server_submit(trv_server* s, const trv_request* req, uint64_t* id) {
    return no_throw([&] { return server_submit_impl(s, req, id); });
}

static void result_of(trv_server* s, const Req& r, trv_result* out) {
    out->status = r.phase == DONE ? TRV_OK : TRV_ERR_BUSY;
    out->batch = r.batch;
    out->dst = r.phase >= ADMITTED ? s->arena.base() + r.off : nullptr;
    out->submit_ms = r.submit_ms;
    out->launch_ms = r.launch_ms;
    out->done_ms = r.done_ms;
}

int32_t trv_server_poll(trv_server* s, uint64_t id, trv_result* out) {
    if (!s) return TRV_ERR_INVALID_ARGUMENT;
    std::lock_guard<std::mutex> g(s->mu);
    if (s->error != TRV_OK) return s->error;
    auto it = s->reqs.find(id);
    if (it == s->reqs.end() || (it->second.released && !s->cfg.release_when_done)) return TRV_ERR_NOT_FOUND;
    if (out) result_of(s, it->second, out);
    return it->second.phase == DONE ? TRV_OK : TRV_ERR_BUSY;
}

int32_t trv_server_wait(trv_server* s, uint64_t id, double timeout_ms, trv_result* out) {
    if (!s) return TRV_ERR_INVALID_ARGUMENT;
    std::unique_lock<std::mutex> lk(s->mu);
    const auto deadline = clock_type::now() + std::chrono::microseconds(int64_t(timeout_ms * 1000.0));
    for (;;) {
        if (s->error != TRV_OK) return s->error;
        auto it = s->reqs.find(id);
        if (it == s->reqs.end()) return TRV_ERR_NOT_FOUND;
        if (it->second.phase == DONE) {
            if (out) result_of(s, it->second, out);
            return TRV_OK;
        }
        if (s->finished.wait_until(lk, deadline) == std::cv_status::timeout) {
            it = s->reqs.find(id);
            if (it != s->reqs.end() && it->second.phase == DONE) continue;
            return TRV_ERR_TIMEOUT;
        }
    }
}

int32_t trv_server_release(trv_server* s, uint64_t id) {
    if (!s) return TRV_ERR_INVALID_ARGUMENT;
    std::lock_guard<std::mutex> g(s->mu);
    auto it = s->reqs.find(id);
    if (it == s->reqs.end()) return TRV_ERR_NOT_FOUND;
    Req& r = it->second;
    if (r.phase != DONE) return TRV_ERR_BUSY;
    if (!r.released) s->arena.release(r.off, r.bytes);
    s->reqs.erase(it);
    s->kick = true;
    s->wake.notify_one();
    return TRV_OK;
}

static int32_t server_stats_get_impl(trv_server* s, trv_server_stats* out) {
    if (!s || !out) return TRV_ERR_INVALID_ARGUMENT;
    std::lock_guard<std::mutex> g(s->mu);
    *out = s->st;
    out->budget_in_use = s->arena.used();
    fill_stats(s->latencies, out);
    return s->error;
}

int32_t trv_server_stats_get(trv_server* s, trv_server_stats* out) {
    return no_throw([&] { return server_stats_get_impl(s, out); });
}

static int32_t server_replay_impl(trv_server* s, const trv_request* reqs, const double* arrival_ms, uint64_t count,
                          uint64_t* ids, trv_server_stats* out) {
    if (!s || (count && (!reqs || !arrival_ms))) return TRV_ERR_INVALID_ARGUMENT;
    std::vector<uint64_t> mine(count, 0);
    const auto start = clock_type::now();
    for (uint64_t k = 0; k < count; ++k) {
        const auto when = start + std::chrono::nanoseconds(int64_t(arrival_ms[k] * 1e6));
        if (clock_type::now() + std::chrono::microseconds(200) < when)
            std::this_thread::sleep_until(when - std::chrono::microseconds(100));
        while (clock_type::now() < when) {
        }
        const int rc = trv_server_submit(s, &reqs[k], &mine[k]);
        if (rc != TRV_OK) return rc;
    }
    std::unique_lock<std::mutex> lk(s->mu);
    trv_server_stats r{};
    std::vector<double> lat;
    lat.reserve(count);
    for (uint64_t k = 0; k < count; ++k) {
        for (;;) {
            if (s->error != TRV_OK) return s->error;
            auto it = s->reqs.find(mine[k]);
            if (it == s->reqs.end() || it->second.phase == DONE) break;
            s->finished.wait_for(lk, std::chrono::milliseconds(50));
        }
        auto it = s->reqs.find(mine[k]);
        if (it == s->reqs.end()) continue;
        const Req& q = it->second;
        lat.push_back(q.done_ms - q.submit_ms);
        r.bytes += request_bytes(q.r);
        r.first_submit_ms = k == 0 ? q.submit_ms : std::min(r.first_submit_ms, q.submit_ms);
        r.last_done_ms = std::max(r.last_done_ms, q.done_ms);
    }
    r.submitted = count;
    r.completed = lat.size();
    r.admitted = lat.size();
    r.batches = s->st.batches;
    r.max_queued = s->st.max_queued;
    r.budget_in_use = s->arena.used();
    fill_stats(lat, &r);
    if (ids)
        for (uint64_t k = 0; k < count; ++k) ids[k] = mine[k];
    if (out) *out = r;
    return TRV_OK;
}

int32_t trv_server_replay(trv_server* s, const trv_request* reqs, const double* arrival_ms, uint64_t count,
                          uint64_t* ids, trv_server_stats* out) {
    return no_throw([&] { return server_replay_impl(s, reqs, arrival_ms, count, ids, out); });
}

static int32_t server_destroy_impl(trv_server* s) {
    if (!s) return TRV_ERR_INVALID_ARGUMENT;
    {
        std::lock_guard<std::mutex> g(s->mu);
        s->stop = true;
        s->kick = true;
        s->wake.notify_one();
    }
    if (s->dispatcher.joinable()) s->dispatcher.join();
    for (Slot& x : s->slots) {
        if (x.stream) cudaStreamSynchronize(x.stream);
        free_slot(x);
    }
    const int err = s->error;
    delete s;
    return err;
}

int32_t trv_server_destroy(trv_server* s) {
    return no_throw([&] { return server_destroy_impl(s); });
}

}  // extern "C"
