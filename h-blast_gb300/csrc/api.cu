// api.cu -- the C ABI (include/hblast_gpu.h): resident database, batches,
// search launch, ordering and result collection.
//
// Replaces H-BLAST's host runtime (h_blast_v1.1/H-BLAST/h_blast.cu): no
// process-static state, no exit() on error, the database uploaded once and
// kept resident, every launch on a caller-chosen stream.
#include <cuda_runtime.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <array>
#include <atomic>
#include <exception>
#include <map>
#include <memory>
#include <mutex>
#include <new>
#include <numeric>
#include <shared_mutex>
#include <string>
#include <vector>

#include "../host/batch_builder.h"
#include "../host/blastdb.h"
#include "kernels.h"

namespace {

thread_local std::string g_err;

int fail(int code, const std::string &msg) {
    g_err = msg;
    return code;
}

#define CU(call)                                                                  \
    do {                                                                          \
        cudaError_t e_ = (call);                                                  \
        if (e_ != cudaSuccess)                                                    \
            return fail(e_ == cudaErrorMemoryAllocation ? HBG_ERR_NOMEM : HBG_ERR_CUDA, \
                        std::string(#call) + ": " + cudaGetErrorString(e_));      \
    } while (0)

int bits_for(int64_t v) {
    int b = 0;
    while (v > 0) {
        ++b;
        v >>= 1;
    }
    return b;
}

// Device allocations of batches and search results go through a small
// per-device cache: blocks freed while idle are kept (up to kPoolBytes per
// device, blocks of up to kPoolBlock) and handed out again for requests of
// at least half their size, so repeated small searches do not pay for
// cudaMalloc / cudaFree each time.  Large blocks (databases) are not kept.
constexpr size_t kPoolBytes = (size_t)2 << 30;
constexpr size_t kPoolBlock = (size_t)512 << 20;

struct DevicePool {
    std::mutex mu;
    std::map<void *, size_t> size_of;                 // every live allocation
    std::map<int, std::multimap<size_t, void *>> idle; // per device, by size
    std::map<int, size_t> idle_bytes;
};
DevicePool &pool() {
    static DevicePool *p = new DevicePool;   // never destroyed: frees may run at exit
    return *p;
}

// Allocation failures injected for tests (hbg_debug_fail_allocations): the
// next this many dalloc calls report cudaErrorMemoryAllocation.
std::atomic<int32_t> g_fail_allocs{0};

template <class T>
cudaError_t dalloc(T **p, size_t n) {
    *p = nullptr;
    for (int32_t k = g_fail_allocs.load(); k > 0;)
        if (g_fail_allocs.compare_exchange_weak(k, k - 1))
            return cudaErrorMemoryAllocation;
    if (n == 0)
        n = 1;
    const size_t bytes = n * sizeof(T);
    int dev = 0;
    cudaGetDevice(&dev);
    DevicePool &P = pool();
    {
        std::lock_guard<std::mutex> lock(P.mu);
        auto &idle = P.idle[dev];
        auto it = idle.lower_bound(bytes);
        if (it != idle.end() && it->first <= 2 * bytes) {
            *p = (T *)it->second;
            P.idle_bytes[dev] -= it->first;
            idle.erase(it);
            return cudaSuccess;
        }
    }
    void *q = nullptr;
    cudaError_t e = cudaMalloc(&q, bytes);
    if (e != cudaSuccess) {
        cudaGetLastError();   // a failed allocation must not surface at a later launch check
        return e;
    }
    std::lock_guard<std::mutex> lock(P.mu);
    P.size_of[q] = bytes;
    *p = (T *)q;
    return cudaSuccess;
}

// Free now (cudaFree waits for the device).
template <class T>
void dfree(T *&p) {
    if (p) {
        {
            DevicePool &P = pool();
            std::lock_guard<std::mutex> lock(P.mu);
            P.size_of.erase((void *)p);
        }
        cudaFree(p);
    }
    p = nullptr;
}

// Give back a block that no GPU work still uses (the caller has synchronised):
// kept for reuse when it fits the cache, else freed.
template <class T>
void dfree_idle(T *&p) {
    if (!p)
        return;
    int dev = 0;
    cudaGetDevice(&dev);
    DevicePool &P = pool();
    bool keep = false;
    {
        std::lock_guard<std::mutex> lock(P.mu);
        auto it = P.size_of.find((void *)p);
        if (it != P.size_of.end() && it->second <= kPoolBlock && P.idle_bytes[dev] + it->second <= kPoolBytes) {
            P.idle[dev].emplace(it->second, (void *)p);
            P.idle_bytes[dev] += it->second;
            keep = true;
        }
    }
    if (!keep)
        dfree(p);
    p = nullptr;
}

// A wait for the whole device is an error while any of its streams is captured,
// and ends the capture.  So captures of this library hold this mutex shared, and
// its waits for a device hold it alone; a search that would be captured meanwhile
// is launched directly.
std::shared_mutex &capture_mutex() {
    static std::shared_mutex *m = new std::shared_mutex;   // never destroyed, like the pool
    return *m;
}
cudaError_t wait_device() {
    std::unique_lock<std::shared_mutex> lock(capture_mutex());
    const cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess)
        cudaGetLastError();   // must not surface at a later launch check
    return e;
}

// Zeros before the first letter of a letter buffer; 64 follow the last:
// extensions read whole blocks.
constexpr size_t kFrontPad = 64;

// Device guard: make `dev` current for the scope.
struct DeviceScope {
    int prev = -1;
    explicit DeviceScope(int dev) {
        cudaGetDevice(&prev);
        if (prev != dev)
            cudaSetDevice(dev);
    }
    ~DeviceScope() {
        int cur = -1;
        cudaGetDevice(&cur);
        if (prev >= 0 && cur != prev)
            cudaSetDevice(prev);
    }
};

}  // namespace

// Databases and batches carry a process-unique id: a new object can reuse a
// freed one's address, so reuse checks and graph keys compare ids, never
// pointers.
static std::atomic<uint64_t> g_next_object_id{1};

// Groups are searched in launch classes: one hit mode and one shared-table
// size per launch, so a long query's large table does not cut the occupancy
// of every other group in its batch.
struct LaunchClass {
    int mode;        // 0 chunk mode, 1 offset mode; + 2 for groups with global tables
    int smem_diag;   // per-warp 16-bit table entries (small for the global class)
    int first;       // groups [first, first + count) of the batch's group list
    int count;
    int cell;        // bytes of a diagonal cell in byte_kernel (0: these groups cannot use it)
    int table_len;   // its cells per warp
    bool wide;       // its groups may have cells of kByteWide entries or more
};
// byte_kernel's part of a class.
struct LaunchShape {
    int byte_threads;   // CTA and grid (0: not used)
    int byte_blocks;
    int n_long;         // subjects left to wordfinder_kernel: the longest n_long
};
// A launch of wordfinder_kernel: groups [first, first + count) of the batch's
// group list against the longest n_subj subjects.
struct GeneralLaunch {
    int mode, smem_diag;
    int first, count;
    int32_t n_subj, tile;   // subjects, of them per tile
    int64_t tiles;
    int threads, blocks;
    int team;               // groups per tile (warps that share each subject)
};
struct SearchPlan {
    std::vector<LaunchShape> shapes;   // one per launch class of the batch
    std::vector<GeneralLaunch> general;
    bool beside = false;               // both kernels have a part, at the same time
    int lanes = 1;                     // streams that byte_kernel's launches are spread over
    int sides() const { return lanes - 1 + beside; }
};
constexpr int kMaxLaunchClasses = 64;

// What a search keeps on the host side beside its device buffers: events, the
// pinned copy of its counters, streams for launches side by side.  Making and freeing them took 250 us of a
// small search, so a database keeps a few for its next searches.
struct HostKit {
    cudaEvent_t ev[3] = {nullptr, nullptr, nullptr};
    // for work beside the caller's stream, with the events around it: made when
    // first needed
    static constexpr int kSides = 3;
    cudaStream_t side[kSides] = {nullptr, nullptr, nullptr};
    cudaEvent_t fork = nullptr, join[kSides] = {nullptr, nullptr, nullptr};
    unsigned long long *counters = nullptr;
    size_t n = 0;                 // counters it has room for
};
class KitPool {
  public:
    explicit KitPool(int device) : device_(device) {}
    ~KitPool() {
        DeviceScope ds(device_);
        for (HostKit &k : idle_)
            drop(k);
        if (upload_)
            cudaStreamDestroy(upload_);
    }
    // A stream for copies that must not wait for anybody's kernels.
    cudaError_t upload_stream(cudaStream_t *out) {
        std::lock_guard<std::mutex> lock(mu_);
        cudaError_t e = upload_ ? cudaSuccess : cudaStreamCreateWithFlags(&upload_, cudaStreamNonBlocking);
        *out = upload_;
        return e;
    }
    // A kit with room for n counters.
    cudaError_t take(size_t n, HostKit *out) {
        {
            std::lock_guard<std::mutex> lock(mu_);
            if (!idle_.empty()) {
                *out = idle_.back();
                idle_.pop_back();
            }
        }
        cudaError_t e = cudaSuccess;
        for (cudaEvent_t &ev : out->ev)
            if (e == cudaSuccess && !ev)
                e = cudaEventCreate(&ev);
        if (e == cudaSuccess && out->n < n) {
            cudaFreeHost(out->counters);
            out->counters = nullptr;
            out->n = 0;
            n = std::max<size_t>(n, 1024);
            e = cudaMallocHost((void **)&out->counters, n * sizeof(unsigned long long));
            if (e == cudaSuccess)
                out->n = n;
        }
        if (e != cudaSuccess) {
            cudaGetLastError();
            drop(*out);
        }
        return e;
    }
    // The kit's first n side streams and their events.
    static cudaError_t add_sides(HostKit *k, int n) {
        cudaError_t e = cudaSuccess;
        for (int i = 0; i < n; ++i) {
            if (e == cudaSuccess && !k->side[i])
                e = cudaStreamCreateWithFlags(&k->side[i], cudaStreamNonBlocking);
            for (cudaEvent_t *ev : {&k->fork, &k->join[i]})
                if (e == cudaSuccess && !*ev)
                    e = cudaEventCreateWithFlags(ev, cudaEventDisableTiming);
        }
        return e;
    }
    // Nothing on the side streams still runs.
    static void wait_sides(const HostKit &k) {
        for (cudaStream_t st : k.side)
            if (st)
                cudaStreamSynchronize(st);
    }
    // Give back a kit that no GPU work still uses.
    void give(HostKit &k) {
        {
            std::lock_guard<std::mutex> lock(mu_);
            if (k.n > 0 && k.n <= kMost && idle_.size() < kKept) {
                idle_.push_back(k);
                k = HostKit();
                return;
            }
        }
        drop(k);
    }

  private:
    static constexpr size_t kKept = 4, kMost = 1 << 17;   // kits, and counters of one (1 MiB)
    static void drop(HostKit &k) {
        for (cudaEvent_t &ev : k.ev)
            if (ev)
                cudaEventDestroy(ev);
        if (k.fork)
            cudaEventDestroy(k.fork);
        for (int i = 0; i < HostKit::kSides; ++i) {
            if (k.join[i])
                cudaEventDestroy(k.join[i]);
            if (k.side[i])
                cudaStreamDestroy(k.side[i]);
        }
        if (k.counters)
            cudaFreeHost(k.counters);
        k = HostKit();
    }
    int device_;
    std::mutex mu_;
    std::vector<HostKit> idle_;
    cudaStream_t upload_ = nullptr;
};

struct hbg_db {
    uint64_t id = g_next_object_id++;
    int device = 0;
    int32_t n = 0;
    int64_t n_res = 0;
    int64_t letters_len = 0;
    int32_t max_len = 0;
    std::vector<int32_t> sched_len;   // subject lengths in scheduling order (descending)
    std::shared_ptr<KitPool> kits;    // also held by the database's results
    uint8_t *d_arena = nullptr;       // one block that holds all of the following
    uint8_t *d_letters = nullptr;
    int64_t *d_off = nullptr;
    int32_t *d_len = nullptr;
    int32_t *d_order = nullptr;
    unsigned long long *d_hist = nullptr;
    int64_t bytes = 0;
};

// The device's build of a batch's tables: it runs on the stream of the batch's
// first search, which therefore waits for nothing on the host; searches on other
// streams wait for `done`.  Its scratch goes back when a search that came after
// it has ended, or with the batch.
struct TableBuild {
    explicit TableBuild(int dev) : device(dev) {}
    ~TableBuild() {
        if (done) {
            DeviceScope ds(device);
            cudaEventDestroy(done);
        }
    }
    void ended() {
        DeviceScope ds(device);
        std::lock_guard<std::mutex> lock(mu);
        dfree_idle(d_counts);
        over = true;
    }
    const int device;
    cudaEvent_t done = nullptr;
    uint32_t *d_counts = nullptr;
    std::atomic<bool> over{false};

  private:
    std::mutex mu;
};

struct hbg_batch {
    uint64_t id = g_next_object_id++;
    hbg::HostBatch host;
    int device = -1;
    uint8_t *d_arena = nullptr;        // one block that holds all of the following
    HbgGroup *d_groups = nullptr;
    HbgContext *d_ctx = nullptr;
    HbgQueryDesc *d_queries = nullptr;
    uint8_t *d_letters = nullptr;
    int32_t *d_ctx_of = nullptr;
    uint32_t *d_cells = nullptr;
    uint16_t *d_entries = nullptr;
    uint32_t *d_pv = nullptr;
    uint16_t *d_qcells = nullptr;
    int32_t *d_group_list = nullptr;   // groups ordered by launch class
    uint32_t *d_packed = nullptr;      // cells of byte_kernel
    std::shared_ptr<TableBuild> build; // running, or done
    std::vector<LaunchClass> classes;
    std::mutex tables_mu;              // host tables and entry counts are made when first asked for
    bool caller_tables = false;        // the tables are the caller's (in `host`)
    bool repeated_entries = false;     // a caller's lookup table lists an offset twice in a cell
    bool tuned = false;                // the caller chose tiles or table placement (hbg_batch_tune)
    int32_t tile_subjects = 0;   // 0 = automatic (hbg_batch_tune)
    int64_t tile_bytes = 0;      // > 0: tiles of about this many subject letters (hbg_batch_schedule)
    int32_t team = 1;            // groups searched together per pass over a subject (hbg_batch_schedule)
};

struct hbg_result {
    hbg_db *db = nullptr;
    hbg_batch *batch = nullptr;
    hbg_gpu_options opt{};
    cudaStream_t stream = nullptr;
    int device = 0;
    int64_t cap = 0;
    SearchPlan plan;
    hbg_gpu_options plan_opt{};      // options it was made for
    // device
    hbg_hsp *d_raw = nullptr, *d_sorted = nullptr;
    unsigned long long *d_counters = nullptr;  // [0]=hsp count, then per query ext, kept, hits; per group
                                               // hits; per query first, end of its HSPs, subjects passed; per
                                               // group subjects taken; the ordering's barrier and error
    unsigned int *d_tile = nullptr;
    uint32_t *d_gdiag = nullptr;
    int64_t gdiag_entries = 0;
    uint16_t *d_side = nullptr;   // flag ends of byte_kernel
    int64_t side_entries = 0;
    int32_t gdiag_len = 0;   // entries per (CTA, warp) slice of the global diagonal tables
    uint64_t *d_keys = nullptr;
    uint32_t *d_vals = nullptr;
    uint32_t *d_hist = nullptr;
    int64_t sort_cap = 0;
    // host
    std::shared_ptr<KitPool> kits;
    std::shared_ptr<TableBuild> build;         // of the batch last searched
    HostKit kit;                               // events, pinned counters
    size_t n_counters = 0;
    size_t nq = 0, ng = 0;                     // queries and groups of the batch, which may go before its result
    std::vector<hbg_query_stats> stats;
    std::vector<int64_t> q_first, q_count;
    int64_t n_hsps = 0;
    bool launched = false, synced = false, done = false;
    float wf_ms = 0.f, ord_ms = 0.f;
    int32_t launches = 0;   // kernels per search
    int64_t launch_count = 0;
    cudaGraphExec_t graph_exec = nullptr;
    uint64_t db_id = 0, batch_id = 0;   // what the buffers were last prepared for
    long long graph_key[5] = {0, 0, 0, 0, 0};
};

namespace {

void free_batch_device(hbg_batch *b) {
    // searches of this batch may run on any stream: wait for the device (as
    // cudaFree would), then keep the buffers for reuse
    if (wait_device() == cudaSuccess) {
        dfree_idle(b->d_arena);
    } else {                                   // a caller captures: cudaFree waits by itself
        dfree(b->d_arena);
        if (b->build)
            dfree(b->build->d_counts);
    }
    if (b->build)
        b->build->ended();
    b->build.reset();
}

int upload_batch_buffers(hbg_batch *b, const hbg_db *db, cudaStream_t stream);

// Run host code that allocates or starts threads: what it throws must not leave
// a C entry point.
template <typename F>
int guarded(F &&f) {
    try {
        return f();
    } catch (const std::exception &e) {
        return fail(HBG_ERR_NOMEM, std::string("host allocation: ") + e.what());
    }
}

// A batch on the device: one block, 256-byte aligned parts in it.  First what
// is copied there (`upload` bytes; with a caller's own tables, these too), then
// what the device makes.
struct BatchLayout {
    std::vector<hbg::TableSegment> segs;       // of the table build
    int32_t slice = 0;                         // most of them built at a time
    size_t groups = 0, ctx = 0, queries = 0, letters = 0, ctx_of = 0, list = 0, segments = 0, cells = 0, pv = 0, qcells = 0,
           entries = 0, packed = 0;
    size_t upload = 0, total = 0;

    size_t scratch() const { return (size_t)slice * HBG_NUM_CELLS * sizeof(uint32_t); }
};

// Segments of the table build that are in hand at a time: 128 KiB of scratch
// each.  A slice is whole groups, and a group of 65,000 letters has at most 191
// segments.
constexpr int32_t kSliceSegments = 512;

// The groups of the slice that starts with group g, and its segments.
int32_t slice_end(const hbg::HostBatch &h, int32_t g, int32_t *n_segs) {
    int32_t n = 0;
    for (; g < (int32_t)h.groups.size() && (n == 0 || n + h.groups[g].n_segs <= kSliceSegments); ++g)
        n += h.groups[g].n_segs;
    *n_segs = n;
    return g;
}

// Counts the batch's entries, cuts it into segments and lays it out (the groups
// learn their segments and the place of their entries).  Under tables_mu.
BatchLayout lay_out(hbg_batch *b) {
    hbg::HostBatch &h = b->host;
    BatchLayout L;
    const size_t ng = h.groups.size(), nq = h.queries.size();
    const size_t n_entries = (size_t)hbg::count_entries(&h);
    int64_t base = 0;
    for (size_t g = 0; g < ng; ++g) {
        HbgGroup &G = h.groups[g];
        G.entry_base = base;
        base += G.n_entries;
        G.seg_base = (int32_t)L.segs.size();
        for (int32_t q = G.first_query; q < G.first_query + G.n_queries; ++q) {
            const int32_t at = h.queries[q].start, end = at + h.queries[q].len - HBG_WORD_SIZE + 1;
            for (int32_t p = at; p == at || p < end; p += hbg::kTableSegment)
                L.segs.push_back({(int32_t)g, q, p, std::min(end, p + hbg::kTableSegment)});
        }
        G.n_segs = (int32_t)L.segs.size() - G.seg_base;
    }
    size_t at = 0;
    auto place = [&](size_t bytes, size_t before = 0, size_t after = 0) {
        const size_t p = at + before;
        at = (p + bytes + after + 255) / 256 * 256;
        return p;
    };
    auto tables = [&] {
        L.cells = place(ng * HBG_CELL_STRIDE * sizeof(uint32_t));
        L.pv = place(ng * HBG_PV_WORDS * sizeof(uint32_t));
        L.qcells = place(nq * HBG_NUM_CELLS * sizeof(uint16_t));
        L.entries = place(n_entries * sizeof(uint16_t), 0, 128);   // byte_kernel reads up to 31 entries past a cell
    };
    L.groups = place(ng * sizeof(HbgGroup));
    L.ctx = place(h.contexts.size() * sizeof(HbgContext));
    L.queries = place(nq * sizeof(HbgQueryDesc));
    L.letters = place(h.letters.size(), kFrontPad, 64);            // extensions read whole blocks
    L.ctx_of = place(h.ctx_of.size() * sizeof(int32_t), 0, 64);
    L.list = place(ng * sizeof(int32_t));
    if (b->caller_tables) {
        L.segs.clear();
        tables();
    } else {
        L.segments = place(L.segs.size() * sizeof(hbg::TableSegment));
        for (int32_t g = 0, n; g < (int32_t)ng;) {
            g = slice_end(h, g, &n);
            L.slice = std::max(L.slice, n);
        }
    }
    L.upload = at;
    if (!b->caller_tables)
        tables();
    L.packed = place(ng * HBG_NUM_CELLS * sizeof(uint32_t));
    L.total = at;
    return L;
}

// Host tables, built when a caller first asks for them.
void ensure_tables(const hbg_batch *batch) {
    hbg_batch *b = const_cast<hbg_batch *>(batch);
    std::lock_guard<std::mutex> lock(b->tables_mu);
    if (b->host.cells.empty())
        hbg::build_tables(&b->host);
}

// Upload at the first search; a failed upload gives back what it allocated,
// so the batch can be searched again later.
// Searches on `stream` come after the batch's table build.
int after_build(const hbg_batch *b, cudaStream_t stream) {
    if (!b->build || b->build->over)
        return HBG_OK;
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    CU(cudaStreamIsCapturing(stream, &capture));
    if (capture == cudaStreamCaptureStatusNone) {
        CU(cudaStreamWaitEvent(stream, b->build->done, 0));
    } else {                           // an event from outside the capture: wait here
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        CU(cudaThreadExchangeStreamCaptureMode(&mode));
        const cudaError_t e = cudaEventSynchronize(b->build->done);
        cudaThreadExchangeStreamCaptureMode(&mode);
        CU(e);
    }
    return HBG_OK;
}

int upload_batch(hbg_batch *b, const hbg_db *db, cudaStream_t stream) {
    const int device = db->device;
    if (b->device == device)
        return after_build(b, stream);
    if (b->device >= 0)
        return fail(HBG_ERR_STATE, "batch already resident on another device");
    DeviceScope ds(device);
    const int rc = guarded([&] { return upload_batch_buffers(b, db, stream); });
    if (rc != HBG_OK) {
        free_batch_device(b);
        b->device = -1;
    }
    return rc;
}

// Longest diagonal tables byte_kernel keeps in 16-bit cells: 4096 entries leave
// room for 22 warps per SM (a 4056-letter query against 400,000 subjects: 9.2
// ms; 8-bit cells, 24 warps: 10.3 ms, the sweeps cut its rounds of extensions
// short).  Longer tables take 8-bit cells (8152 letters against
// 200,000 subjects: 9.5 ms, 12.2 ms with 16-bit cells and 12 warps).
constexpr int kByteTable16 = 4096;
// Fewest warps per SM it is used with.  Against 20,000 subjects, ms here and
// with wordfinder_kernel: 20,000 letters (10 warps) 3.7 / 8.1, 35,000 (6 warps)
// 9.9 / 18.0, 50,000 (4) 20.6 / 32.3, 64,900 (3, the longest) 35.2 / 45.4.
constexpr int kByteMinWarps = 2;
// Fewest tiles, per CTA of a wave, with which a launch class of wordfinder_kernel
// is launched by itself: what automatic tiles aim at.
constexpr int kFewTiles = 8;

// Bytes of a diagonal cell in byte_kernel for a group, 0 when it cannot take
// the group: its window, table or entry count do not fit, or the caller's own
// table lists an offset twice in a cell (two hits in one place).
int byte_cell(const hbg_batch *b, int32_t g) {
    const hbg::HostBatch &h = b->host;
    const HbgGroup &G = h.groups[g];
    if (h.window < hbg::kByteMinWindow || h.window > hbg::kByteMaxWindow || G.n_entries >= hbg::kByteMaxEntries ||
        b->repeated_entries)
        return 0;
    return G.diag_len <= kByteTable16 ? 2 : 1;
}

// The launch classes of a batch and its groups in class order.
int make_classes(const hbg_batch *b, std::vector<LaunchClass> *classes, std::vector<int32_t> *list) {
    const hbg::HostBatch &h = b->host;
    // launch classes: (mode, table size); groups with shared tables are
    // launched by table size, so a short query's warps reserve only the
    // shared memory its table needs (the rest is L1 for cells and entries:
    // one 350-aa query vs 10 M subjects 8 % faster than with 2048-entry
    // tables for every group); groups that byte_kernel can take by its table
    // and whether their cells may be wide, longest first.  With tiles of the
    // caller's (not byte_kernel's) all of a size stay in the order they came.
    const bool tiles = b->tile_subjects > 0 || b->tile_bytes > 0;
    std::vector<std::pair<std::array<int, 3>, int32_t>> keyed;
    for (int32_t g = 0; g < (int32_t)h.groups.size(); ++g) {
        const HbgGroup &G = h.groups[g];
        const int size = G.placement ? 64 : std::max<int>(64, G.diag_len);
        const int cell = byte_cell(b, g), wide = cell == 2 && G.max_cell >= hbg::kByteWide;
        keyed.push_back({{G.mode, size, cell && !tiles ? -(8 * std::max<int>(64, G.diag_len) + 4 * wide + cell) : 0}, g});
    }
    std::stable_sort(keyed.begin(), keyed.end(),
                     [](const auto &x, const auto &y) { return x.first < y.first; });
    list->clear();
    classes->clear();
    for (size_t i = 0; i < keyed.size(); ++i) {
        const bool global = h.groups[keyed[i].second].placement != 0;
        if (i == 0 || keyed[i].first != keyed[i - 1].first)
            classes->push_back(LaunchClass{keyed[i].first[0] + (global ? 2 : 0), keyed[i].first[1], (int)i, 0,
                                             -keyed[i].first[2] & 3, -keyed[i].first[2] / 8,
                                             (-keyed[i].first[2] & 4) != 0});
        LaunchClass &lc = classes->back();
        lc.count++;
        if (lc.cell == 1)              // the longest group's exact table
            lc.table_len = std::max(lc.count == 1 ? 0 : lc.table_len,
                                    hbg::byte_table_len(h.groups[keyed[i].second].glen + h.window));
        list->push_back(keyed[i].second);
    }
    if ((int)classes->size() > kMaxLaunchClasses)
        return fail(HBG_ERR_INVALID, "too many launch classes");
    return HBG_OK;
}

// The batch's letters go up on the database's upload stream, behind nothing but
// other such copies, and the host waits for the copy; the tables are built on the
// search's stream.  (Built on the upload stream, with the host waiting: 56 ms
// for a 300-letter query while a batch was searched on another stream, whose
// CTAs keep their SMs to the end; now 0.07.)
int upload_batch_buffers(hbg_batch *b, const hbg_db *db, cudaStream_t stream) {
    hbg::HostBatch &h = b->host;
    const size_t ng = h.groups.size();
    std::unique_lock<std::mutex> lock(b->tables_mu);
    const BatchLayout L = lay_out(b);
    std::vector<int32_t> list;
    const int rc = make_classes(b, &b->classes, &list);
    if (rc != HBG_OK)
        return rc;
    // one copy (ten of their own took 80 us)
    std::unique_ptr<uint8_t[]> stage(new (std::nothrow) uint8_t[L.upload]);
    if (!stage)
        return fail(HBG_ERR_NOMEM, "host allocation");
    size_t done = 0;
    auto put = [&](size_t at, const void *src, size_t bytes) {     // in ascending order; zeros between
        memset(stage.get() + done, 0, at - done);
        if (bytes)
            memcpy(stage.get() + at, src, bytes);
        done = at + bytes;
    };
    put(L.groups, h.groups.data(), ng * sizeof(HbgGroup));
    put(L.ctx, h.contexts.data(), h.contexts.size() * sizeof(HbgContext));
    put(L.queries, h.queries.data(), h.queries.size() * sizeof(HbgQueryDesc));
    put(L.letters, h.letters.data(), h.letters.size());
    put(L.ctx_of, h.ctx_of.data(), h.ctx_of.size() * sizeof(int32_t));
    put(L.list, list.data(), list.size() * sizeof(int32_t));
    if (b->caller_tables) {
        put(L.cells, h.cells.data(), h.cells.size() * sizeof(uint32_t));
        put(L.pv, h.pv.data(), h.pv.size() * sizeof(uint32_t));
        put(L.qcells, h.query_cells.data(), h.query_cells.size() * sizeof(uint16_t));
        put(L.entries, h.entries.data(), h.entries.size() * sizeof(uint16_t));
    } else {
        put(L.segments, L.segs.data(), L.segs.size() * sizeof(hbg::TableSegment));
    }
    put(L.upload, nullptr, 0);
    lock.unlock();
    CU(dalloc(&b->d_arena, L.total));
    b->d_groups = reinterpret_cast<HbgGroup *>(b->d_arena + L.groups);
    b->d_ctx = reinterpret_cast<HbgContext *>(b->d_arena + L.ctx);
    b->d_queries = reinterpret_cast<HbgQueryDesc *>(b->d_arena + L.queries);
    b->d_letters = b->d_arena + L.letters;
    b->d_ctx_of = reinterpret_cast<int32_t *>(b->d_arena + L.ctx_of);
    b->d_group_list = reinterpret_cast<int32_t *>(b->d_arena + L.list);
    b->d_cells = reinterpret_cast<uint32_t *>(b->d_arena + L.cells);
    b->d_pv = reinterpret_cast<uint32_t *>(b->d_arena + L.pv);
    b->d_qcells = reinterpret_cast<uint16_t *>(b->d_arena + L.qcells);
    b->d_entries = reinterpret_cast<uint16_t *>(b->d_arena + L.entries);
    b->d_packed = reinterpret_cast<uint32_t *>(b->d_arena + L.packed);
    b->build = std::make_shared<TableBuild>(db->device);
    TableBuild &build = *b->build;
    CU(cudaEventCreateWithFlags(&build.done, cudaEventDisableTiming));
    if (!b->caller_tables)
        CU(dalloc(&build.d_counts, L.scratch() / sizeof(uint32_t)));
    cudaStream_t up = nullptr;
    CU(db->kits->upload_stream(&up));
    CU(cudaMemcpyAsync(b->d_arena, stage.get(), L.upload, cudaMemcpyHostToDevice, up));
    CU(cudaStreamSynchronize(up));
    // a captured build would run with the graph only
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    CU(cudaStreamIsCapturing(stream, &capture));
    cudaStream_t st = capture == cudaStreamCaptureStatusNone ? stream : up;
    if (b->caller_tables) {
        CU(hbg::launch_pack_cells(b->d_cells, (int32_t)ng, b->d_packed, st));
    } else {
        hbg::TableArgs t{b->d_groups, reinterpret_cast<const hbg::TableSegment *>(b->d_arena + L.segments), 0, 0,
                         b->d_letters, b->d_ctx_of, h.threshold, b->d_cells, b->d_packed, b->d_pv, b->d_entries,
                         b->d_qcells, build.d_counts};
        for (int32_t g = 0, n; g < (int32_t)ng;) {
            const int32_t end = slice_end(h, g, &n);
            t.first_group = g;
            t.first_seg = h.groups[g].seg_base;
            CU(hbg::launch_tables(t, end - g, n, st));
            g = end;
        }
    }
    CU(cudaEventRecord(build.done, st));
    if (st == up)
        CU(cudaStreamSynchronize(up));
    b->device = db->device;
    return HBG_OK;
}

// Length of the per-warp global diagonal table: groups too long for shared
// memory, and subjects whose offsets do not fit the 16-bit shared cells
// (window + length > 32767), use it.
int32_t global_diag_len(const hbg::HostBatch &h, const hbg_db *db) {
    int32_t len = h.max_diag_len;
    if (db->max_len + h.window > 0x7fff)
        len = std::max<int32_t>(len, h.smem_diag_len);
    return len;
}

// Subjects per work tile of one launch class: the batch's tuned value, else
// up to 128, fewer when the class has too little work to give every CTA about
// eight tiles (small databases and single queries would otherwise leave most
// SMs idle).
int32_t class_tile_subjects(const hbg_batch *b, int32_t n_subj, const hbg_db *db, int count, int blocks) {
    if (b->tile_subjects > 0)
        return b->tile_subjects;
    if (b->tile_bytes > 0) {                  // subjects of the database's mean length
        const int64_t mean = std::max<int64_t>(1, db->n_res / std::max<int32_t>(1, db->n));
        return (int32_t)std::max<int64_t>(1, std::min<int64_t>(1 << 20, b->tile_bytes / mean));
    }
    const int64_t want = (int64_t)n_subj * count / (8 * (int64_t)std::max(blocks, 1));
    return (int32_t)std::max<int64_t>(8, std::min<int64_t>(128, want));
}

// Which classes byte_kernel takes, with which CTA, and the subjects that stay
// with wordfinder_kernel: those whose positions do not fit its cells.
void plan_bytes(const hbg_batch *b, const std::vector<LaunchClass> &classes, const hbg_db *db, const hbg_gpu_options &o,
                int optin, int sms, std::vector<LaunchShape> *shapes) {
    shapes->assign(classes.size(), LaunchShape{0, 0, 0});
    hbg_gpu_options std_opt;
    hbg_default_gpu_options(&std_opt);
    if (o.num_blocksx != std_opt.num_blocksx || o.num_threadsx != std_opt.num_threadsx || b->tuned || b->team > 1 ||
        b->tile_bytes > 0)
        return;                                  // the caller chose a launch shape of wordfinder_kernel
    for (size_t c = 0; c < classes.size(); ++c) {
        const LaunchClass &lc = classes[c];
        LaunchShape &sh = (*shapes)[c];
        if (!lc.cell || (lc.mode & 1))
            continue;
        // one CTA per SM, with as many warps as their tables leave room for
        int t = hbg::kByteThreads;
        while (t > 0 && hbg::byte_smem_bytes(lc.cell, t, lc.table_len) > (size_t)optin)
            t -= 32;
        if (t < 32 * kByteMinWarps)
            continue;
        // a group's subjects go to the warps of one CTA: with fewer subjects than
        // warps, groups in great number are better off with wordfinder_kernel,
        // whose CTAs take several at a time.  Here / there, ms: 1000 groups of 300
        // letters against 12 subjects 0.227 / 0.169, 25 subjects 0.223 / 0.236;
        // 1500 of 4000 letters 1.64 / 1.32, 1.62 / 1.87; 300 groups of 1500 letters
        // against 12 subjects 0.143 / 0.162.
        if (db->n < t / 32 && lc.count > 4 * sms)
            continue;
        const int32_t cut = lc.cell == 2 ? 0x7ffe - b->host.window : 0xffff;
        const auto &L = db->sched_len;
        sh.n_long = (int)(std::partition_point(L.begin(), L.end(), [&](int32_t l) { return l > cut; }) - L.begin());
        sh.byte_threads = t;
        sh.byte_blocks = sms;
    }
}

// CTA size and CTAs per SM of wordfinder_kernel: the CTA is halved until its
// per-warp tables fit the shared-memory carve-out.
int general_shape(const hbg_batch *b, const hbg_gpu_options &o, int optin, int mode, int smem_diag, int *threads,
                  int *per_sm) {
    // num_threadsx is the largest CTA size: take the size (halving down to 64)
    // that keeps the most warps resident per SM -- large diagonal tables fill
    // shared memory, and smaller CTAs pack it better
    // with several groups per pass (team > 1) the CTA keeps at least one
    // warp per group
    int best_warps = -1;
    *threads = 0;
    for (int t = o.num_threadsx; t >= 32; t = t > 64 ? ((t / 2) + 31) / 32 * 32 : 0) {
        const int team = std::min(b->team, t / 32);
        if (team < b->team && *threads > 0)
            break;
        if (hbg::wordfinder_smem_bytes(t, smem_diag, team) > (size_t)optin)
            continue;
        int per = 0;
        if (hbg::wordfinder_occupancy(mode, t, smem_diag, team, &per) != cudaSuccess || per < 1)
            per = 1;
        if (per * (t / 32) > best_warps) {
            *threads = t;
            *per_sm = per;
            best_warps = per * (t / 32);
        }
        if (o.num_blocksx > 0)
            break;                 // a fixed grid keeps the caller's CTA size when it fits
    }
    return *threads > 0 ? HBG_OK : fail(HBG_ERR_TOO_LONG, "group diagonal tables exceed shared memory");
}

// The launches of a search.  Neighbouring classes that wordfinder_kernel does not
// tell apart share a launch, longest groups first, when one of them alone has too
// few tiles for its CTAs, or when the CTAs are small (few warps work on the last
// tiles).  ms, together and apart: three groups of 11,000 to 39,000 letters against
// 81 subjects, three to a pass, 5.0 / 9.0; 40 groups of 1100 to 4100 letters against
// 217 subjects, global tables, 1.32 / 2.86; 128 threads, five groups of 2500 to
// 40,000 letters against 20,000 subjects, 36.9 / 44.2.  With tiles enough: the last
// in offset mode 48 / 27.
// The grid is one wave (or the caller's num_blocksx), at most a CTA per tile.
int plan_search(const hbg_batch *b, const std::vector<LaunchClass> &classes, const hbg_db *db, const hbg_gpu_options &o,
                SearchPlan *plan) {
    int optin = 0, sms = 1;
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, db->device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, db->device);
    plan_bytes(b, classes, db, o, optin, sms, &plan->shapes);
    plan->general.clear();
    hbg_gpu_options std_opt;
    hbg_default_gpu_options(&std_opt);
    auto subjects = [&](size_t c) { return plan->shapes[c].byte_threads > 0 ? plan->shapes[c].n_long : db->n; };
    int most = 0;                      // CTAs that search long subjects beside byte_kernel
    bool some = false;
    for (size_t c = 0, e; c < classes.size(); c = e) {
        GeneralLaunch l{classes[c].mode, classes[c].smem_diag, classes[c].first, 0, subjects(c), 0, 0, 0, 0, 1};
        for (e = c; e < classes.size() && classes[e].mode == l.mode && classes[e].smem_diag == l.smem_diag &&
                    subjects(e) == l.n_subj; ++e)
            l.count += classes[e].count;
        some = some || plan->shapes[c].byte_threads > 0;
        if (l.n_subj == 0)
            continue;
        int per = 1;
        const int rc = general_shape(b, o, optin, l.mode, l.smem_diag, &l.threads, &per);
        if (rc != HBG_OK)
            return rc;
        l.team = std::min(b->team, l.threads / 32);
        const int wave = o.num_blocksx > 0 ? o.num_blocksx : sms * per;
        auto size = [&](GeneralLaunch *x) {
            x->tile = class_tile_subjects(b, x->n_subj, db, x->count, wave);
            x->tiles = (int64_t)((x->n_subj + x->tile - 1) / x->tile) * ((x->count + x->team - 1) / x->team);
            x->blocks = o.num_blocksx > 0 ? wave : (int)std::min<int64_t>(wave, x->tiles);
        };
        bool together = o.num_threadsx < std_opt.num_threadsx;
        for (size_t k = c; k < e; ++k) {
            GeneralLaunch x = l;
            x.count = classes[k].count;
            size(&x);
            together = together || x.tiles < kFewTiles * (int64_t)wave;
        }
        for (size_t k = c; k < e; ++k) {
            GeneralLaunch x = l;
            if (!together) {
                x.first = classes[k].first;
                x.count = classes[k].count;
            }
            size(&x);
            if (plan->shapes[c].byte_threads > 0)
                most = std::max(most, x.blocks);
            plan->general.push_back(x);
            if (together)
                break;
        }
    }
    // the long subjects are searched beside byte_kernel, which leaves SMs for
    // them (its CTAs stay to the end and fill theirs)
    plan->beside = some && most > 0;
    // byte_kernel's launches side by side hide the walk of the longest subjects at
    // the end of one.  Where the warps' shares of all groups together are more than
    // five such walks they are better off in turn, each with all SMs: 14 nucleotide
    // queries against 175,000 subjects 18.03 ms side by side, 17.79 in turn (a share
    // of some 40 walks); 14 proteins in groups of 1000 letters and more against
    // 22,000 subjects 1.086, 1.049 (eight)
    int n = 0;
    double share = 0;                  // letters of a warp
    for (size_t c = 0; c < classes.size(); ++c) {
        const LaunchShape &sh = plan->shapes[c];
        if (sh.byte_threads == 0)
            continue;
        ++n;
        share += (double)db->n_res * classes[c].count / (sh.byte_blocks * (sh.byte_threads / 32));
    }
    const bool tails = share < 5.0 * db->max_len;
    // (one beside wordfinder_kernel's: a second would take the SMs left for it)
    plan->lanes = tails && !plan->beside ? std::max(1, std::min(n, HostKit::kSides + 1)) : 1;
    for (LaunchShape &sh : plan->shapes)
        if (sh.byte_threads > 0)
            sh.byte_blocks = std::max(1, sh.byte_blocks - std::min(most, sms / 8));
    return HBG_OK;
}

void drop_graph(hbg_result *r) {
    if (r->graph_exec)
        cudaGraphExecDestroy(r->graph_exec);
    r->graph_exec = nullptr;
}

void free_result_device(hbg_result *r) {
    if (r->graph_exec)
        cudaGraphExecDestroy(r->graph_exec);
    r->graph_exec = nullptr;
    if (r->launched && !r->synced) {
        cudaStreamSynchronize(r->stream);    // nothing of this search may still run
        r->build->ended();
    }
    dfree_idle(r->d_raw);
    dfree_idle(r->d_sorted);
    dfree_idle(r->d_counters);
    dfree_idle(r->d_tile);
    dfree_idle(r->d_gdiag);
    dfree_idle(r->d_side);
    dfree_idle(r->d_keys);
    dfree_idle(r->d_vals);
    dfree_idle(r->d_hist);
    if (r->kits)
        r->kits->give(r->kit);
}

// Entries of the scratch that the launches of a search share: global diagonal
// tables of wordfinder_kernel, flag ends of byte_kernel.
int64_t gdiag_need(const hbg::HostBatch &h, const hbg_db *db, const SearchPlan &plan) {
    int64_t warps = 0;
    for (const GeneralLaunch &l : plan.general)
        warps = std::max<int64_t>(warps, (int64_t)l.blocks * (l.threads / 32));
    return warps * global_diag_len(h, db);
}
int64_t side_need(const LaunchClass &lc, const LaunchShape &sh) {
    return sh.byte_threads > 0 && lc.cell == 1 ? (int64_t)sh.byte_blocks * (sh.byte_threads / 32) * lc.table_len : 0;
}
int64_t side_need(const std::vector<LaunchClass> &classes, const SearchPlan &plan) {
    int64_t side = 0;
    for (size_t c = 0; c < classes.size(); ++c)    // launches run side by side
        side += side_need(classes[c], plan.shapes[c]);
    return side;
}
size_t counters_need(const hbg::HostBatch &h) { return 3 + 6 * h.queries.size() + 2 * h.groups.size(); }

// Allocate (or grow) the result's device buffers for capacity cap.
int prepare_result(hbg_result *r, int64_t cap) {
    const hbg::HostBatch &h = r->batch->host;
    if (!r->d_tile)
        CU(dalloc(&r->d_tile, kMaxLaunchClasses));
    // a failed allocation below leaves the recorded size at 0, so the next
    // search allocates again instead of using a missing buffer
    if (r->n_counters < counters_need(h)) {   // first use, or a larger batch
        drop_graph(r);
        dfree(r->d_counters);
        r->kits->give(r->kit);
        r->n_counters = 0;
        CU(dalloc(&r->d_counters, counters_need(h)));
        CU(r->kits->take(counters_need(h), &r->kit));
        r->n_counters = counters_need(h);
    }
    r->gdiag_len = global_diag_len(h, r->db);
    const int64_t gdiag = gdiag_need(h, r->db, r->plan), side = side_need(r->batch->classes, r->plan);
    if (gdiag > r->gdiag_entries) {
        drop_graph(r);
        dfree(r->d_gdiag);
        r->gdiag_entries = 0;
        CU(dalloc(&r->d_gdiag, (size_t)gdiag));
        r->gdiag_entries = gdiag;
    }
    CU(KitPool::add_sides(&r->kit, r->plan.sides()));
    if (side > r->side_entries) {
        drop_graph(r);
        dfree(r->d_side);
        r->side_entries = 0;
        CU(dalloc(&r->d_side, (size_t)side));
        r->side_entries = side;
    }
    if (cap > r->cap) {
        drop_graph(r);
        r->cap = 0;
        dfree(r->d_raw);
        dfree(r->d_sorted);
        dfree(r->d_keys);
        dfree(r->d_vals);
        dfree(r->d_hist);
        CU(dalloc(&r->d_raw, (size_t)cap));
        CU(dalloc(&r->d_sorted, (size_t)cap));
        CU(dalloc(&r->d_keys, (size_t)cap * 2));
        CU(dalloc(&r->d_vals, (size_t)cap * 2));
        CU(dalloc(&r->d_hist, (size_t)256 * hbg::kOrderMaxGrid));
        r->cap = cap;
    }
    return HBG_OK;
}

// HSPs a search has room for when the caller does not say: 2e-7 per letter of
// the queries and of the database (random proteins give 1.6e-7 at the default
// cutoff), at least one per subject and 1 Mi.  A search that overflows runs
// twice: 64 queries against 500,000 subjects find 1.4 M HSPs, 302 ms from host
// queries to host HSPs with room for 1 Mi, 154 ms with this.
int64_t default_capacity(const hbg_db *db, const hbg_batch *b) {
    double letters = 0;
    for (const HbgQueryDesc &q : b->host.queries)
        letters += q.len;
    return std::max<int64_t>(std::max<int64_t>(1 << 20, (int64_t)db->n), (int64_t)(2e-7 * letters * (double)db->n_res));
}

// byte_kernel's view of a database and of one launch class of a batch; the
// caller adds counters, scratch and outputs.
hbg::ByteArgs byte_args(const hbg_db *db, const hbg_batch *b, const LaunchClass &lc, const LaunchShape &sh) {
    hbg::ByteArgs t;
    memset(&t, 0, sizeof(t));
    t.db = db->d_letters;
    t.db_off = db->d_off;
    t.db_len = db->d_len;
    t.order = db->d_order;
    t.sub_lo = sh.n_long;
    t.n_subj = db->n - sh.n_long;
    t.groups = b->d_groups;
    t.group_list = b->d_group_list + lc.first;
    t.n_list = lc.count;
    t.packed = b->d_packed;
    t.cells = b->d_cells;
    t.entries = b->d_entries;
    t.pv = b->d_pv;
    t.letters = b->d_letters;
    t.ctx_of = b->d_ctx_of;
    t.contexts = b->d_ctx;
    t.queries = b->d_queries;
    t.window = b->host.window;
    t.table_len = lc.table_len;
    // the first subjects are the longest: a take of them is at most an eighth
    // of a warp's share of a group's letters (with more groups than CTAs each
    // has a CTA to itself; taken as the share of all letters, 5000 one-query
    // groups against 400 subjects had takes of 12 and took 14.6 ms, now 8.2)
    const int64_t warps = (int64_t)sh.byte_blocks * (sh.byte_threads / 32), groups = std::min(lc.count, sh.byte_blocks);
    t.chunk = (int32_t)std::max<int64_t>(
        1, std::min<int64_t>(16, db->n_res * groups / (8 * warps * std::max<int32_t>(1, db->max_len))));
    return t;
}

// The word finder's launches: byte_kernel for each class it takes, then
// wordfinder_kernel for the rest.  `a` holds scratch and outputs (tile_counter: one
// counter per launch), `next` a subject counter per group, both zeroed.  The
// caller has run wordfinder_configure and byte_configure (not stream operations).
//
// With `kit`, launches run side by side on its streams: at the end of one, a few
// warps walk its last or longest subjects while the next could have the other SMs.
// (Without, one after another, byte_kernel's first: `next` may be a.g_hits, which
// it must find zeroed.)  ms, side by side and in turn: groups of 100, 300, 900, 2000
// and 4000 letters against 20,000 subjects 1.14 / 1.29; three of 5000 to 34,000
// against 17 subjects and one of 33,000 letters 102 / 202 (175 in one launch of
// wordfinder_kernel).  Short tables first: where the long ones' CTAs get half of
// the SMs at first, their last group starts late with its longest subject (100 to
// 1500 letters in two launches against 200,000 subjects 14.13 / 14.05; 14.06 so).
// Subjects too long for byte_kernel's cells, a warp each: one query of 350 letters
// against 300,000 subjects 1.30 ms, with one subject of 35,000 letters besides 1.60,
// after the others 2.85; 16 queries of 500 letters against 100,000 4.67, 11.0, 15.8.
int launch_finders(const hbg_db *db, const hbg_batch *b, const SearchPlan &plan, hbg::WordFinderArgs a,
                   unsigned long long *next, uint16_t *side, const HostKit *kit, cudaStream_t st, int *launches) {
    if (db->n == 0)
        return HBG_OK;
    const int sides = kit ? plan.sides() : 0;
    if (sides > 0)
        CU(cudaEventRecord(kit->fork, st));
    for (int i = 0; i < sides; ++i)
        CU(cudaStreamWaitEvent(kit->side[i], kit->fork, 0));
    int lane = 0;                      // of byte_kernel's next launch; 0: st
    for (size_t c = b->classes.size(); c-- > 0;) {
        const LaunchClass &lc = b->classes[c];
        const LaunchShape &sh = plan.shapes[c];
        if (sh.byte_threads == 0 || sh.n_long >= db->n)
            continue;
        hbg::ByteArgs t = byte_args(db, b, lc, sh);
        t.next = next;
        t.side = side;
        if (side)
            side += side_need(lc, sh);
        t.hsps = a.hsps;
        t.hsp_count = a.hsp_count;
        t.hsp_cap = a.hsp_cap;
        t.q_extended = a.q_extended;
        t.q_kept = a.q_kept;
        CU(hbg::launch_byte(t, lc.cell, lc.wide, sh.byte_blocks, sh.byte_threads, lane == 0 ? st : kit->side[lane - 1]));
        lane = sides > 0 ? (lane + 1) % plan.lanes : 0;
        ++*launches;
    }
    cudaStream_t other = kit && plan.beside ? kit->side[sides - 1] : st;   // wordfinder_kernel's, in turn: they share scratch
    for (const GeneralLaunch &l : plan.general) {
        a.n_subj = l.n_subj;
        a.tile_subjects = l.tile;
        a.tiles_per_group = (l.n_subj + l.tile - 1) / l.tile;
        a.n_tiles = l.tiles;
        a.team = l.team;
        a.n_list = l.count;
        a.group_list = b->d_group_list + l.first;
        a.smem_diag = l.smem_diag;
        CU(hbg::launch_wordfinder(a, l.mode, l.blocks, l.threads, other));
        ++a.tile_counter;
        ++*launches;
    }
    for (int i = 0; i < sides; ++i) {
        CU(cudaEventRecord(kit->join[i], kit->side[i]));
        CU(cudaStreamWaitEvent(st, kit->join[i], 0));
    }
    return HBG_OK;
}

// Enqueue one search on r->stream: counter resets, the word finder, the
// ordering pass, the lookup-hit counters and the copy of the counters to
// pinned host memory.  No host synchronisation, so it can be captured.
int enqueue_search(hbg_result *r) {
    hbg_db *db = r->db;
    const hbg::HostBatch &h = r->batch->host;
    const size_t nq = h.queries.size(), ng = h.groups.size();
    cudaStream_t st = r->stream;
    CU(cudaMemsetAsync(r->d_counters, 0, r->n_counters * sizeof(unsigned long long), st));
    CU(cudaMemsetAsync(r->d_tile, 0, kMaxLaunchClasses * sizeof(unsigned int), st));

    hbg::WordFinderArgs a;
    memset(&a, 0, sizeof(a));
    a.db = db->d_letters;
    a.db_off = db->d_off;
    a.db_len = db->d_len;
    a.order = db->d_order;
    a.n_subj = db->n;
    hbg_batch *b = r->batch;
    a.groups = b->d_groups;
    a.n_groups = (int32_t)ng;
    a.group_list = b->d_group_list;
    a.cells = b->d_cells;
    a.entries = b->d_entries;
    a.pv = b->d_pv;
    a.letters = b->d_letters;
    a.ctx_of = b->d_ctx_of;
    a.contexts = b->d_ctx;
    a.queries = b->d_queries;
    a.window = h.window;
    a.tile_subjects = 128;
    a.tiles_per_group = (db->n + a.tile_subjects - 1) / a.tile_subjects;
    a.n_tiles = 0;
    a.tile_counter = r->d_tile;
    a.hsps = r->d_raw;
    a.hsp_count = r->d_counters;
    a.hsp_cap = r->cap;
    a.q_extended = r->d_counters + 1;
    a.q_kept = r->d_counters + 1 + nq;
    a.g_hits = r->d_counters + 1 + 3 * nq;
    a.gdiag = r->d_gdiag;
    a.gdiag_len = r->gdiag_len;
    a.smem_diag = h.smem_diag_len;

    // external records while capturing: they become event-record nodes of
    // the graph (usable for timing), not internal fork/join edges; the flag
    // is only accepted during a capture
    cudaStreamCaptureStatus cap_status = cudaStreamCaptureStatusNone;
    CU(cudaStreamIsCapturing(st, &cap_status));
    const unsigned ev_flags =
        cap_status == cudaStreamCaptureStatusActive ? cudaEventRecordExternal : cudaEventRecordDefault;
    CU(cudaEventRecordWithFlags(r->kit.ev[0], st, ev_flags));
    int wf_launches = 0;
    const int rc = launch_finders(db, b, r->plan, a, r->d_counters + 1 + 6 * nq + ng, r->d_side, &r->kit, st, &wf_launches);
    if (rc != HBG_OK)
        return rc;
    CU(cudaEventRecordWithFlags(r->kit.ev[1], st, ev_flags));

    hbg::OrderArgs o;
    memset(&o, 0, sizeof(o));
    o.in = r->d_raw;
    o.out = r->d_sorted;
    o.count = r->d_counters;
    o.cap = r->cap;
    o.keys[0] = r->d_keys;
    o.keys[1] = r->d_keys + r->cap;
    o.vals[0] = r->d_vals;
    o.vals[1] = r->d_vals + r->cap;
    o.hist = r->d_hist;
    o.bits_q = bits_for((int64_t)nq - 1);
    o.bits_s = bits_for((int64_t)db->n - 1);
    o.bits_so = bits_for(db->max_len);
    o.bits_qo = bits_for(h.max_query_len);
    o.q_first = r->d_counters + 1 + 3 * nq + ng;
    o.q_end = o.q_first + nq;
    o.q_passed = o.q_end + nq;
    if (o.bits_q + o.bits_s + o.bits_so + o.bits_qo > 64)
        return fail(HBG_ERR_TOO_LONG, "ordering key exceeds 64 bits for this database and batch");
    o.barrier = r->d_counters + 1 + 6 * nq + 2 * ng;
    o.error = o.barrier + 1;
    o.db_hist = db->d_hist;
    o.query_cells = b->d_qcells;
    o.n_queries = (int32_t)nq;
    o.lookup_hits = r->d_counters + 1 + 2 * nq;
    CU(hbg::launch_order(o, hbg::order_grid(r->device), st));
    r->launches = wf_launches + 1;
    CU(cudaEventRecordWithFlags(r->kit.ev[2], st, ev_flags));
    CU(cudaMemcpyAsync(r->kit.counters, r->d_counters, r->n_counters * sizeof(unsigned long long),
                       cudaMemcpyDeviceToHost, st));
    return HBG_OK;
}

// Launch a search.  A result that is launched again on the same non-default
// stream with the same buffers replays a CUDA graph of the whole sequence
// (captured on its second launch) instead of ~30 separate launches.
int launch_search(hbg_result *r) {
    const bool graphable = r->stream != nullptr && r->launch_count > 0;
    const long long key[5] = {(long long)r->batch_id, (long long)r->cap,
                              ((long long)r->plan_opt.num_blocksx << 32) | (unsigned)r->plan_opt.num_threadsx,
                              (long long)r->gdiag_entries, (long long)(uintptr_t)r->stream};
    const bool same_graph = r->graph_exec && memcmp(key, r->graph_key, sizeof(key)) == 0;
    std::shared_lock<std::shared_mutex> capture(capture_mutex(), std::defer_lock);
    if (!graphable || (!same_graph && !capture.try_lock())) {
        int rc = enqueue_search(r);
        if (rc != HBG_OK)
            return rc;
    } else {
        if (!same_graph) {
            drop_graph(r);
            cudaGraph_t graph = nullptr;
            CU(cudaStreamBeginCapture(r->stream, cudaStreamCaptureModeThreadLocal));
            int rc = enqueue_search(r);
            cudaError_t e = cudaStreamEndCapture(r->stream, &graph);
            if (rc != HBG_OK) {
                if (graph)
                    cudaGraphDestroy(graph);
                return rc;
            }
            if (e != cudaSuccess)
                return fail(HBG_ERR_CUDA, std::string("cudaStreamEndCapture: ") + cudaGetErrorString(e));
            e = cudaGraphInstantiate(&r->graph_exec, graph, 0);
            cudaGraphDestroy(graph);
            if (e != cudaSuccess) {
                r->graph_exec = nullptr;
                return fail(HBG_ERR_CUDA, std::string("cudaGraphInstantiate: ") + cudaGetErrorString(e));
            }
            memcpy(r->graph_key, key, sizeof(key));
            capture.unlock();
        }
        CU(cudaGraphLaunch(r->graph_exec, r->stream));
    }
    r->launch_count++;
    r->launched = true;
    r->synced = false;
    r->done = false;
    return HBG_OK;
}

bool valid_opts(const hbg_gpu_options *o) {
    return o && o->num_threadsx >= 32 && o->num_threadsx <= 256 && (o->num_threadsx % 32) == 0 &&
           o->num_blocksx >= 0;
}

}  // namespace

// Device memory of one search: the batch with the scratch of its table build, and
// a result's buffers, as upload_batch and prepare_result allocate them.
int hbg::search_bytes(const hbg_db *db, const hbg_batch *batch, const hbg_gpu_options *opt, int64_t cap, int64_t *bytes) {
    return guarded([&] {
        hbg_batch *b = const_cast<hbg_batch *>(batch);
        DeviceScope ds(db->device);
        CU(hbg::wordfinder_configure());
        std::lock_guard<std::mutex> lock(b->tables_mu);
        const BatchLayout L = lay_out(b);
        std::vector<LaunchClass> classes;
        std::vector<int32_t> list;
        SearchPlan plan;
        int rc = make_classes(b, &classes, &list);
        if (rc != HBG_OK)
            return rc;
        rc = plan_search(b, classes, db, *opt, &plan);
        if (rc != HBG_OK)
            return rc;
        if (cap == 0)
            cap = default_capacity(db, b);
        *bytes = (int64_t)(L.total + L.scratch()) + cap * (int64_t)(2 * sizeof(hbg_hsp) + 2 * sizeof(uint64_t) + 2 * sizeof(uint32_t)) +
                 256 * hbg::kOrderMaxGrid * (int64_t)sizeof(uint32_t) + (int64_t)counters_need(b->host) * 8 +
                 kMaxLaunchClasses * 4 + gdiag_need(b->host, db, plan) * 4 + side_need(classes, plan) * 2;
        return (int)HBG_OK;
    });
}

extern "C" {

const char *hbg_last_error(void) { return g_err.c_str(); }

int hbg_device_count(int32_t *count) {
    if (!count)
        return fail(HBG_ERR_INVALID, "null count");
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess) {
        *count = 0;
        return fail(HBG_ERR_NO_DEVICE, cudaGetErrorString(e));
    }
    *count = n;
    return HBG_OK;
}

int hbg_default_gpu_options(hbg_gpu_options *opt) {
    if (!opt)
        return fail(HBG_ERR_INVALID, "null options");
    opt->use_gpu = 1;
    opt->num_blocksx = 0;
    opt->num_threadsx = 256;
    opt->method = 0;
    opt->cpu_threads = 1;
    return HBG_OK;
}

}  // extern "C"

namespace {

// Checks shared by the database entry points: options, device.
int db_device(const hbg_gpu_options *opt, hbg_gpu_options *o) {
    hbg_default_gpu_options(o);
    if (opt)
        *o = *opt;
    if (!o->use_gpu)
        return fail(HBG_ERR_NO_DEVICE, "use_gpu is 0 and this library has no CPU path");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0)
        return fail(HBG_ERR_NO_DEVICE, "no CUDA device");
    if (o->method < 0 || o->method >= ndev)
        return fail(HBG_ERR_INVALID, "method selects a device that does not exist");
    return HBG_OK;
}

// Subjects by descending length, equal lengths in database order.
std::vector<int32_t> schedule(const std::vector<int32_t> &len, int32_t max_len) {
    std::vector<int32_t> order(len.size());
    if (max_len > (1 << 20)) {
        std::iota(order.begin(), order.end(), 0);
        std::stable_sort(order.begin(), order.end(), [&](int32_t x, int32_t y) { return len[x] > len[y]; });
        return order;
    }
    std::vector<int32_t> at((size_t)max_len + 2, 0);   // at[k]: next place of length max_len - k
    for (int32_t l : len)
        ++at[(size_t)(max_len - l) + 1];
    for (size_t k = 1; k < at.size(); ++k)
        at[k] += at[k - 1];
    for (size_t i = 0; i < len.size(); ++i)
        order[at[(size_t)(max_len - len[i])]++] = (int32_t)i;
    return order;
}

// Allocate the resident database for a validated layout (subject i at
// device offset off[i], len[i] letters, sentinels between), let `fill` copy
// the letters (it returns "" or an error), then the offsets, the
// length-descending schedule and the word histogram.
template <typename Fill>
int db_create(int device, int32_t n, const std::vector<int64_t> &off, const std::vector<int32_t> &len,
              int64_t total, int32_t max_len, int64_t letters_len, Fill &&fill, hbg_db **out) {
    const std::vector<int32_t> order = schedule(len, max_len);

    hbg_db *db = new (std::nothrow) hbg_db;
    if (!db)
        return fail(HBG_ERR_NOMEM, "host allocation");
    db->device = device;
    db->kits = std::make_shared<KitPool>(device);
    DeviceScope ds(db->device);
    auto bail = [&](int code) {
        dfree(db->d_arena);
        delete db;
        return code;
    };
#define CUB(call)                                                                   \
    do {                                                                            \
        cudaError_t e_ = (call);                                                    \
        if (e_ != cudaSuccess)                                                      \
            return bail(fail(e_ == cudaErrorMemoryAllocation ? HBG_ERR_NOMEM : HBG_ERR_CUDA, \
                             std::string(#call) + ": " + cudaGetErrorString(e_)));  \
    } while (0)
    // one block: letters (with zeros before them and after), offsets, lengths,
    // schedule, histogram
    auto up = [](size_t x) { return (x + 255) / 256 * 256; };
    const size_t o_off = up(kFrontPad + (size_t)letters_len), o_len = up(o_off + sizeof(int64_t) * n),
                 o_order = up(o_len + sizeof(int32_t) * n), o_hist = up(o_order + sizeof(int32_t) * n);
    CUB(dalloc(&db->d_arena, o_hist + sizeof(unsigned long long) * HBG_NUM_CELLS));
    db->d_letters = db->d_arena + kFrontPad;
    db->d_off = reinterpret_cast<int64_t *>(db->d_arena + o_off);
    db->d_len = reinterpret_cast<int32_t *>(db->d_arena + o_len);
    db->d_order = reinterpret_cast<int32_t *>(db->d_arena + o_order);
    db->d_hist = reinterpret_cast<unsigned long long *>(db->d_arena + o_hist);
    CUB(cudaMemset(db->d_arena, 0, kFrontPad + (size_t)letters_len));
    {
        int code = HBG_OK;
        std::string err = fill(db->d_letters, &code);
        if (!err.empty())
            return bail(fail(code, err));
    }
    if (n > 0) {
        CUB(cudaMemcpy(db->d_off, off.data(), sizeof(int64_t) * n, cudaMemcpyHostToDevice));
        CUB(cudaMemcpy(db->d_len, len.data(), sizeof(int32_t) * n, cudaMemcpyHostToDevice));
        CUB(cudaMemcpy(db->d_order, order.data(), sizeof(int32_t) * n, cudaMemcpyHostToDevice));
    }
    CUB(cudaMemset(db->d_hist, 0, sizeof(unsigned long long) * HBG_NUM_CELLS));
    CUB(hbg::launch_db_histogram(db->d_letters, letters_len, db->d_hist, 0));
    CUB(wait_device());
#undef CUB
    db->sched_len.resize(n);
    for (int32_t i = 0; i < n; ++i)
        db->sched_len[i] = len[order[i]];
    db->n = n;
    db->n_res = total;
    db->letters_len = letters_len;
    db->max_len = max_len;
    db->bytes = letters_len + (int64_t)n * 16 + HBG_NUM_CELLS * 8;
    *out = db;
    return HBG_OK;
}

std::string cuda_msg(const char *what, cudaError_t e, int *code) {
    *code = e == cudaErrorMemoryAllocation ? HBG_ERR_NOMEM : HBG_ERR_CUDA;
    return std::string(what) + ": " + cudaGetErrorString(e);
}

std::string bad_letter(int32_t subject) {
    return "subject " + std::to_string(subject) + ": letter outside NCBIstdaa 1..27";
}

// Volumes of a BLAST database with their place in the resident layout:
// volume v's .psq byte b lands at device offset base[v] + b (a volume's
// leading 0 is the previous volume's last separator).
struct BlastDbPlan {
    std::vector<hbg::BlastDbVolume> vols;
    std::vector<int64_t> base;
    int64_t n = 0, total = 0, bytes = 0;
    int32_t max_len = 0;
};

int blastdb_plan(const char *path, BlastDbPlan *plan) {
    if (!path)
        return fail(HBG_ERR_INVALID, "null database name");
    std::vector<std::string> names;
    std::string err = hbg::blastdb_volumes(path, &names);
    if (!err.empty())
        return fail(HBG_ERR_INVALID, err);
    plan->vols.resize(names.size());
    int64_t at = 0;
    for (size_t v = 0; v < names.size(); ++v) {
        err = hbg::blastdb_read_index(names[v], &plan->vols[v]);
        if (!err.empty())
            return fail(HBG_ERR_INVALID, err);
        const hbg::BlastDbVolume &V = plan->vols[v];
        if (V.max_len > HBG_MAX_SUBJECT_LEN)
            return fail(HBG_ERR_TOO_LONG, names[v] + ": a sequence longer than the subject limit");
        plan->base.push_back(v == 0 ? 0 : at - 1);
        at = plan->base.back() + V.psq_bytes;
        plan->n += V.n;
        plan->total += V.residues;
        plan->max_len = std::max(plan->max_len, V.max_len);
    }
    if (plan->n > 0x7fffffff)
        return fail(HBG_ERR_TOO_LONG, "more than 2^31 - 1 sequences");
    plan->bytes = at;
    return HBG_OK;
}

}  // namespace

extern "C" {

int hbg_db_open(const uint8_t *residues, const int64_t *offsets, int32_t n,
                const hbg_gpu_options *opt, hbg_db **out) {
    if (!out || !offsets || n < 0 || (n > 0 && !residues))
        return fail(HBG_ERR_INVALID, "hbg_db_open: null argument or negative count");
    *out = nullptr;
    hbg_gpu_options o;
    int rc = db_device(opt, &o);
    if (rc != HBG_OK)
        return rc;
    // lay out: one sentinel before every subject and after the last
    std::vector<int64_t> off(n);
    std::vector<int32_t> len(n);
    int64_t pos = 1, total = 0;
    int32_t max_len = 0;
    for (int32_t i = 0; i < n; ++i) {
        const int64_t L = offsets[i + 1] - offsets[i];
        if (L < 0 || L > HBG_MAX_SUBJECT_LEN) {
            for (int32_t j = 0; j < i; ++j)         // an earlier subject's fault comes first
                for (int64_t k = offsets[j]; k < offsets[j + 1]; ++k)
                    if (residues[k] == 0 || residues[k] >= HBG_ALPHABET)
                        return fail(HBG_ERR_INVALID, bad_letter(j));
            return fail(L < 0 ? HBG_ERR_INVALID : HBG_ERR_TOO_LONG, "subject " + std::to_string(i) + ": bad length");
        }
        off[i] = pos;
        len[i] = (int32_t)L;
        pos += L + 1;
        total += L;
        max_len = std::max<int32_t>(max_len, (int32_t)L);
    }
    const int64_t letters_len = pos + 64;
    // the letters go up as they lie, 64 MiB at a time, and are checked and
    // spread out on the device
    auto fill = [&](uint8_t *d_letters, int *code) -> std::string {
        if (total == 0)
            return std::string();
        const int64_t piece = std::min<int64_t>(total, (int64_t)64 << 20);
        uint8_t *d_raw = nullptr;
        int64_t *d_first = nullptr;
        int32_t *d_bad = nullptr;
        int32_t bad = INT32_MAX;
        cudaError_t e = dalloc(&d_raw, (size_t)piece);
        if (e == cudaSuccess)
            e = dalloc(&d_first, (size_t)n + 1);
        if (e == cudaSuccess)
            e = dalloc(&d_bad, 1);
        if (e == cudaSuccess)
            e = cudaMemcpy(d_first, offsets, sizeof(int64_t) * ((size_t)n + 1), cudaMemcpyHostToDevice);
        if (e == cudaSuccess)
            e = cudaMemcpy(d_bad, &bad, sizeof(bad), cudaMemcpyHostToDevice);
        for (int64_t at = 0; at < total && e == cudaSuccess; at += piece) {
            const int64_t m = std::min<int64_t>(piece, total - at);
            e = cudaMemcpy(d_raw, residues + offsets[0] + at, (size_t)m, cudaMemcpyHostToDevice);
            if (e == cudaSuccess)
                e = hbg::launch_spread_letters(d_raw, offsets[0] + at, m, d_first, n, d_letters, d_bad, 0);
        }
        if (e == cudaSuccess)
            e = cudaMemcpy(&bad, d_bad, sizeof(bad), cudaMemcpyDeviceToHost);
        else
            wait_device();                          // nothing may still use the buffers
        dfree_idle(d_raw);
        dfree_idle(d_first);
        dfree_idle(d_bad);
        if (e != cudaSuccess)
            return cuda_msg("laying out the subjects", e, code);
        if (bad != INT32_MAX) {
            *code = HBG_ERR_INVALID;
            return bad_letter(bad);
        }
        return std::string();
    };
    return db_create(o.method, n, off, len, total, max_len, letters_len, fill, out);
}

int hbg_blastdb_info(const char *path, int32_t *n_subjects, int64_t *n_residues, int32_t *max_len,
                     int32_t *n_volumes) {
    BlastDbPlan plan;
    int rc = blastdb_plan(path, &plan);
    if (rc != HBG_OK)
        return rc;
    if (n_subjects)
        *n_subjects = (int32_t)plan.n;
    if (n_residues)
        *n_residues = plan.total;
    if (max_len)
        *max_len = plan.max_len;
    if (n_volumes)
        *n_volumes = (int32_t)plan.vols.size();
    return HBG_OK;
}

int hbg_blastdb_read(const char *path, uint8_t *residues, int64_t *offsets) {
    if (!offsets)
        return fail(HBG_ERR_INVALID, "hbg_blastdb_read: null offsets");
    BlastDbPlan plan;
    int rc = blastdb_plan(path, &plan);
    if (rc != HBG_OK)
        return rc;
    if (plan.total > 0 && !residues)
        return fail(HBG_ERR_INVALID, "hbg_blastdb_read: null residues");
    int64_t at = 0, k = 0;
    offsets[0] = 0;
    for (const hbg::BlastDbVolume &V : plan.vols) {
        std::unique_ptr<uint8_t[]> buf(new (std::nothrow) uint8_t[(size_t)V.psq_bytes]);   // not zero-filled
        if (!buf)
            return fail(HBG_ERR_NOMEM, "host allocation");
        std::string err = hbg::blastdb_read_psq(V, 0, V.psq_bytes, buf.get());
        if (!err.empty())
            return fail(HBG_ERR_INVALID, err);
        for (int32_t i = 0; i < V.n; ++i) {
            const int64_t L = (int64_t)V.seq_off[i + 1] - V.seq_off[i] - 1;
            memcpy(residues + at, buf.get() + V.seq_off[i], (size_t)L);
            at += L;
            offsets[++k] = at;
        }
    }
    return HBG_OK;
}

int hbg_db_open_blastdb(const char *path, const hbg_gpu_options *opt, hbg_db **out) {
    if (!out)
        return fail(HBG_ERR_INVALID, "hbg_db_open_blastdb: null out");
    *out = nullptr;
    hbg_gpu_options o;
    int rc = db_device(opt, &o);
    if (rc != HBG_OK)
        return rc;
    BlastDbPlan plan;
    rc = blastdb_plan(path, &plan);
    if (rc != HBG_OK)
        return rc;
    const int32_t n = (int32_t)plan.n;
    std::vector<int64_t> off(n);
    std::vector<int32_t> len(n);
    {
        int64_t k = 0;
        for (size_t v = 0; v < plan.vols.size(); ++v) {
            const hbg::BlastDbVolume &V = plan.vols[v];
            for (int32_t i = 0; i < V.n; ++i, ++k) {
                off[k] = plan.base[v] + V.seq_off[i];
                len[k] = (int32_t)(V.seq_off[i + 1] - V.seq_off[i] - 1);
            }
        }
    }
    const int64_t letters_len = plan.bytes + 64;
    // each volume's .psq is already the device layout: read whole sequences
    // in ~64 MiB pieces into two pinned buffers, checking each piece while
    // the previous one is copied
    auto fill = [&](uint8_t *d_letters, int *code) -> std::string {
        const size_t piece = std::max<size_t>(64u << 20, (size_t)plan.max_len + 2);
        uint8_t *pin[2] = {nullptr, nullptr};
        cudaStream_t st = nullptr;
        cudaEvent_t done[2] = {nullptr, nullptr};
        std::string err;
        cudaError_t e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
        for (int j = 0; j < 2 && e == cudaSuccess; ++j) {
            e = cudaMallocHost(&pin[j], piece);
            if (e == cudaSuccess)
                e = cudaEventCreateWithFlags(&done[j], cudaEventDisableTiming);
        }
        // db_create zeroed the letters on the legacy stream, where a search may
        // still run ahead of it: the copies come after
        if (e == cudaSuccess)
            e = cudaEventRecord(done[0], cudaStreamLegacy);
        if (e == cudaSuccess)
            e = cudaStreamWaitEvent(st, done[0], 0);
        if (e != cudaSuccess)
            err = cuda_msg("staging buffers", e, code);
        int cur = 0;
        bool used[2] = {false, false};
        for (size_t v = 0; v < plan.vols.size() && err.empty(); ++v) {
            const hbg::BlastDbVolume &V = plan.vols[v];
            int32_t i = 0;
            int64_t from = 0;                      // the leading 0 of volume 0 is copied too
            while (err.empty() && (from == 0 || i < V.n)) {
                // whole sequences (with separators) up to the piece size
                int32_t j = i;
                while (j < V.n && (int64_t)V.seq_off[j + 1] - from <= (int64_t)piece)
                    ++j;
                if (j == i && i < V.n)
                    j = i + 1;                     // piece >= longest + 2, so one always fits
                const int64_t to = i < V.n ? (int64_t)V.seq_off[j] : (int64_t)V.seq_off[0];
                if (used[cur]) {
                    e = cudaEventSynchronize(done[cur]);
                    if (e != cudaSuccess) {
                        err = cuda_msg("cudaEventSynchronize", e, code);
                        break;
                    }
                }
                err = hbg::blastdb_read_psq(V, from, to - from, pin[cur]);
                if (!err.empty()) {
                    *code = HBG_ERR_INVALID;
                    break;
                }
                // volume v > 0: its leading 0 is already in place (the buffer starts zeroed)
                const int64_t skip = (from == 0 && v > 0) ? 1 : 0;
                e = cudaMemcpyAsync(d_letters + plan.base[v] + from + skip, pin[cur] + skip,
                                    (size_t)(to - from - skip), cudaMemcpyHostToDevice, st);
                if (e == cudaSuccess)
                    e = cudaEventRecord(done[cur], st);
                if (e != cudaSuccess) {
                    err = cuda_msg("cudaMemcpyAsync (volume)", e, code);
                    break;
                }
                used[cur] = true;
                cur ^= 1;
                from = to;
                i = j;
            }
        }
        if (st) {
            e = cudaStreamSynchronize(st);
            if (e != cudaSuccess && err.empty())
                err = cuda_msg("cudaStreamSynchronize", e, code);
            cudaStreamDestroy(st);
        }
        for (int j = 0; j < 2; ++j) {
            if (done[j])
                cudaEventDestroy(done[j]);
            if (pin[j])
                cudaFreeHost(pin[j]);
        }
        return err;
    };
    return db_create(o.method, n, off, len, plan.total, plan.max_len, letters_len, fill, out);
}

int hbg_db_close(hbg_db *db) {
    if (!db)
        return fail(HBG_ERR_INVALID, "null db");
    DeviceScope ds(db->device);
    dfree(db->d_arena);
    delete db;
    return HBG_OK;
}

int hbg_db_info(const hbg_db *db, int32_t *n, int64_t *res, int64_t *bytes) {
    if (!db)
        return fail(HBG_ERR_INVALID, "null db");
    if (n)
        *n = db->n;
    if (res)
        *res = db->n_res;
    if (bytes)
        *bytes = db->bytes;
    return HBG_OK;
}

static int finish_batch(std::vector<hbg::QueryIn> &qs, const hbg_word_params *params,
                        int32_t max_group_len, hbg_batch **out) {
    hbg_batch *b = new (std::nothrow) hbg_batch;
    if (!b)
        return fail(HBG_ERR_NOMEM, "host allocation");
    std::string err = hbg::build_batch(qs, params->threshold, params->window, max_group_len, &b->host);
    if (!err.empty()) {
        delete b;
        return fail(err.find("length") != std::string::npos ? HBG_ERR_TOO_LONG : HBG_ERR_INVALID, err);
    }
    *out = b;
    return HBG_OK;
}

int hbg_batch_create(const hbg_query *queries, int32_t n_queries, const hbg_word_params *params,
                     int32_t max_group_len, hbg_batch **out) {
    if (!out || !params || !queries || n_queries <= 0)
        return fail(HBG_ERR_INVALID, "hbg_batch_create: null argument or empty batch");
    *out = nullptr;
    std::vector<hbg::QueryIn> qs(n_queries);
    for (int32_t k = 0; k < n_queries; ++k) {
        const hbg_query &q = queries[k];
        if (!q.sequence || q.num_contexts <= 0 || !q.context_offset || !q.context_length ||
            !q.x_dropoff || !q.cutoff_score)
            return fail(HBG_ERR_INVALID, "query " + std::to_string(k) + ": null field");
        qs[k].seq = q.sequence;
        qs[k].len = q.length;
        qs[k].ctx_off.assign(q.context_offset, q.context_offset + q.num_contexts);
        qs[k].ctx_len.assign(q.context_length, q.context_length + q.num_contexts);
        qs[k].xdrop.assign(q.x_dropoff, q.x_dropoff + q.num_contexts);
        qs[k].cutoff.assign(q.cutoff_score, q.cutoff_score + q.num_contexts);
    }
    return finish_batch(qs, params, max_group_len, out);
}

int hbg_seg_default_params(hbg_seg_params *p) {
    if (!p)
        return fail(HBG_ERR_INVALID, "hbg_seg_default_params: null argument");
    p->window = 12;
    p->pad = 0;
    p->locut = 2.2;
    p->hicut = 2.5;
    return HBG_OK;
}

static bool valid_seg(const hbg_seg_params *p) {
    return p && p->window >= 1 && p->window <= 1000 && p->locut >= 0 && p->hicut >= p->locut;
}

int hbg_seg_mask(uint8_t *seq, int32_t len, const hbg_seg_params *p, int64_t *n_masked) {
    if (!seq || len < 0 || !valid_seg(p))
        return fail(HBG_ERR_INVALID, "hbg_seg_mask: null sequence, negative length or bad parameters");
    const int64_t n = hbg::seg_mask(seq, len, p->window, p->locut, p->hicut);
    if (n_masked)
        *n_masked = n;
    return HBG_OK;
}

int hbg_batch_create_blastx(const uint8_t *const *nt, const int32_t *nt_len, int32_t n_queries,
                            const int32_t *x_dropoff, const int32_t *cutoff,
                            const hbg_word_params *params, int32_t max_group_len, hbg_batch **out) {
    return hbg_batch_create_blastx_masked(nt, nt_len, n_queries, x_dropoff, cutoff, params, nullptr,
                                          max_group_len, out);
}

int hbg_batch_create_blastx_masked(const uint8_t *const *nt, const int32_t *nt_len, int32_t n_queries,
                                   const int32_t *x_dropoff, const int32_t *cutoff,
                                   const hbg_word_params *params, const hbg_seg_params *seg,
                                   int32_t max_group_len, hbg_batch **out) {
    if (!out || !params || !nt || !nt_len || !x_dropoff || !cutoff || n_queries <= 0)
        return fail(HBG_ERR_INVALID, "hbg_batch_create_blastx: null argument or empty batch");
    if (seg && !valid_seg(seg))
        return fail(HBG_ERR_INVALID, "hbg_batch_create_blastx_masked: bad SEG parameters");
    *out = nullptr;
    std::vector<std::vector<uint8_t>> prot(n_queries);
    std::vector<hbg::QueryIn> qs(n_queries);
    for (int32_t k = 0; k < n_queries; ++k) {
        if (!nt[k] || nt_len[k] < 3)
            return fail(HBG_ERR_INVALID, "query " + std::to_string(k) + ": need >= 3 nucleotides");
        if ((int64_t)nt_len[k] * 2 + 6 > HBG_MAX_QUERY_LEN)
            return fail(HBG_ERR_TOO_LONG, "query " + std::to_string(k) + ": too long");
        prot[k] = hbg::translate_six_frames(nt[k], nt_len[k], &qs[k].ctx_off, &qs[k].ctx_len);
        if (seg)                                  // each frame is masked as a protein of its own
            for (int f = 0; f < 6; ++f)
                hbg::seg_mask(prot[k].data() + qs[k].ctx_off[f], qs[k].ctx_len[f], seg->window, seg->locut,
                              seg->hicut);
        qs[k].seq = prot[k].data();
        qs[k].len = qs[k].ctx_off[5] + qs[k].ctx_len[5];
        qs[k].xdrop.assign(x_dropoff + 6 * k, x_dropoff + 6 * k + 6);
        qs[k].cutoff.assign(cutoff + 6 * k, cutoff + 6 * k + 6);
        // translated letters may include the sentinel-free stop '*' (25): allowed
    }
    return finish_batch(qs, params, max_group_len, out);
}

int hbg_batch_create_from_smallbone(const hbg_query *query, const hbg_word_params *params,
                                    const void *backbone, int32_t backbone_size,
                                    const uint16_t *overflow, int64_t overflow_size,
                                    hbg_batch **out) {
    if (!out || !params || !query || !backbone || backbone_size <= 0 ||
        backbone_size > HBG_NUM_CELLS || overflow_size < 0 || (overflow_size > 0 && !overflow))
        return fail(HBG_ERR_INVALID, "hbg_batch_create_from_smallbone: bad argument");
    int rc = hbg_batch_create(query, 1, params, 1, out);
    if (rc != HBG_OK)
        return rc;
    hbg::HostBatch &h = (*out)->host;
    // NCBI AaLookupSmallboneCell: Int4 num_used; union { Uint2 entries[3]; Int4 cursor; }
    struct Cell {
        int32_t num_used;
        union {
            uint16_t entries[3];
            int32_t cursor;
        } payload;
    };
    const Cell *cells = (const Cell *)backbone;
    std::vector<uint32_t> cs(HBG_CELL_STRIDE, 0);
    std::vector<uint16_t> ents;
    std::vector<uint32_t> pv(HBG_PV_WORDS, 0);
    std::vector<uint16_t> qc(HBG_NUM_CELLS, 0);
    const int32_t qlen = query->length;
    for (int32_t w = 0; w < HBG_NUM_CELLS; ++w) {
        cs[w] = (uint32_t)ents.size();
        if (w >= backbone_size)
            continue;
        const Cell &c = cells[w];
        if (c.num_used < 0)
            goto bad;
        if (c.num_used == 0)
            continue;
        {
            std::vector<uint16_t> v;
            if (c.num_used <= 3) {
                v.assign(c.payload.entries, c.payload.entries + c.num_used);
            } else {
                if (c.payload.cursor < 0 || (int64_t)c.payload.cursor + c.num_used > overflow_size)
                    goto bad;
                v.assign(overflow + c.payload.cursor, overflow + c.payload.cursor + c.num_used);
            }
            std::sort(v.begin(), v.end());
            h.groups[0].max_cell = std::max(h.groups[0].max_cell, c.num_used);
            if (std::adjacent_find(v.begin(), v.end()) != v.end())
                (*out)->repeated_entries = true;
            for (uint16_t x : v)
                if ((int32_t)x + HBG_WORD_SIZE > qlen)
                    goto bad;
            ents.insert(ents.end(), v.begin(), v.end());
            pv[w >> 5] |= 1u << (w & 31);
            qc[w] = (uint16_t)c.num_used;
        }
    }
    cs[HBG_NUM_CELLS] = (uint32_t)ents.size();
    h.cells = cs;
    h.entries = ents;
    h.pv = pv;
    h.query_cells = qc;
    h.groups[0].entry_base = 0;
    h.groups[0].n_entries = (int32_t)ents.size();
    (*out)->caller_tables = true;
    return HBG_OK;
bad:
    hbg_batch_destroy(*out);
    *out = nullptr;
    return fail(HBG_ERR_INVALID, "smallbone table: bad cell");
}

int hbg_batch_lookup_table(const hbg_batch *b, int32_t g, uint32_t *cells, uint16_t *entries,
                           int64_t entries_cap, int64_t *n_entries, int32_t *first_query,
                           int32_t *n_queries, int32_t *query_start) {
    if (!b || !n_entries || g < 0 || g >= (int32_t)b->host.groups.size())
        return fail(HBG_ERR_INVALID, "hbg_batch_lookup_table: bad argument");
    const int rc = guarded([&] {
        ensure_tables(b);
        return HBG_OK;
    });
    if (rc != HBG_OK)
        return rc;
    const hbg::HostBatch &h = b->host;
    const HbgGroup &G = h.groups[g];
    const uint32_t *cs = h.cells.data() + (size_t)g * HBG_CELL_STRIDE;
    const int64_t n = cs[HBG_NUM_CELLS];
    *n_entries = n;
    if (first_query)
        *first_query = G.first_query;
    if (n_queries)
        *n_queries = G.n_queries;
    if (query_start)
        for (int32_t k = 0; k < G.n_queries; ++k)
            query_start[k] = h.queries[G.first_query + k].start;
    if (cells)
        memcpy(cells, cs, sizeof(uint32_t) * HBG_CELL_STRIDE);
    if (entries) {
        if (entries_cap < n)
            return fail(HBG_ERR_CAPACITY, "entries buffer too small");
        if (n)
            memcpy(entries, h.entries.data() + G.entry_base, sizeof(uint16_t) * (size_t)n);
    }
    return HBG_OK;
}

int hbg_batch_set_mode(hbg_batch *b, int32_t g, int32_t mode) {
    if (!b || (mode != 0 && mode != 1) || g >= (int32_t)b->host.groups.size())
        return fail(HBG_ERR_INVALID, "hbg_batch_set_mode: bad argument");
    if (b->device >= 0)
        return fail(HBG_ERR_STATE, "batch already uploaded: set modes before the first search");
    for (int32_t i = 0; i < (int32_t)b->host.groups.size(); ++i)
        if (g < 0 || i == g)
            b->host.groups[i].mode = mode;
    return HBG_OK;
}

int hbg_batch_tune(hbg_batch *b, int32_t tile_subjects, int32_t global_tables) {
    if (!b || tile_subjects < 0 || (tile_subjects > 0 && (tile_subjects < 8 || tile_subjects > 4096)) ||
        (global_tables != 0 && global_tables != 1))
        return fail(HBG_ERR_INVALID, "hbg_batch_tune: bad argument");
    if (b->device >= 0)
        return fail(HBG_ERR_STATE, "batch already uploaded: tune before the first search");
    b->tile_subjects = tile_subjects;
    b->tuned = b->tuned || tile_subjects > 0 || global_tables;
    if (global_tables) {
        hbg::HostBatch &h = b->host;
        for (HbgGroup &G : h.groups) {
            if (G.placement)
                continue;
            int32_t n = 1;
            while (n < G.glen + h.window)
                n <<= 1;
            G.diag_len = n;                      // global tables are powers of two
            G.placement = 1;
            h.max_diag_len = std::max(h.max_diag_len, G.diag_len);
        }
    }
    return HBG_OK;
}

int hbg_batch_schedule(hbg_batch *b, int32_t warps_per_subject, int64_t tile_bytes) {
    if (!b || warps_per_subject < 1 || warps_per_subject > 8 || tile_bytes < 0 ||
        (tile_bytes > 0 && (tile_bytes < 1024 || tile_bytes > ((int64_t)1 << 24))))
        return fail(HBG_ERR_INVALID, "hbg_batch_schedule: warps_per_subject 1..8, tile_bytes 0 or 1 KiB..16 MiB");
    if (b->device >= 0)
        return fail(HBG_ERR_STATE, "batch already uploaded: schedule before the first search");
    b->team = warps_per_subject;
    b->tile_bytes = tile_bytes;
    return HBG_OK;
}

int hbg_batch_destroy(hbg_batch *b) {
    if (!b)
        return fail(HBG_ERR_INVALID, "null batch");
    if (b->device >= 0) {
        DeviceScope ds(b->device);
        free_batch_device(b);
    }
    delete b;
    return HBG_OK;
}

int hbg_batch_info(const hbg_batch *b, int32_t *nq, int32_t *ng, int64_t *qlen, int64_t *entries,
                   int64_t *device_bytes) {
    if (!b)
        return fail(HBG_ERR_INVALID, "null batch");
    if (nq)
        *nq = (int32_t)b->host.queries.size();
    if (ng)
        *ng = (int32_t)b->host.groups.size();
    if (qlen) {
        int64_t t = 0;
        for (auto &q : b->host.queries)
            t += q.len;
        *qlen = t;
    }
    if (!entries && !device_bytes)
        return HBG_OK;
    return guarded([&] {
        hbg_batch *m = const_cast<hbg_batch *>(b);
        std::lock_guard<std::mutex> lock(m->tables_mu);
        if (entries)
            *entries = hbg::count_entries(&m->host);
        if (device_bytes)
            *device_bytes = (int64_t)lay_out(m).total;
        return HBG_OK;
    });
}

int hbg_mem_required(const hbg_db *db, const hbg_batch *b, int64_t cap, int64_t *bytes) {
    if (!db || !b || !bytes || cap < 0)
        return fail(HBG_ERR_INVALID, "hbg_mem_required: bad argument");
    hbg_gpu_options o;
    hbg_default_gpu_options(&o);
    return hbg::search_bytes(db, b, &o, cap, bytes);
}

int hbg_search(hbg_db *db, hbg_batch *batch, const hbg_gpu_options *opt, int64_t cap,
               void *stream, hbg_result **out) {
    if (!db || !batch || !out || cap < 0)
        return fail(HBG_ERR_INVALID, "hbg_search: null argument");
    hbg_gpu_options o;
    hbg_default_gpu_options(&o);
    if (opt)
        o = *opt;
    if (!o.use_gpu)
        return fail(HBG_ERR_NO_DEVICE, "use_gpu is 0 and this library has no CPU path");
    if (!valid_opts(&o))
        return fail(HBG_ERR_INVALID, "num_threadsx must be a multiple of 32 in 32..256");
    DeviceScope ds(db->device);
    int rc = upload_batch(batch, db, (cudaStream_t)stream);
    if (rc != HBG_OK)
        return rc;
    hbg_result *r = *out;
    if (r && (r->db != db || r->db_id != db->id))
        return fail(HBG_ERR_STATE, "a reused result must belong to the same database");
    if (r && r->launched && !r->synced)
        return fail(HBG_ERR_STATE, "the result's previous search has not been waited for");
    if (r && (r->batch != batch || r->batch_id != batch->id)) {
        // re-target the buffers to another batch of the same database
        r->batch = batch;
        r->batch_id = batch->id;
        r->graph_exec ? (void)cudaGraphExecDestroy(r->graph_exec) : (void)0;
        r->graph_exec = nullptr;
        r->launch_count = 0;
    }
    if (!r) {
        r = new (std::nothrow) hbg_result;
        if (!r)
            return fail(HBG_ERR_NOMEM, "host allocation");
        r->db = db;
        r->db_id = db->id;
        r->batch = batch;
        r->batch_id = batch->id;
        r->device = db->device;
        r->kits = db->kits;
    }
    r->opt = o;
    r->stream = (cudaStream_t)stream;
    r->build = batch->build;
    r->nq = batch->host.queries.size();
    r->ng = batch->host.groups.size();
    // a repeated search has its plan
    if (r->launch_count == 0 || memcmp(&r->plan_opt, &o, sizeof(o)) != 0) {
        if (hbg::wordfinder_configure() != cudaSuccess || hbg::byte_configure() != cudaSuccess)
            rc = fail(HBG_ERR_CUDA, "cannot configure the word-finder kernel (wrong GPU?)");
        else
            rc = plan_search(batch, batch->classes, db, o, &r->plan);
        if (rc != HBG_OK) {
            r->launch_count = 0;                 // no plan
            if (!*out)
                delete r;
            return rc;
        }
        r->plan_opt = o;
    }
    // a default capacity that does not fit the device falls back to the
    // smallest one: a search that finds more HSPs is run again with room for them
    const int64_t least = std::max<int64_t>(1 << 20, (int64_t)db->n);
    const bool chosen = cap > 0;
    if (!chosen)
        cap = default_capacity(db, batch);
    rc = prepare_result(r, std::max<int64_t>(cap, r->cap));
    if (rc == HBG_ERR_NOMEM && !chosen && cap > least)
        rc = prepare_result(r, std::max<int64_t>(least, r->cap));
    if (rc == HBG_OK)
        rc = launch_search(r);
    if (rc != HBG_OK) {
        cudaStreamSynchronize(r->stream);       // a partly enqueued search may still run
        KitPool::wait_sides(r->kit);
        if (!*out) {
            free_result_device(r);
            delete r;
        }
        return rc;
    }
    *out = r;
    return HBG_OK;
}

int hbg_result_sync(hbg_result *r) {
    if (!r || !r->launched)
        return fail(HBG_ERR_STATE, "no search launched on this result");
    if (r->synced)
        return HBG_OK;
    DeviceScope ds(r->device);
    CU(cudaStreamSynchronize(r->stream));
    unsigned long long n = r->kit.counters[0];
    if ((int64_t)n > r->cap) {
        // the HSP buffer was too small: relaunch once with the exact size.  If
        // that cannot be set up, nothing of this search runs any more and the
        // result may be relaunched (or reused for another batch) later.
        int rc = prepare_result(r, (int64_t)n);
        if (rc == HBG_OK)
            rc = launch_search(r);
        if (rc != HBG_OK) {
            cudaStreamSynchronize(r->stream);
            KitPool::wait_sides(r->kit);
            r->launched = false;
            return rc;
        }
        CU(cudaStreamSynchronize(r->stream));
        n = r->kit.counters[0];
        if ((int64_t)n > r->cap)
            return fail(HBG_ERR_STATE, "HSP count changed between identical launches");
    }
    if (r->kit.counters[2 + 6 * r->nq + 2 * r->ng]) {   // a result may be launched again
        r->launched = false;
        return fail(HBG_ERR_CUDA, "the ordering pass gave up waiting for its own blocks");
    }
    r->n_hsps = (int64_t)n;
    if (!r->build->over)
        r->build->ended();
    CU(cudaEventElapsedTime(&r->wf_ms, r->kit.ev[0], r->kit.ev[1]));
    CU(cudaEventElapsedTime(&r->ord_ms, r->kit.ev[1], r->kit.ev[2]));
    r->synced = true;
    return HBG_OK;
}

int hbg_result_wait(hbg_result *r) {
    int rc = hbg_result_sync(r);
    if (rc != HBG_OK)
        return rc;
    if (r->done)
        return HBG_OK;
    // the ordered HSPs stay on the device (read with hbg_result_hsps); the
    // ordering pass left per-query ranges and subject counts beside the counters
    const size_t nq = r->nq, ng = r->ng;
    const unsigned long long *rng = r->kit.counters + 1 + 3 * nq + ng;
    r->stats.assign(nq, hbg_query_stats{0, 0, 0, 0});
    r->q_first.assign(nq, 0);
    r->q_count.assign(nq, 0);
    for (size_t q = 0; q < nq; ++q) {
        r->stats[q].init_extends = (int64_t)r->kit.counters[1 + q];
        r->stats[q].good_init_extends = (int64_t)r->kit.counters[1 + nq + q];
        r->stats[q].lookup_hits = (int64_t)r->kit.counters[1 + 2 * nq + q];
        r->stats[q].subjects_passed = (int64_t)rng[2 * nq + q];
        r->q_first[q] = (int64_t)rng[q];
        r->q_count[q] = (int64_t)rng[nq + q] - (int64_t)rng[q];
    }
    r->done = true;
    return HBG_OK;
}

int hbg_result_timing(const hbg_result *r, float *wf, float *ord, int32_t *launches) {
    if (!r || !r->synced)
        return fail(HBG_ERR_STATE, "result not collected");
    if (wf)
        *wf = r->wf_ms;
    if (ord)
        *ord = r->ord_ms;
    if (launches)
        *launches = r->launches;
    return HBG_OK;
}

int hbg_result_counts(const hbg_result *r, int64_t *n_hsps, int32_t *n_queries) {
    if (!r || !r->synced)
        return fail(HBG_ERR_STATE, "result not collected");
    if (n_hsps)
        *n_hsps = r->n_hsps;
    if (n_queries)
        *n_queries = (int32_t)r->nq;
    return HBG_OK;
}

int hbg_result_hsps(const hbg_result *r, int64_t first, int64_t count, hbg_hsp *out) {
    if (!r || !r->done)
        return fail(HBG_ERR_STATE, "result not collected");
    if (first < 0 || count < 0 || first + count > r->n_hsps || (count > 0 && !out))
        return fail(HBG_ERR_INVALID, "range outside the result");
    if (count) {
        // on the search's own stream, so the copy neither waits for nor races
        // with work on other streams
        DeviceScope ds(r->device);
        CU(cudaMemcpyAsync(out, r->d_sorted + first, (size_t)count * sizeof(hbg_hsp), cudaMemcpyDeviceToHost,
                           r->stream));
        CU(cudaStreamSynchronize(r->stream));
    }
    return HBG_OK;
}

int hbg_result_query_range(const hbg_result *r, int32_t q, int64_t *first, int64_t *count) {
    if (!r || !r->done)
        return fail(HBG_ERR_STATE, "result not collected");
    if (q < 0 || q >= (int32_t)r->q_first.size() || !first || !count)
        return fail(HBG_ERR_INVALID, "query index outside the batch");
    *first = r->q_first[q];
    *count = r->q_count[q];
    return HBG_OK;
}

int hbg_result_stats(const hbg_result *r, int32_t q, hbg_query_stats *out) {
    if (!r || !r->done)
        return fail(HBG_ERR_STATE, "result not collected");
    if (q < 0 || q >= (int32_t)r->stats.size() || !out)
        return fail(HBG_ERR_INVALID, "query index outside the batch");
    *out = r->stats[q];
    return HBG_OK;
}

int hbg_result_free(hbg_result *r) {
    if (!r)
        return fail(HBG_ERR_INVALID, "null result");
    DeviceScope ds(r->device);
    free_result_device(r);
    delete r;
    return HBG_OK;
}

int hbg_search_sync(hbg_db *db, hbg_batch *batch, const hbg_gpu_options *opt, hbg_hsp *out,
                    int64_t out_cap, int64_t *n_hsps, hbg_query_stats *stats, void *stream) {
    if (!n_hsps || out_cap < 0)
        return fail(HBG_ERR_INVALID, "hbg_search_sync: bad argument");
    hbg_result *r = nullptr;
    int rc = hbg_search(db, batch, opt, 0, stream, &r);
    if (rc != HBG_OK)
        return rc;
    rc = hbg_result_wait(r);
    if (rc == HBG_OK) {
        *n_hsps = r->n_hsps;
        if (stats)
            for (size_t q = 0; q < r->stats.size(); ++q)
                stats[q] = r->stats[q];
        if (out) {
            if (r->n_hsps > out_cap)
                rc = fail(HBG_ERR_CAPACITY, "output buffer too small");
            else if (r->n_hsps) {
                DeviceScope ds(r->device);
                cudaError_t e = cudaMemcpyAsync(out, r->d_sorted, (size_t)r->n_hsps * sizeof(hbg_hsp),
                                                cudaMemcpyDeviceToHost, r->stream);
                if (e == cudaSuccess)
                    e = cudaStreamSynchronize(r->stream);
                if (e != cudaSuccess)
                    rc = fail(HBG_ERR_CUDA, std::string("cudaMemcpy (HSPs): ") + cudaGetErrorString(e));
            }
        }
    }
    hbg_result_free(r);
    return rc;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Search without allocation.
//
// For callers that may not allocate device memory at search time --
// allocator-free real-time services whose latency budget has no room for
// cudaMalloc's implicit synchronisation, and hosts that hand the library a
// fixed memory budget at start-up and own every device byte after that -- this
// entry point launches the word finder with its scratch in a file-scope device
// array instead of cudaMalloc'd buffers.  The array is HBG_STATIC_SCRATCH_BYTES
// on every device that loads the library and stays allocated until exit.

namespace {

constexpr int kStaticMaxDevices = 64;
__device__ __align__(256) unsigned char g_static_scratch[HBG_STATIC_SCRATCH_BYTES];

std::mutex g_static_mu;
void *g_static_ptr[kStaticMaxDevices];   // device address of g_static_scratch, per device

// Device address of the scratch array on `device` (current device on entry).
// The array's name is only a host-side stand-in in host code, so the address
// is looked up once per device with cudaGetSymbolAddress.
int static_scratch(int device, void **out) {
    if (device < 0 || device >= kStaticMaxDevices)
        return fail(HBG_ERR_INVALID, "device index outside the static scratch table");
    std::lock_guard<std::mutex> lock(g_static_mu);
    if (!g_static_ptr[device]) {
        void *p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_static_scratch);
        if (e != cudaSuccess || !p)
            return fail(HBG_ERR_CUDA, std::string("cudaGetSymbolAddress(static scratch): ") +
                                          cudaGetErrorString(e));
        g_static_ptr[device] = p;
    }
    *out = g_static_ptr[device];
    return HBG_OK;
}

}  // namespace

extern "C" int hbg_search_static(const hbg_db *db, const hbg_batch *batch, const hbg_gpu_options *opt,
                                 hbg_hsp *d_hsps, int64_t hsp_cap, unsigned long long *d_counts,
                                 void *stream) {
    if (!db || !batch || !d_counts || hsp_cap < 0 || (hsp_cap > 0 && !d_hsps))
        return fail(HBG_ERR_INVALID, "hbg_search_static: null argument or negative capacity");
    if (batch->device != db->device)
        return fail(HBG_ERR_STATE, "hbg_search_static: the batch is not resident on the database's device "
                                   "(run hbg_search on it once during set-up)");
    hbg_gpu_options o;
    hbg_default_gpu_options(&o);
    if (opt)
        o = *opt;
    if (!o.use_gpu)
        return fail(HBG_ERR_NO_DEVICE, "use_gpu is 0 and this library has no CPU path");
    if (!valid_opts(&o))
        return fail(HBG_ERR_INVALID, "num_threadsx must be a multiple of 32 in 32..256");
    const hbg::HostBatch &h = batch->host;
    const int64_t nq = (int64_t)h.queries.size(), ng = (int64_t)h.groups.size();
    // scratch layout: [tile counters (one per launch class) | per-query extensions |
    //                  per-query kept | per-group hits]
    static_assert(kMaxLaunchClasses * sizeof(unsigned int) <= 256,
                  "the tile counters must fit the 256-byte head of the static scratch");
    const int64_t need = 256 + 8 * (2 * nq + ng);
    if (need > HBG_STATIC_SCRATCH_BYTES)
        return fail(HBG_ERR_TOO_LONG, "hbg_search_static: the batch needs " + std::to_string(need) +
                                          " scratch bytes, more than HBG_STATIC_SCRATCH_BYTES");
    if (global_diag_len(h, db) > 0)
        return fail(HBG_ERR_TOO_LONG, "hbg_search_static: groups longer than 2008 letters or subjects "
                                      "longer than 32767 - window need global diagonal tables");
    DeviceScope ds(db->device);
    void *scratch = nullptr;
    int rc = static_scratch(db->device, &scratch);
    if (rc != HBG_OK)
        return rc;
    CU(hbg::wordfinder_configure());
    CU(hbg::byte_configure());
    SearchPlan plan;                   // host-side only; no device allocation
    rc = plan_search(batch, batch->classes, db, o, &plan);
    if (rc != HBG_OK)
        return rc;
    cudaStream_t st = (cudaStream_t)stream;
    rc = after_build(batch, st);
    if (rc != HBG_OK)
        return rc;
    unsigned char *base = (unsigned char *)scratch;
    unsigned int *tile = (unsigned int *)base;
    unsigned long long *q_ext = (unsigned long long *)(base + 256);
    unsigned long long *q_kept = q_ext + nq;
    unsigned long long *g_hits = q_kept + nq;
    // every call shares the array: clear what the kernel accumulates into
    CU(cudaMemsetAsync(scratch, 0, (size_t)need, st));
    CU(cudaMemsetAsync(d_counts, 0, sizeof(unsigned long long) * (size_t)(1 + 2 * nq), st));

    hbg::WordFinderArgs a;
    memset(&a, 0, sizeof(a));
    a.db = db->d_letters;
    a.db_off = db->d_off;
    a.db_len = db->d_len;
    a.order = db->d_order;
    a.n_subj = db->n;
    a.groups = batch->d_groups;
    a.n_groups = (int32_t)ng;
    a.cells = batch->d_cells;
    a.entries = batch->d_entries;
    a.pv = batch->d_pv;
    a.letters = batch->d_letters;
    a.ctx_of = batch->d_ctx_of;
    a.contexts = batch->d_ctx;
    a.queries = batch->d_queries;
    a.window = h.window;
    a.tile_subjects = 128;
    a.tiles_per_group = (db->n + a.tile_subjects - 1) / a.tile_subjects;
    a.n_tiles = 0;
    a.tile_counter = tile;
    a.hsps = d_hsps;
    a.hsp_count = d_counts;
    a.hsp_cap = hsp_cap;
    a.q_extended = q_ext;
    a.q_kept = q_kept;
    a.g_hits = g_hits;
    a.gdiag = nullptr;
    a.gdiag_len = 0;
    a.smem_diag = h.smem_diag_len;
    // 16-bit cells (longer groups are refused above), so no side table; the
    // group counters serve as subject counters
    int launches = 0;
    rc = launch_finders(db, batch, plan, a, g_hits, nullptr, nullptr, st, &launches);
    if (rc != HBG_OK)
        return rc;
    // per-query extension and kept counts follow the HSP count in d_counts
    CU(cudaMemcpyAsync(d_counts + 1, q_ext, sizeof(unsigned long long) * (size_t)(2 * nq),
                       cudaMemcpyDeviceToDevice, st));
    return HBG_OK;
}

extern "C" int hbg_debug_fail_allocations(int32_t count) {
    if (count < 0)
        return fail(HBG_ERR_INVALID, "hbg_debug_fail_allocations: negative count");
    g_fail_allocs.store(count);
    return HBG_OK;
}
