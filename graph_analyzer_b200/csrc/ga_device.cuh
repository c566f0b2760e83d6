// ga_device.cuh - device helpers and the ga_graph handle shared by the CUDA translation units of libga_b200.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>
#include <vector>

#include "ga_internal.h"

#define GA_FULL_MASK 0xFFFFFFFFu
#define GA_EMPTY 0xFFFFFFFFu

// Returns GA_ERR_CUDA / GA_ERR_OUT_OF_MEMORY with the failing call's text when a CUDA call fails (and takes the error
// off the runtime's record, where the next call's launch check would find it).
#define GA_CUDA(call)                                                                                          \
    do {                                                                                                       \
        cudaError_t e_ = (call);                                                                               \
        if (e_ != cudaSuccess) {                                                                               \
            (void)cudaGetLastError();                                                                          \
            return ::ga::fail(e_ == cudaErrorMemoryAllocation ? GA_ERR_OUT_OF_MEMORY : GA_ERR_CUDA,            \
                              "%s failed: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__);     \
        }                                                                                                      \
    } while (0)

#define GA_TRY(expr)                         \
    do {                                     \
        ga_status s_ = (expr);               \
        if (s_ != GA_OK) return s_;          \
    } while (0)

namespace ga {

constexpr int kSmCountB200 = 148;

// ---- warp-level helpers --------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t x, uint32_t lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(GA_FULL_MASK, x, o);
        if (lane >= (uint32_t)o) x += t;
    }
    return x;
}
__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(GA_FULL_MASK, x, o);
    return x;
}

// Additions to global counters whose old value nobody wants, as the reduction they are: in a kernel that also has a
// __threadfence (the last block's turn), an atomicAdd without a use of its result is compiled to an atomic that returns
// one, and a warp then waits for it (R-MAT 22 edge supports 7.2 ms against 6.3).
__device__ __forceinline__ void red_add(uint32_t* p, uint32_t v) {
    asm volatile("red.relaxed.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void red_add(unsigned long long* p, unsigned long long v) {
    asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Multiplicative hash onto `bits` bits (Knuth): the high bits of x * 2654435761 mod 2^32.
__device__ __forceinline__ uint32_t hash_slot(uint32_t x, uint32_t bits) {
    return (x * 2654435761u) >> (32 - bits);
}

// First index in sorted a[lo, hi) whose value is >= x.
__device__ __forceinline__ uint32_t lower_bound_u32(const uint32_t* __restrict__ a, uint32_t lo, uint32_t hi,
                                                    uint32_t x) {
    while (lo < hi) {
        const uint32_t mid = lo + ((hi - lo) >> 1);
        if (a[mid] < x) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// ---- the index's formats --------------------------------------------------------------------------------------------
constexpr uint32_t kPad = 0xFFFFFFFFu;   // padding of the last oct of a row in colr: above every place

// in_rng: the padded position of the edge's entry in its source's row plus one (35 bits: up to 2^32 octs of 8) and the
// octs from there to the row's end that hold entries after it (29 bits: a row has fewer than 2^32 entries).
__host__ __device__ __forceinline__ unsigned long long pack_rng(unsigned long long at, uint32_t octs) {
    return (unsigned long long)octs << 35 | (at + 1);
}
__device__ __forceinline__ unsigned long long rng_at(unsigned long long r) { return (r & ((1ull << 35) - 1)) - 1; }
__device__ __forceinline__ uint32_t rng_oct(unsigned long long r) {   // the first oct of the suffix
    return (uint32_t)((r & ((1ull << 35) - 1)) >> 3);
}
__device__ __forceinline__ uint32_t rng_octs(unsigned long long r) { return (uint32_t)(r >> 35); }

// The tiny bin: anchors of so few out-neighbours (two octs) that an in-edge is one lane's work, without hubs among
// their in-lists (a warp takes 32 such anchors at once).
constexpr uint32_t kTinyDeg = 16, kTinyIn = 32, kTinyWork = 256, kTinyGroups = 4;
__device__ __forceinline__ uint32_t is_tiny(uint32_t d, uint32_t in, uint32_t work, uint32_t light_max_deg) {
    return d && work && d <= kTinyDeg && in <= kTinyIn && work <= kTinyWork && d <= light_max_deg;
}

// ---- grid sizing ------------------------------------------------------------------------------------------------
inline unsigned grid_for(uint64_t threads, int block, unsigned cap = 148u * 64u) {
    uint64_t b = (threads + block - 1) / block;
    if (b < 1) b = 1;
    if (b > cap) b = cap;
    return (unsigned)b;
}

}  // namespace ga

struct ga_loops;   // round-loop state (ga_loops.cu)

// Work items of the triangle kernels, heavy then light then tiny, each bin by ascending anchor: item i covers in-edges
// [k0[i], k1[i]) of anchor (place) v[i]. The bins' sizes are on the device (info[0..2]).
struct ga_items {
    uint32_t *v = nullptr, *k0 = nullptr, *k1 = nullptr, *info = nullptr;
    uint64_t capacity = 0, bound = 0;   // entries allocated; at least the number of items
};

// Counters of a handle's triangle passes (device). Synchronous calls use the first work queues, `ticket` (blocks that
// have finished) and `acc` (triangles so far), all zero between passes: the last block of a pass clears them. A pass
// that an _async call enqueues shares none of these, since it may be captured and replayed beside other passes: it adds
// to the caller's total, and its work queues, cleared before it, are the second ones, or for a captured pass its own
// (captured_work). bounds: the item ranges of a shard.
struct ga_work {
    uint32_t queue[4], bounds[6];
};
struct ga_sync {
    ga_work work[2];
    uint32_t ticket, pad;
    unsigned long long acc;
};

struct ga_graph {
    int device = 0;
    int sm_count = 148;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    uint32_t n = 0, m = 0, max_out_degree = 0;

    // oriented CSR, the reference's layout (graph.h:19-26)
    uint32_t* rowptr = nullptr;   // n+1
    uint32_t* col = nullptr;      // m
    uint32_t* src = nullptr;      // m (built on the device)

    uint32_t* deg = nullptr;      // n: degree, out + in (built on the device with the upload checks)
    uint32_t max_degree = 0, isolated = 0;   // largest degree, vertices of degree 0 (the first places)
    uint64_t octs = 0;            // octs of all rows: sum of ceil(d+ / 8)
    uint64_t row_work = 0;        // sum of d+ * ceil(d+ / 8): bounds the probe work
    uint64_t row_hist[33] = {};   // edges by 1 + floor(log2) of their row's length
    bool misoriented = false;     // an edge is not oriented by (degree, id): every use that needs it refuses

    // the index (ga_graph.cu): vertices numbered by (degree, id), rows and in-lists in these numbers (places)
    uint32_t* vrank = nullptr;    // n: place of every id
    uint32_t* order = nullptr;    // n: id of every place
    uint32_t* dout = nullptr;     // n: out-degree, by place
    uint32_t* work = nullptr;     // n: octs to probe for an anchor, by place
    uint2* pos = nullptr;         // n+1, by place: start of its in-edges in in_rng (x), of its row in colr (y, octs)
    uint32_t* colr = nullptr;     // 8 * octs: rows as ascending places, padded with kPad
    uint32_t* osrc = nullptr;     // octs: place of the row an oct belongs to
    unsigned long long* in_rng = nullptr;   // m: in-edge u->v as pack_rng(padded position of v in u's row, suffix octs)

    unsigned long long* anchor_work = nullptr;   // n+1: probe work of the anchors below a place (cuts shards; lazy)
    ga_items items;               // work lists of the triangle kernels
    bool index_ready = false;     // vrank .. in_rng built
    bool prepared = false;        // ... and the work items for the current light_max_deg / item_work
    bool counted_bare = false;    // counted once without the index (ga_tc_count)
    cudaEvent_t built = nullptr;  // recorded behind the latest build of the index or the items
    ga_loops* loops = nullptr;    // peeling / core loop state, allocated on first use
    // a batch: the graph is the disjoint union of seg_count graphs, graph s owning vertices [seg_off[s], seg_off[s+1])
    const unsigned long long* seg_off = nullptr;
    uint32_t seg_count = 0;

    // small device / pinned host scalars
    unsigned long long* d_scalars = nullptr;   // 64 slots
    unsigned long long* h_scalars = nullptr;   // their page-locked host side (64 slots; host_slot_acquire)
    ga_sync* sync = nullptr;                   // counters of the triangle passes
    ga_work* captured = nullptr;               // work queues for the next captured passes ...
    uint32_t captured_left = 0;                // ... and how many there are
    bool items_captured = false;               // a captured pass reads the current work lists

    // options (ga_option)
    int64_t opt_tc_kernel = 0, opt_loop_mode = 0, opt_max_rounds = 0, opt_update_mode = 0, opt_count_bitmap = 0;
    int tuned_kernel = 0;          // count kernel chosen by the autotuner (1 plain, 2 hash; 0 not tuned yet)
    uint64_t tune_key = 0;         // degree-distribution signature it was chosen for
    float tune_ms = 0;             // the chosen configuration's count time when it was measured (0: from the cache)
    uint32_t item_work = 4096, heavy_bits_cap = 0, light_max_deg = 128;
    bool item_work_set = false, light_max_deg_set = false;   // set by the caller: the autotuner leaves them

    // every device allocation, freed by ga_graph_destroy
    std::vector<std::pair<void*, size_t>> allocations;
    uint64_t bytes = 0;
    // every C-ABI call on this graph holds it (recursive: some entry points call others), so calls from several
    // host threads on one handle are serialised instead of racing on its scratch arrays and stream
    mutable std::recursive_mutex mu;
};

#define GA_GRAPH_LOCK(g) std::lock_guard<std::recursive_mutex> ga_graph_lock_((g)->mu)

namespace ga {

// Creates the library's own memory pool of a device once per process: freed blocks stay cached (up to 8 GiB) so
// that graphs created and destroyed repeatedly reuse memory instead of returning it to the driver. A pool of its own
// leaves the device's default pool (which other code in the process may use) as it was.
ga_status init_pool(int device);

// 512 page-locked bytes every device can write, for the small results of one handle: from slabs the process keeps (at
// most 64 KB of them: 128 handles; further handles allocate their own), handed back at destroy. nullptr: out of memory.
unsigned long long* host_slot_acquire();
void host_slot_release(unsigned long long* slot);

// A non-blocking stream of the device, and its return (idle) when the handle ends. device < 64 (init_pool checks).
cudaError_t stream_acquire(int device, cudaStream_t* st);
void stream_release(int device, cudaStream_t st);

// Copies a result to host memory of the caller on g's stream and waits for it.
ga_status download(ga_graph* g, void* dst, const void* src, size_t bytes);

// The pool of the current device (init_pool must have run for it; every entry point that allocates calls it).
cudaMemPool_t pool_of_current();

// Stream-ordered allocation from the library's pool of the current device.
template <class T>
inline cudaError_t pool_malloc(T** p, size_t bytes, cudaStream_t st) {
    return cudaMallocFromPoolAsync((void**)p, bytes, pool_of_current(), st);
}

// A temporary of a call, given back (stream-ordered) when it goes out of scope, whatever ends the scope.
struct Scratch {
    void* p = nullptr;
    cudaStream_t st = nullptr;
    explicit Scratch(cudaStream_t s) : st(s) {}
    Scratch(const Scratch&) = delete;
    ~Scratch() { if (p) cudaFreeAsync(p, st); }
    template <class T>
    ga_status alloc(T** out, size_t count) {
        const size_t bytes = (count ? count : 1) * sizeof(T);
        if (pool_malloc(&p, bytes, st) != cudaSuccess) {
            (void)cudaGetLastError();
            p = nullptr;
            return fail(GA_ERR_OUT_OF_MEMORY, "device scratch of %zu bytes failed", bytes);
        }
        *out = (T*)p;
        return GA_OK;
    }
};

// Device allocation owned by g (stream-ordered from the pool on g's stream, freed at destroy), counted in g->bytes.
template <class T>
inline ga_status dalloc(ga_graph* g, T** p, size_t count) {
    void* q = nullptr;
    const size_t bytes = (count ? count : 1) * sizeof(T);
    cudaError_t e = pool_malloc(&q, bytes, g->stream);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return fail(GA_ERR_OUT_OF_MEMORY, "cudaMalloc of %zu bytes failed: %s", bytes, cudaGetErrorString(e));
    }
    g->allocations.emplace_back(q, bytes);
    g->bytes += bytes;
    *p = (T*)q;
    return GA_OK;
}

// Releases one allocation made by dalloc early (e.g. a work list that is rebuilt).
void dfree(ga_graph* g, void* p);

// Makes g's device current for the calling thread.
ga_status use_device(const ga_graph* g);

// Frees the loop state (CUDA graphs, pinned buffers) of g.
void destroy_loops(ga_graph* g);

// Refuses (GA_ERR_CUDA) while g's stream is being captured: what a handle builds and keeps must not become part of a
// graph, where it would not exist until the graph runs.
ga_status not_captured(const ga_graph* g);
// Builds the index (once) and the work lists for the current options (idempotent; refuses under capture).
ga_status prepare(ga_graph* g);
// prepare, and the work prefix that cuts shards.
ga_status prepare_shards(ga_graph* g);
// What the pass of an _async call needs. The call may be captured on a handle that is prepared, or that has been
// counted without the index: what is missing then is built beside the capture.
ga_status prepare_enqueued(ga_graph* g, bool shards);
// Work queues for a pass being captured: no other pass's. Allocated 64 at a time, beside the capture.
ga_status captured_work(ga_graph* g, ga_work** work);

// Picks the count kernel for GA_OPT_TC_KERNEL = 0 from the graph's degree-distribution signature (cached per
// signature; times both kernels once for a new one). Called by ga_graph_prepare.
ga_status autotune(ga_graph* g);
// prepare + autotune (GA_OPT_TC_KERNEL = 0): what every synchronous entry point does first.
ga_status ready(ga_graph* g);

// In-place exclusive scan of n uint64 values on g's stream.
ga_status scan_u64(ga_graph* g, unsigned long long* data, uint64_t n);

// Frees the loop state and its device buffers (the next loop call rebuilds them).
void reset_loops(ga_graph* g);

// The core numbers of g (device, n entries, valid until the next loop call): those of the last core loop when no
// other loop has run since, else from a new run of the core loop.
ga_status core_numbers(ga_graph* g, const uint32_t** d_core, uint32_t* kmax);
// The triangle incidence lists of g (device): for every vertex v the other two corners of each triangle through v
// in inc[inc_ptr[v] .. inc_ptr[v+1]), (middle, highest) in the list of a triangle's lowest corner. Built when
// missing, whatever GA_OPT_UPDATE_MODE says; *T = triangles.
ga_status incidence_lists(ga_graph* g, const uint2** inc, const unsigned long long** inc_ptr, uint64_t* T);

// Batches: g is the disjoint union of `count` graphs, graph s owning vertices [d_off[s], d_off[s+1]) (device array
// of count + 1 offsets that outlives g's use of it). set_segments installs the per-graph loop state once;
// count_segments gives every graph's triangle count; peel_segments peels all graphs in one loop, each exactly as if
// alone (any output may be null; removed_round has n entries in union order).
ga_status set_segments(ga_graph* g, const unsigned long long* d_off, uint32_t count);
ga_status count_segments(ga_graph* g, uint64_t* triangles);
ga_status peel_segments(ga_graph* g, uint64_t num, uint64_t den, uint64_t* triangles, ga_peel_result* res,
                        uint32_t* status, uint32_t* removed_round);

}  // namespace ga
