// ga_tc.cuh - interface of the triangle kernels to the other translation units (peeling, cores, batching).
#pragma once
#include "ga_device.cuh"

namespace ga {

// COUNT: T only. VSUP: per-vertex counts. ESUP: per-edge counts. LIST: every triangle written once into the
// incidence lists of its three corners (the other two corners of each triangle through v, in inc[inc_ptr[v] ..]).
enum TcMode { TC_COUNT = 0, TC_VSUP = 1, TC_ESUP = 2, TC_LIST = 3 };

// The index the hash kernel reads (ga_graph.cu; everything by place).
struct TcIndex {
    const uint32_t *vrank, *order, *dout, *work;
    const uint2* pos;
    const uint32_t *colr, *osrc;
    const unsigned long long* in_rng;
};

inline TcIndex tc_index(const ga_graph* g) {
    return TcIndex{g->vrank, g->order, g->dout, g->work, g->pos, g->colr, g->osrc, g->in_rng};
}

// Outputs of one triangle pass. `total` (device) receives T; `vsup` (n counters of type CT) the per-vertex counts;
// `esup` (m) the per-edge counts; `alive` (n bytes, optional) restricts the pass to the induced subgraph;
// `inc`/`inc_ptr`/`fill` the incidence lists of TC_LIST (fill: n zeroed cursors).
template <class CT>
struct TcArgs {
    unsigned long long* total = nullptr;
    unsigned long long* host_total = nullptr;   // page-locked slot that receives T as well (optional)
    CT* vsup = nullptr;
    uint32_t* esup = nullptr;
    const uint8_t* alive = nullptr;
    uint2* inc = nullptr;
    const unsigned long long* inc_ptr = nullptr;
    uint32_t* fill = nullptr;
    uint32_t* overflow = nullptr;   // TC_LIST: entries that found their list full (must stay 0)
    // set by the launchers (alive is by place for the kernels on the index)
    TcIndex ix = {};
    ga_sync* sync = nullptr;        // where the blocks of a synchronous call meet (null: they add to *total)
    ga_work* work = nullptr;        // this pass's work queues
    uint32_t* esupk = nullptr;      // ESUP: supports by padded position in colr, zeroed
    bool bitmaps = false;           // heavy anchors may use bitmaps
    // shard `shard` of `nshards` (0 = the whole graph): equal parts of the probe work (hash kernel) or of the edges
    // (plain kernel); the shards of a graph partition its triangles
    uint32_t shard = 0, nshards = 0;
    bool enqueued = false;   // an _async call: the pass may run at any time, beside others of the handle
};

// One triangle pass on g's stream (asynchronous). total is written whole; zero_outputs: clear vsup/esup first.
template <int MODE, bool ALIVE, class CT>
ga_status run_tc(ga_graph* g, const TcArgs<CT>& a, bool zero_outputs);

}  // namespace ga
