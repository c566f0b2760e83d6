// ga_loops.cu - device-resident round loops: triangle-density batch peeling and the (k, triangle)-core decomposition.
//
// Both loops remove a FRONTIER of vertices per round and keep tri[v] (triangles of v inside the alive subgraph)
// up to date by decrements instead of recounting:
//   * batch peeling (densest.h:138-160, batch_peel_loop densest.h:279-303): frontier = alive v with
//     tri[v] * nalive * den <= 3 * (den + num) * T (the integer rule of mark_peel, kernels.cuh:443-459);
//     the best density is tracked on the device with peel_improves' strict rule (densest.h:76-78);
//   * cores (core_decomp_loop_inc, dsg.h:724-751): k = max(k, min over alive of tri); frontier = alive v with
//     tri[v] <= k, core[v] = k (core_find_frontier, kernels.cuh:549-562; level rule and proof dsg.h:666-680).
// After a frontier F is chosen, exactly the triangles with a corner in F and all corners alive-or-in-F disappear.
// k_frontier_update enumerates, for every x in F, every triangle through x: with N(x) = N+(x) ∪ In(x) (out-list
// and in-list of the oriented CSR) the triangles through x are {x, y, w} for y in N(x), w in N+(y) ∩ N(x), each
// found exactly once from x (x lowest: y = middle; x middle: y = lowest; x highest: y = lowest). The triangle is
// handled only by its smallest-id frontier corner (the owner rule of core_update_frontier, kernels.cuh:607), which
// subtracts 1 from tri[] of its alive corners and counts it as destroyed (T -= destroyed). This reproduces the
// recount of the reference's loops exactly, so rounds, removed_round[], best density and core[] are bit-identical.
//
// Round structure (one kernel boundary = one grid-wide barrier, no host sync):
//   peel : k_peel_mark -> k_frontier_update
//   core : k_core_min  -> k_core_mark -> k_frontier_update
// The alive set is kept as a compacted id list (double-buffered, parity on the device), so late rounds scan only the
// survivors. The last block of the update kernel advances the round and decides whether to continue; the frontier
// (double-buffered by round parity) is retired by the next round's first kernel. In GA_OPT_LOOP_MODE 2
// the round is the body of a CUDA graph conditional WHILE node (cudaGraphSetConditional from the tail), so the
// whole loop is one graph launch; mode 1 launches the same kernels round by round and reads the 100-byte round state
// back after each (the reference's host loop with its one sync per round). Mode 0 is mode 2, except for core loops that
// one cluster can hold from the start (run_loop).
//
// Small core rounds: most of the thousands of core rounds of a power-law graph are small (R-MAT scale 22: 9,543
// rounds, nine in ten with at most 131,072 alive vertices, the median removing three), and a grid round of three
// dependent kernels costs tens of microseconds of launch and drain latency whatever its size. The body of a captured
// core round therefore starts with k_core_small_rounds (a loop that fits from the start launches it directly), ONE
// cluster (16 CTAs of 1,024 threads, 8 where 16 cannot be co-scheduled) that keeps the whole loop state in its shared
// memory and runs consecutive rounds itself with cluster barriers between the phases, for as long as the alive list
// fits its slots and the next round reads at most kSmallWork incidence entries. The first round that does not fit is
// left untouched for the grid kernels that follow in the same body; the loop decisions and every result are the grid
// round's, so the output is unchanged.
#include <cooperative_groups.h>

#include <algorithm>

#include "ga_device.cuh"
#include "ga_tc.cuh"

namespace ga {

constexpr uint32_t kChunk = 256;     // neighbours of a frontier vertex per update item (enumeration update)
constexpr uint32_t kListChunk = 512;    // incidence entries of a frontier vertex per update item (list update)
constexpr int kUpdWarps = 8;

enum LoopKind { LOOP_PEEL = 0, LOOP_CORE = 1 };

// Device round state (one struct, read back whole by the host-driven mode).
struct LoopScalars {
    unsigned long long T, nalive, num, den;
    unsigned long long best_num, best_den, destroyed;
    uint32_t round, best_round, parity, max_rounds;
    uint32_t alive_count[2];
    uint32_t fcount, nitems, kcur, kround, min_tri;
    uint32_t fprev;   // frontier size of the previous round (retired by the next round's first kernel)
    uint32_t status, done_blocks, cont;
    uint32_t iters;   // rounds started, counted independently of the tail (loop bound of last resort)
};

// status codes written by the device
enum : uint32_t { LS_OK = 0, LS_NO_PROGRESS = 1, LS_ROUND_LIMIT = 2, LS_LEVEL_DOWN = 3, LS_OVER_REMOVED = 4,
                  LS_ARITH = 5 };

// Per-graph state when one loop peels many disjoint graphs at once (a batch): graph s owns vertices
// [off[s], off[s+1]) and has its own T, alive count, threshold, best density, round count and status, exactly as if
// it were peeled alone. count == 0: a single graph (the LoopScalars fields are used instead).
struct Segs {
    uint32_t count = 0;
    const unsigned long long* off = nullptr;          // count + 1
    unsigned long long *T = nullptr, *nalive = nullptr, *removed = nullptr, *destroyed = nullptr;
    unsigned long long *best_num = nullptr, *best_den = nullptr, *T0 = nullptr;
    uint32_t *best_round = nullptr, *rounds = nullptr, *status = nullptr;
};

// Segment of vertex v: the last s with off[s] <= v.
__device__ __forceinline__ uint32_t seg_of(const Segs& sg, uint32_t v) {
    uint32_t lo = 0, hi = sg.count;
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (sg.off[mid] <= v) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// peel_arith_ok (densest.h:65-72) for one graph with n vertices and T0 triangles (eps already range-checked).
__host__ __device__ inline bool peel_arith_fits(unsigned long long n, unsigned long long T0, unsigned long long num,
                                                unsigned long long den) {
    if (T0 >= (1ull << 32)) return false;
    if (n > 0 && T0 > ~0ull / (n * den)) return false;
    if (T0 > ~0ull / (3ull * (den + num))) return false;
    return true;
}

}  // namespace ga

struct ga_loops {
    uint32_t* tri = nullptr;          // n
    uint8_t* state = nullptr;         // n: 0 removed, 1 alive, 2 frontier of this round
    uint32_t* out = nullptr;          // n: removed_round (peel) or core (core)
    uint32_t* alive[2] = {nullptr, nullptr};
    uint32_t* frontier[2] = {nullptr, nullptr};   // n each: the frontier of even / odd rounds
    uint32_t* loc = nullptr;          // n, core loops: local ids of the cluster rounds (all ones outside them)
    uint32_t* item_x = nullptr;       // item capacity
    uint32_t* item_c = nullptr;
    uint64_t item_cap = 0;
    ga::LoopScalars* sc = nullptr;    // device
    uint64_t list_T = 0;              // triangles in the incidence lists, once built
    cudaGraphExec_t exec[2] = {nullptr, nullptr};
    cudaGraph_t graph[2] = {nullptr, nullptr};
    unsigned grid_scan = 1, grid_update = 1, grid_list = 1;
    // triangle incidence lists (built once per graph when memory allows): for every vertex v the other two corners
    // of each triangle through v, in inc[inc_ptr[v] .. inc_ptr[v+1])
    int lists = -1;                    // -1 undecided, 0 enumeration update, 1 incidence-list update
    bool cores_in_out = false;         // out[] holds the core numbers of a finished core loop (kmax in cores_kmax)
    uint32_t cores_kmax = 0;
    uint2* inc = nullptr;
    unsigned long long* inc_ptr = nullptr;   // n+1
    ga::Segs segs;                     // per-graph state of a batch (count 0 for a single graph)
    cudaGraphExec_t exec_seg = nullptr;
    cudaGraph_t graph_seg = nullptr;
};

namespace ga {

// The state a loop starts from, in one pass: every vertex alive, its triangle count (the length of its incidence list
// when the lists exist), and the scalars (total: T, or null for the ends of the lists).
__global__ void __launch_bounds__(256) k_loop_init(uint8_t* __restrict__ state, uint32_t* __restrict__ out,
                                                   uint32_t* __restrict__ alive0, uint32_t* __restrict__ loc,
                                                   const unsigned long long* __restrict__ inc_ptr,
                                                   uint32_t* __restrict__ tri, const unsigned long long* total,
                                                   LoopScalars* sc, uint32_t n, unsigned long long num,
                                                   unsigned long long den, uint32_t max_rounds) {
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
        state[v] = 1;
        out[v] = 0xFFFFFFFFu;
        alive0[v] = (uint32_t)v;
        if (loc) loc[v] = GA_EMPTY;
        if (inc_ptr) tri[v] = (uint32_t)(inc_ptr[v + 1] - inc_ptr[v]);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        LoopScalars s = {};
        s.T = inc_ptr ? inc_ptr[n] / 3 : *total;
        s.nalive = n;
        s.num = num;
        s.den = den;
        s.max_rounds = max_rounds;
        s.alive_count[0] = n;
        s.min_tri = 0xFFFFFFFFu;
        s.cont = n > 0;
        *sc = s;
    }
}

constexpr int kMarkThreads = 256;

// Where the mark kernels' blocks meet: per warp the frontier vertices, survivors and update items, then their bases.
struct MarkShared {
    uint32_t n[3][kMarkThreads / 32], base[3];
};

// Appends this block's vertices (one per thread, every thread calls it): frontier vertices `rem` with their update
// items (ceil(|Tri(v)| / kListChunk) slices of v's incidence list, or ceil(deg(v) / kChunk) of its neighbours without
// lists) and survivors `keep` to the next alive list. One atomic per block and list: with one per warp, the first round
// over eight million vertices waited for 750,000 atomics on three addresses (0.55 ms).
__device__ __forceinline__ void append_block(bool rem, bool keep, uint32_t v, const uint32_t* __restrict__ degree,
                                             const unsigned long long* __restrict__ inc_ptr, LoopScalars* sc,
                                             uint32_t* __restrict__ frontier, uint32_t* __restrict__ item_x,
                                             uint32_t* __restrict__ item_c, uint32_t* __restrict__ out_list,
                                             uint32_t* out_count, MarkShared& sh) {
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t br = __ballot_sync(GA_FULL_MASK, rem), bk = __ballot_sync(GA_FULL_MASK, keep);
    uint32_t nc = 0;
    if (rem)
        nc = inc_ptr ? (uint32_t)((inc_ptr[v + 1] - inc_ptr[v] + kListChunk - 1) / kListChunk)
                     : (uint32_t)(((uint64_t)degree[v] + kChunk - 1) / kChunk);
    const uint32_t incl = br ? warp_incl_scan(nc, lane) : 0u;   // br is the same in the whole warp
    if (lane == 31) {
        sh.n[0][w] = __popc(br);
        sh.n[1][w] = __popc(bk);
        sh.n[2][w] = incl;
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        uint32_t sum = 0;
        for (int q = 0; q < kMarkThreads / 32; q++) sum += sh.n[threadIdx.x][q];
        uint32_t* counter = threadIdx.x == 0 ? &sc->fcount : threadIdx.x == 1 ? out_count : &sc->nitems;
        sh.base[threadIdx.x] = sum ? atomicAdd(counter, sum) : 0u;
    }
    __syncthreads();
    uint32_t at[3] = {sh.base[0], sh.base[1], sh.base[2]};
    for (uint32_t q = 0; q < w; q++) {
        at[0] += sh.n[0][q];
        at[1] += sh.n[1][q];
        at[2] += sh.n[2][q];
    }
    const uint32_t below = (1u << lane) - 1;
    if (rem) {
        frontier[at[0] + __popc(br & below)] = v;
        for (uint32_t c = 0; c < nc; c++) {
            item_x[at[2] + incl - nc + c] = v;
            item_c[at[2] + incl - nc + c] = c;
        }
    }
    if (keep) out_list[at[1] + __popc(bk & below)] = v;
    __syncthreads();   // the counts are read before the next tile's replace them
}

// The previous round's frontier leaves for good (state 2 -> 0). Run by the first kernel of a round, before any
// kernel of the round reads state[] of frontier corners.
__device__ __forceinline__ void retire_previous(const LoopScalars* sc, uint8_t* __restrict__ state,
                                                const uint32_t* __restrict__ prev) {
    const uint32_t F = sc->fprev;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < F; i += gridDim.x * blockDim.x) state[prev[i]] = 0;
}

// Peel round, step 1: best-density bookkeeping (peel_improves, densest.h:297) and the mark_peel rule
// (kernels.cuh:448-451) over the alive list. With segments each vertex uses its own graph's T and alive count (the
// per-graph best density is kept by the tail), removals are counted per graph (one atomic per graph per warp), and
// the vertices of a graph that was refused or failed leave the loop silently.
__global__ void __launch_bounds__(kMarkThreads) k_peel_mark(LoopScalars* sc, const uint32_t* __restrict__ tri,
                                                   uint8_t* __restrict__ state, uint32_t* __restrict__ removed_round,
                                                   uint32_t* alive0, uint32_t* alive1, uint32_t* fr0, uint32_t* fr1,
                                                   uint32_t* __restrict__ item_x,
                                                   uint32_t* __restrict__ item_c, const uint32_t* __restrict__ degree,
                                                   const unsigned long long* __restrict__ inc_ptr, Segs sg) {
    const uint32_t p = sc->parity;
    uint32_t* frontier = (sc->round & 1) ? fr1 : fr0;
    retire_previous(sc, state, (sc->round & 1) ? fr0 : fr1);
    const uint32_t* in = p ? alive1 : alive0;
    uint32_t* outl = p ? alive0 : alive1;
    const uint32_t na = sc->alive_count[p];
    const unsigned long long T = sc->T, nalive = sc->nalive, num = sc->num, den = sc->den;
    const unsigned long long rhs = 3ull * (den + num) * T;
    const uint32_t round = sc->round;
    if (!sg.count && blockIdx.x == 0 && threadIdx.x == 0) {
        if (sc->best_den == 0 || T * sc->best_den > sc->best_num * nalive) {
            sc->best_num = T;
            sc->best_den = nalive;
            sc->best_round = round;
        }
    }
    __shared__ MarkShared sh;
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t stride = (uint64_t)gridDim.x * kMarkThreads;
    for (uint64_t i0 = (uint64_t)blockIdx.x * kMarkThreads; i0 < na; i0 += stride) {   // block-uniform
        const uint64_t i = i0 + threadIdx.x;
        const bool valid = i < na;
        const uint32_t v = valid ? in[i] : 0;
        bool rem = false, drop = false;
        uint32_t s = 0;
        if (valid) {
            if (sg.count) {
                s = seg_of(sg, v);
                if (sg.status[s] != LS_OK) {
                    drop = true;
                    state[v] = 0;
                } else {
                    const unsigned long long Ts = sg.T[s], ns = sg.nalive[s];
                    rem = (unsigned long long)tri[v] * ns * den <= 3ull * (den + num) * Ts;
                }
            } else {
                rem = (unsigned long long)tri[v] * nalive * den <= rhs;
            }
            if (rem) {
                state[v] = 2;
                removed_round[v] = round;
            }
        }
        if (sg.count) {   // removals per graph: lanes of the same graph combine into one atomic
            const uint32_t bal = __ballot_sync(GA_FULL_MASK, rem);
            if (bal) {
                const uint32_t peers = __match_any_sync(GA_FULL_MASK, rem ? s : 0xFFFFFFFFu);
                if (rem && lane == (uint32_t)(__ffs(peers) - 1))
                    atomicAdd(&sg.removed[s], (unsigned long long)__popc(peers));
            }
        }
        append_block(rem, valid && !rem && !drop, v, degree, inc_ptr, sc, frontier, item_x, item_c, outl,
                     &sc->alive_count[p ^ 1], sh);
    }
}

// Core round, step 1: minimum of tri over the alive list (core_min_alive_tri, kernels.cuh:484-491).
__global__ void __launch_bounds__(256) k_core_min(LoopScalars* sc, const uint32_t* __restrict__ tri,
                                                  const uint32_t* alive0, const uint32_t* alive1,
                                                  uint8_t* __restrict__ state, const uint32_t* fr0,
                                                  const uint32_t* fr1, cudaGraphConditionalHandle handle,
                                                  int use_handle) {
    if (!sc->cont) {   // the small-round cluster kernel ended the loop in this body: the WHILE node stops
        if (use_handle && blockIdx.x == 0 && threadIdx.x == 0) cudaGraphSetConditional(handle, 0);
        return;
    }
    const uint32_t p = sc->parity;
    retire_previous(sc, state, (sc->round & 1) ? fr0 : fr1);
    const uint32_t* in = p ? alive1 : alive0;
    const uint32_t na = sc->alive_count[p];
    uint32_t mn = 0xFFFFFFFFu;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < na; i += gridDim.x * blockDim.x)
        mn = min(mn, tri[in[i]]);
    mn = __reduce_min_sync(GA_FULL_MASK, mn);
    if ((threadIdx.x & 31) == 0 && mn != 0xFFFFFFFFu) atomicMin(&sc->min_tri, mn);
}

// Core round, step 2: k = max(k, min); frontier = alive with tri <= k, core = k (core_find_frontier,
// kernels.cuh:549-562).
__global__ void __launch_bounds__(kMarkThreads) k_core_mark(LoopScalars* sc, const uint32_t* __restrict__ tri,
                                                   uint8_t* __restrict__ state, uint32_t* __restrict__ core,
                                                   uint32_t* alive0, uint32_t* alive1, uint32_t* fr0, uint32_t* fr1,
                                                   uint32_t* __restrict__ item_x,
                                                   uint32_t* __restrict__ item_c, const uint32_t* __restrict__ degree,
                                                   const unsigned long long* __restrict__ inc_ptr) {
    if (!sc->cont) return;
    const uint32_t p = sc->parity;
    uint32_t* frontier = (sc->round & 1) ? fr1 : fr0;
    const uint32_t* in = p ? alive1 : alive0;
    uint32_t* outl = p ? alive0 : alive1;
    const uint32_t na = sc->alive_count[p];
    const uint32_t k = max(sc->kcur, sc->min_tri);
    if (blockIdx.x == 0 && threadIdx.x == 0) sc->kround = k;
    __shared__ MarkShared sh;
    const uint64_t stride = (uint64_t)gridDim.x * kMarkThreads;
    for (uint64_t i0 = (uint64_t)blockIdx.x * kMarkThreads; i0 < na; i0 += stride) {   // block-uniform
        const uint64_t i = i0 + threadIdx.x;
        const bool valid = i < na;
        const uint32_t v = valid ? in[i] : 0;
        bool rem = false;
        if (valid) {
            rem = tri[v] <= k;
            if (rem) {
                state[v] = 2;
                core[v] = k;
            }
        }
        append_block(rem, valid && !rem, v, degree, inc_ptr, sc, frontier, item_x, item_c, outl,
                     &sc->alive_count[p ^ 1], sh);
    }
}

// Independent bound on the loop: block 0 of the update kernel counts every round started; past max_rounds + 1 the
// loop is forced to stop even if the round bookkeeping were broken (a WHILE node keeps its last condition otherwise).
__device__ __forceinline__ void count_iteration(LoopScalars* sc, cudaGraphConditionalHandle handle, int use_handle) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        const uint32_t it = atomicAdd(&sc->iters, 1u) + 1;
        if (it > sc->max_rounds + 1) {
            atomicMax(&sc->status, (uint32_t)LS_ROUND_LIMIT);
            sc->cont = 0;
            if (use_handle) cudaGraphSetConditional(handle, 0);
        }
    }
}

// The last block of the update kernel to finish closes the round: nalive -= |F|, T -= destroyed, the checks of
// densest.h:298 / dsg.h:744, per-graph closing of a batch, reset of the per-round counters, the alive-list parity
// flip and the loop condition (cudaGraphSetConditional when running as a graph body). The frontier itself is retired
// by the next round's first kernel (retire_previous).
__device__ __forceinline__ void close_round_if_last(LoopScalars* sc, int kind, cudaGraphConditionalHandle handle,
                                                    int use_handle, const Segs& sg) {
    __shared__ bool s_last;
    __shared__ unsigned long long s_alive[32];
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&sc->done_blocks, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const uint32_t F = sc->fcount;
    // every graph of a batch closes its own round (all threads of the last block): removed and destroyed counts,
    // the checks of densest.h:298, then peel_improves for the alive set the next round starts from
    unsigned long long alive = 0;
    if (sg.count) {
        const uint32_t ran = sc->round;
        for (uint32_t s = threadIdx.x; s < sg.count; s += blockDim.x) {
            if (sg.status[s] == LS_OK && sg.nalive[s] > 0) {
                const unsigned long long rem = sg.removed[s], des = sg.destroyed[s];
                uint32_t st = LS_OK;
                if (rem == 0) st = LS_NO_PROGRESS;
                if (rem > sg.nalive[s] || des > sg.T[s]) st = LS_OVER_REMOVED;
                const unsigned long long na = sg.nalive[s] - min(rem, sg.nalive[s]);
                const unsigned long long T = na ? sg.T[s] - min(des, sg.T[s]) : 0ull;   // last round: no update ran
                sg.nalive[s] = na;
                sg.T[s] = T;
                sg.rounds[s] = ran + 1;
                if (st == LS_OK && na > 0 && ran + 1 >= sc->max_rounds) st = LS_ROUND_LIMIT;
                if (st == LS_OK && na > 0 && (sg.best_den[s] == 0 || T * sg.best_den[s] > sg.best_num[s] * na)) {
                    sg.best_num[s] = T;
                    sg.best_den[s] = na;
                    sg.best_round[s] = ran + 1;
                }
                sg.status[s] = st;
                if (st == LS_OK) alive += na;
            }
            sg.removed[s] = 0;
            sg.destroyed[s] = 0;
        }
        alive = warp_sum_u64(alive);
        if ((threadIdx.x & 31) == 0) s_alive[threadIdx.x >> 5] = alive;
        __syncthreads();
        alive = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) alive += s_alive[w];
    }
    if (threadIdx.x != 0) return;
    LoopScalars s = *sc;   // written by earlier kernels of this round and by this kernel's blocks (fenced above)
    uint32_t status = s.status;
    if (sg.count) {
        s.nalive = alive;
    } else {
        if (F == 0 && s.nalive > 0) status = LS_NO_PROGRESS;
        if (F > s.nalive) status = LS_OVER_REMOVED;
        if (s.destroyed > s.T) status = LS_OVER_REMOVED;
        s.T -= F == s.nalive ? s.T : min(s.destroyed, s.T);   // the last round takes what is left (no update ran)
        s.nalive -= min((unsigned long long)F, s.nalive);
    }
    if (kind == LOOP_CORE) {
        if (s.kround < s.kcur) status = LS_LEVEL_DOWN;
        s.kcur = s.kround;
    }
    s.round += 1;
    s.parity ^= 1;
    s.alive_count[s.parity ^ 1] = 0;   // the next round's output list
    s.fprev = F;
    s.fcount = 0;
    s.nitems = 0;
    s.destroyed = 0;
    s.done_blocks = 0;
    s.min_tri = 0xFFFFFFFFu;
    if (status == LS_OK && s.nalive > 0 && s.round >= s.max_rounds) status = LS_ROUND_LIMIT;
    s.status = status;
    s.cont = (status == LS_OK && s.nalive > 0 && s.iters <= s.max_rounds) ? 1u : 0u;
    *sc = s;
    if (use_handle) cudaGraphSetConditional(handle, s.cont);
}

// True when the frontier is everything that was alive: no count is left to update, and every remaining triangle
// goes, so the update has nothing to read (a batch asks per graph, where a graph's last round is one of many). That
// round reads the densest part: 464 M of the 1.57 G incidence entries of R-MAT scale 22's cores.
__device__ __forceinline__ bool last_round(const LoopScalars* sc, const Segs& sg) {
    return !sg.count && sc->fcount == sc->nalive;
}

// Enumerates the triangles through the frontier vertices (see the file comment). One warp per item = up to kChunk
// consecutive entries of the virtual neighbour list N(x) = [N+(x) | In(x)]. Vertices with deg(x) <= kChunk use a
// per-warp shared hash set of their live neighbours; larger ones test an edge {x, w} by binary search in the sorted
// rows N+(x) and N+(w).
__global__ void __launch_bounds__(kUpdWarps * 32) k_frontier_update(
    LoopScalars* sc, const uint32_t* __restrict__ rowptr, const uint32_t* __restrict__ col,
    const uint32_t* __restrict__ degree, TcIndex ix, const uint32_t* __restrict__ item_x,
    const uint32_t* __restrict__ item_c, const uint8_t* __restrict__ state, uint32_t* __restrict__ tri, Segs sg,
    int kind, cudaGraphConditionalHandle handle, int use_handle) {
    constexpr uint32_t kSlots = 2 * kChunk;   // 512 slots, load <= 1/2
    if (!sc->cont) return;
    count_iteration(sc, handle, use_handle);
    constexpr uint32_t kBits = 9;
    __shared__ uint32_t s_key[kUpdWarps][kSlots];
    __shared__ uint32_t s_incl[kUpdWarps][32], s_rb[kUpdWarps][32], s_y[kUpdWarps][32];
    __shared__ uint8_t s_sy[kUpdWarps][32];
    __shared__ unsigned long long s_red[kUpdWarps];
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t* key = s_key[w];
    const uint32_t nitems = last_round(sc, sg) ? 0u : sc->nitems;
    const uint32_t gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    unsigned long long destroyed = 0;
    for (uint32_t it = gwarp; it < nitems; it += nwarps) {
        const uint32_t x = item_x[it], c = item_c[it];
        const uint32_t seg = sg.count ? seg_of(sg, x) : 0u;
        if (sg.count && sg.removed[seg] == sg.nalive[seg]) continue;   // its graph's last round
        const unsigned long long d0 = destroyed;
        const uint32_t xb = rowptr[x], dout = rowptr[x + 1] - xb;
        const uint32_t ib = ix.pos[ix.vrank[x]].x;   // in-edges of x: their sources through the index
        const uint32_t deg = degree[x];
        auto neighbour = [&](uint32_t q) {
            return q < dout ? col[xb + q] : ix.order[ix.osrc[rng_at(ix.in_rng[ib + q - dout]) >> 3]];
        };
        const bool local = deg <= kChunk;
        if (local) {
            for (uint32_t s = lane; s < kSlots; s += 32) key[s] = GA_EMPTY;
            __syncwarp();
            for (uint32_t q = lane; q < deg; q += 32) {
                const uint32_t y = neighbour(q);
                if (state[y] == 0) continue;
                uint32_t h = hash_slot(y, kBits);
                while (atomicCAS(&key[h], GA_EMPTY, y) != GA_EMPTY) h = (h + 1) & (kSlots - 1);
            }
            __syncwarp();
        }
        const uint32_t q0 = c * kChunk, q1 = min(deg, q0 + kChunk);
        for (uint32_t qb = q0; qb < q1; qb += 32) {
            const uint32_t q = qb + lane;
            uint32_t d = 0, rb = 0, y = 0;
            uint8_t sy = 0;
            if (q < q1) {
                y = neighbour(q);
                sy = state[y];
                if (sy) {
                    rb = rowptr[y];
                    d = rowptr[y + 1] - rb;
                }
            }
            const uint32_t incl = warp_incl_scan(d, lane);
            const uint32_t tot = __shfl_sync(GA_FULL_MASK, incl, 31);
            s_incl[w][lane] = incl;
            s_rb[w][lane] = rb;
            s_y[w][lane] = y;
            s_sy[w][lane] = sy;
            __syncwarp();
            uint32_t owner = 0;
            for (uint32_t p = lane; p < tot; p += 32) {
                while (s_incl[w][owner] <= p) owner++;
                const uint32_t wv = col[s_rb[w][owner] + (p - (owner ? s_incl[w][owner - 1] : 0u))];
                bool hit = false;
                if (local) {
                    uint32_t h = hash_slot(wv, kBits);
                    for (;;) {
                        const uint32_t kk = key[h];
                        if (kk == wv) { hit = true; break; }
                        if (kk == GA_EMPTY) break;
                        h = (h + 1) & (kSlots - 1);
                    }
                } else if (wv != x && state[wv] != 0) {
                    const uint32_t j = lower_bound_u32(col, xb, xb + dout, wv);
                    hit = j < xb + dout && col[j] == wv;
                    if (!hit) {
                        const uint32_t wb = rowptr[wv], we = rowptr[wv + 1];
                        const uint32_t j2 = lower_bound_u32(col, wb, we, x);
                        hit = j2 < we && col[j2] == x;
                    }
                }
                if (hit) {
                    const uint32_t yv = s_y[w][owner];
                    const uint8_t syv = s_sy[w][owner], sw = state[wv];
                    const bool owned = !((syv == 2 && yv < x) || (sw == 2 && wv < x));
                    if (owned) {
                        destroyed++;
                        if (syv == 1) red_add(&tri[yv], 0xFFFFFFFFu);
                        if (sw == 1) red_add(&tri[wv], 0xFFFFFFFFu);
                    }
                }
            }
            __syncwarp();
        }
        if (sg.count) {   // per-graph count of destroyed triangles
            const unsigned long long t = warp_sum_u64(destroyed - d0);
            if (lane == 0 && t) atomicAdd(&sg.destroyed[seg], t);
        }
    }
    destroyed = warp_sum_u64(destroyed);
    if (lane == 0) s_red[w] = destroyed;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long t = 0;
        for (int i = 0; i < kUpdWarps; i++) t += s_red[i];
        if (t) atomicAdd(&sc->destroyed, t);
    }
    close_round_if_last(sc, kind, handle, use_handle, sg);
}

// Incidence-list update over items of up to kListChunk entries (y, w) of frontier vertex x's list, read coalesced. The
// triangle {x, y, w} still exists iff y and w are alive or in the frontier; it is handled by its smallest-id frontier
// corner (kernels.cuh:607), which subtracts 1 from tri[] of its alive corners and counts it as destroyed. Over a whole
// run every triangle is read at most three times (once per corner).
// A warp takes up to 32 items at a time - one per lane, their entries flattened by a warp scan like the count's probe
// lists - when there are that many per warp, else fewer: the first rounds of a peeling remove millions of vertices
// whose lists hold some tens of entries, and one item at a time was a chain of four dependent loads for half-empty
// warps (count and peeling of a batch of 256 Holme-Kim graphs: 9.4 ms, 3.5 of them in these updates, against 2.8).
// A lane takes four entries at a time, so that their chains of loads (entry, then two states) overlap: that batch
// 2.82 -> 2.52 ms, count and peeling of a 1.7M-vertex Holme-Kim graph 650 -> 585 us, R-MAT 22 cores 99.3 -> 96.1 ms
// through their 225 grid rounds (two entries 2.60 ms and 600 us, eight like four).
constexpr int kListUnroll = 4;
__global__ void __launch_bounds__(256) k_frontier_update_list(LoopScalars* sc, const uint2* __restrict__ inc,
                                                              const unsigned long long* __restrict__ inc_ptr,
                                                              const uint32_t* __restrict__ item_x,
                                                              const uint32_t* __restrict__ item_c,
                                                              const uint8_t* __restrict__ state,
                                                              uint32_t* __restrict__ tri, Segs sg, int kind,
                                                              cudaGraphConditionalHandle handle, int use_handle) {
    __shared__ unsigned long long s_red[8], s_beg[8][32];
    __shared__ uint32_t s_incl[8][32], s_x[8][32], s_des[8][32];
    if (!sc->cont) return;
    count_iteration(sc, handle, use_handle);
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t nitems = last_round(sc, sg) ? 0u : sc->nitems;
    const uint32_t gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t per = min(32u, max(1u, nitems / nwarps));   // items a warp takes at a time
    unsigned long long destroyed = 0;
    for (uint64_t it0 = (uint64_t)gwarp * per; it0 < nitems; it0 += (uint64_t)nwarps * per) {   // warp-uniform
        uint32_t x = 0, seg = 0, len = 0;
        unsigned long long b = 0;
        if (lane < per && it0 + lane < nitems) {
            x = item_x[it0 + lane];
            seg = sg.count ? seg_of(sg, x) : 0u;
            if (!sg.count || sg.removed[seg] != sg.nalive[seg]) {   // not its graph's last round
                b = inc_ptr[x] + (unsigned long long)item_c[it0 + lane] * kListChunk;
                len = (uint32_t)min(inc_ptr[x + 1] - b, (unsigned long long)kListChunk);
            }
        }
        const uint32_t incl = warp_incl_scan(len, lane), tot = __shfl_sync(GA_FULL_MASK, incl, 31);
        s_incl[w][lane] = incl;
        s_beg[w][lane] = b - (incl - len);
        s_x[w][lane] = x;
        s_des[w][lane] = 0;
        __syncwarp();
        uint32_t owner = 0, end = s_incl[w][0], mine = 0, mine_of = 0;   // triangles of item mine_of not booked yet
        for (uint32_t p0 = lane; p0 < tot; p0 += 32 * kListUnroll) {
            uint2 yw[kListUnroll];
            uint32_t of[kListUnroll];
            uint8_t sy[kListUnroll], sw[kListUnroll];
#pragma unroll
            for (int q = 0; q < kListUnroll; q++) {
                const uint32_t p = p0 + 32 * q;
                of[q] = GA_EMPTY;
                if (p >= tot) continue;
                while (end <= p) end = s_incl[w][++owner];
                of[q] = owner;
                yw[q] = inc[s_beg[w][owner] + p];
            }
#pragma unroll
            for (int q = 0; q < kListUnroll; q++) {
                sy[q] = sw[q] = 0;
                if (of[q] != GA_EMPTY) sy[q] = state[yw[q].x], sw[q] = state[yw[q].y];
            }
#pragma unroll
            for (int q = 0; q < kListUnroll; q++) {
                if (!sy[q] || !sw[q]) continue;                     // past the end, or destroyed in an earlier round
                const uint32_t xv = s_x[w][of[q]];
                // a smaller frontier corner owns it
                if ((sy[q] == 2 && yw[q].x < xv) || (sw[q] == 2 && yw[q].y < xv)) continue;
                if (of[q] != mine_of) {
                    if (sg.count && mine) atomicAdd(&s_des[w][mine_of], mine);
                    destroyed += mine;
                    mine = 0;
                    mine_of = of[q];
                }
                mine++;
                if (sy[q] == 1) red_add(&tri[yw[q].x], 0xFFFFFFFFu);
                if (sw[q] == 1) red_add(&tri[yw[q].y], 0xFFFFFFFFu);
            }
        }
        destroyed += mine;
        if (sg.count) {   // per-graph count of destroyed triangles, lanes of one graph combined
            if (mine) atomicAdd(&s_des[w][mine_of], mine);
            __syncwarp();
            const uint32_t d = s_des[w][lane];
            const uint32_t peers = __match_any_sync(GA_FULL_MASK, d ? seg : GA_EMPTY);
            const uint32_t sum = __reduce_add_sync(peers, d);
            if (d && lane == (uint32_t)__ffs(peers) - 1) atomicAdd(&sg.destroyed[seg], (unsigned long long)sum);
        }
        __syncwarp();
    }
    destroyed = warp_sum_u64(destroyed);
    if (lane == 0) s_red[w] = destroyed;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long t = 0;
        for (int i = 0; i < 8; i++) t += s_red[i];
        if (t) atomicAdd(&sc->destroyed, t);
    }
    close_round_if_last(sc, kind, handle, use_handle, sg);
}

// ---- core rounds of at most 131,072 alive vertices, in one thread block cluster ------------------------------------
// R-MAT scale 22 runs 9,300 such rounds one after the other, each reading some 20-35K incidence entries of two to four
// frontier vertices, so a round is bound by latency and by what 16 SMs can do with scattered accesses. It is kept to
// two cluster barriers and one chain of global loads (incidence entry -> local id), the rest in shared memory:
//   * alive vertex i of the list the cluster takes over gets local id i, held by CTA i % C in slot i / C: its triangle
//     count, the start and the length of its incidence list. loc[v] maps a vertex to its local id (~0: not alive).
//   * every CTA keeps a copy of all local vertices' states (2 bits each: alive, frontier, removed). The copies stay
//     equal without communication, because every CTA sees the whole frontier.
//   * level: a CTA finds the minimum of its own counts and its candidates (counts at or below max(level, own minimum))
//     and writes both into an inbox of every CTA. After one cluster barrier every CTA has all minima and candidate
//     lists, so all compute the same level, frontier and size of the round, and mark it in their own copy.
//   * update: warps read slices of the frontier's lists. A round's decrements fall on about a thousand vertices, some
//     forty each, and a decrement of another CTA's count costs an SM 3.3 cycles a lane, against 0.3 for one in its own
//     shared memory (1.4 for one in L2), so a CTA first sums its decrements by vertex in a small hash table and then
//     sends each sum once (red.shared::cluster); they are complete at the second barrier. The local ids are read
//     through L1: a round's entries name each vertex many times.
// R-MAT 22 cores: 235 ms with the round's state in global memory, 147 with every decrement sent on its own, 96 as it is
// (9,318 rounds in the cluster, some 18,000 cycles each: 8,400 the update, the rest barriers, pushes and scans).
constexpr uint32_t kSmallThreads = 1024;     // threads per CTA of the cluster
constexpr uint32_t kSmallSlots = 8192;       // local vertices per CTA (8 per thread): 131,072 with 16 CTAs
constexpr uint32_t kSmallWork = 1u << 20;    // incidence entries a round may read in the cluster
constexpr uint32_t kSmallMaxCtas = 16;
// The candidates a round can have - each CTA publishes up to kSmallFront / C of its own, so a round with 65 on one of
// 16 CTAs already goes to the grid - and the slots of a CTA's table of decrements: with 2,048 and 4,096 the CTA left 28
// KB of L1, a fraction of the lines a round's local ids lie in, with these 60 KB (R-MAT 22 cores 105.5 -> 98.9 ms; 640
// candidates send rounds of the 8,298-vertex graph to the grid, 1,024 slots are too few for the thousand vertices a
// round touches: 103.2 ms).
constexpr uint32_t kSmallFront = 1024;
constexpr uint32_t kSmallSums = 2048;
constexpr uint32_t kSmallSumsBits = 11, kSmallSumsTries = 8;
constexpr uint32_t kSmallDead = 0xFFFFFFFFu; // count of a removed (or unused) slot

// A frontier candidate: local id, incidence list (start: 34 bits, the upper two beside the length, which is capped -
// a round with a capped list is over kSmallWork and never read here).
struct alignas(16) SmallEntry {
    uint32_t lid, len_hi, beg_lo, pad;
};
constexpr uint32_t kSmallLenMask = 0x3FFFFFFFu;
constexpr uint32_t kSmallPrefetch = 1u << 15;   // entries of a candidate's list brought to L2
struct SmallHead {    // a CTA's minimum count and number of candidates
    uint32_t mn, count;
};
struct SmallShared {
    uint32_t tri[kSmallSlots];
    uint32_t beg_lo[kSmallSlots];
    uint32_t len_hi[kSmallSlots];
    uint32_t st[kSmallSlots * kSmallMaxCtas / 16];   // 2 bits per local vertex: 1 alive, 2 frontier, 0 removed
    uint32_t sum_key[kSmallSums];                    // local id (GA_EMPTY: free) ...
    uint32_t sum_cnt[kSmallSums];                    // ... and its decrements in this round
    SmallEntry inbox[kSmallFront];                   // every CTA's candidates, this CTA's own among them
    SmallHead head[kSmallMaxCtas];
    uint16_t front[kSmallFront];                     // inbox positions of the round's frontier
    uint32_t flid[2][kSmallFront];                   // its local ids, by round parity (retired in the next round)
    uint32_t wmin[kSmallThreads / 32], wwork[kSmallThreads / 32];
    unsigned long long destroyed;                    // triangles this CTA destroyed since the kernel started
    uint32_t count, survivors;
};
static_assert(sizeof(SmallShared) <= 227 * 1024, "must fit an SM's shared memory");

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t remote_addr(uint32_t addr, uint32_t cta) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(cta));
    return r;
}
__device__ __forceinline__ void remote_sub(uint32_t addr, uint32_t v) {
    asm volatile("red.relaxed.cluster.shared::cluster.add.u32 [%0], %1;" ::"r"(addr), "r"(0u - v) : "memory");
}

// One decrement of local vertex `lid`: summed in the CTA's table, or sent at once when its bucket run is full.
__device__ __forceinline__ void small_dec(SmallShared& s, uint32_t tri0, uint32_t lid, uint32_t C, uint32_t cbits) {
    uint32_t h = hash_slot(lid, kSmallSumsBits);
    for (uint32_t t = 0; t < kSmallSumsTries; t++) {
        uint32_t key = *(volatile uint32_t*)&s.sum_key[h];
        if (key == GA_EMPTY) key = atomicCAS(&s.sum_key[h], GA_EMPTY, lid);
        if (key == GA_EMPTY || key == lid) {
            atomicAdd(&s.sum_cnt[h], 1u);
            return;
        }
        h = (h + 1) & (kSmallSums - 1);
    }
    remote_sub(remote_addr(tri0 + 4 * (lid >> cbits), lid & (C - 1)), 1u);
}

// Runs consecutive core rounds (the work of k_core_min, k_core_mark, k_frontier_update_list and close_round_if_last
// for LOOP_CORE) inside one cluster of C CTAs while the alive list fits the CTAs' slots, a round reads at most
// kSmallWork incidence entries and no CTA has more than kSmallFront / C candidates; returns at the first round that is
// larger (untouched, for the grid kernels, which find tri[], state[] and the alive list as if they had run the rounds
// before), when the loop ends (the WHILE condition is set to 0) or at a status other than LS_OK. Every decision is
// computed by every thread from values all CTAs hold identically, so all CTAs leave in the same round.
__global__ void __launch_bounds__(kSmallThreads, 1) k_core_small_rounds(
    LoopScalars* sc, uint32_t* __restrict__ tri, uint8_t* __restrict__ state, uint32_t* __restrict__ core,
    uint32_t* alive0, uint32_t* alive1, const uint32_t* fr0, const uint32_t* fr1, uint32_t* loc,
    const uint2* __restrict__ inc, const unsigned long long* __restrict__ inc_ptr,
    cudaGraphConditionalHandle handle, int use_handle) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    extern __shared__ __align__(16) unsigned char small_raw[];
    SmallShared& s = *reinterpret_cast<SmallShared*>(small_raw);
    const uint32_t C = cluster.num_blocks(), rank = cluster.block_rank(), cbits = 31 - __clz(C);
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t tid = rank * kSmallThreads + threadIdx.x, nthr = C * kSmallThreads;
    const uint32_t gwarp = warp * C + rank, nwarps = nthr >> 5;   // consecutive slices go to different CTAs
    const bool writer = tid == 0;
    const uint32_t room = kSmallFront >> cbits;   // candidates per CTA
    // the state the grid kernels (or the loop's set-up) left; nothing writes it until the cluster leaves
    const uint32_t p = sc->parity, na0 = sc->alive_count[p];
    const uint32_t max_rounds = sc->max_rounds;
    uint32_t cont = sc->cont, round = sc->round, kcur = sc->kcur, status = sc->status, iters = sc->iters;
    unsigned long long nalive = sc->nalive;
    if (!cont) {   // the loop is over: the WHILE node must stop whoever cleared `cont`
        if (writer && use_handle) cudaGraphSetConditional(handle, 0);
        return;
    }
    if (na0 > kSmallSlots * C) return;
    uint32_t* in = p ? alive1 : alive0;
    uint32_t* outl = p ? alive0 : alive1;
    {   // the previous grid round's frontier leaves for good (the grid kernels do it again: idempotent)
        const uint32_t* prev = (round & 1) ? fr0 : fr1;
        const uint32_t fprev = sc->fprev;
        for (uint32_t i = tid; i < fprev; i += nthr) state[prev[i]] = 0;
    }
    if (threadIdx.x == 0) {
        s.destroyed = 0;
        s.survivors = 0;
        s.count = 0;
    }
    for (uint32_t h = threadIdx.x; h < kSmallSums; h += kSmallThreads) {
        s.sum_key[h] = GA_EMPTY;
        s.sum_cnt[h] = 0;
    }
    for (uint32_t w = threadIdx.x; w < kSmallSlots * C / 16; w += kSmallThreads) {
        const uint32_t left = na0 > 16 * w ? na0 - 16 * w : 0;   // local vertices of this word: all alive
        s.st[w] = left >= 16 ? 0x55555555u : 0x55555555u & ((1u << (2 * left)) - 1);
    }
    for (uint32_t slot = threadIdx.x; slot < kSmallSlots; slot += kSmallThreads) {
        const uint32_t i = slot * C + rank;
        uint32_t t = kSmallDead, lh = 0;
        unsigned long long b = 0;
        if (i < na0) {
            const uint32_t v = in[i];
            t = tri[v];
            b = inc_ptr[v];
            lh = (uint32_t)min(inc_ptr[v + 1] - b, (unsigned long long)kSmallLenMask) | (uint32_t)(b >> 32) << 30;
            loc[v] = i;
        }
        s.tri[slot] = t;
        s.beg_lo[slot] = (uint32_t)b;
        s.len_hi[slot] = lh;
    }
    __threadfence();
    cluster.sync();   // loc[] is complete, and every CTA runs before its shared memory is written from others
    const uint32_t tri0 = smem_addr(s.tri);
    uint32_t done = 0, fprev = 0;   // rounds run here, the last one's frontier
    uint32_t fv = 0;   // the vertex of this thread's frontier entry, when this CTA holds it
    // the last round's frontier (F vertices at level k): out of the states, core numbers written by the owners
    auto retire = [&](uint32_t F, uint32_t k) {
        for (uint32_t f = threadIdx.x; f < F; f += kSmallThreads) {
            const uint32_t lid = s.flid[(done & 1) ^ 1][f];
            atomicAnd(&s.st[lid >> 4], ~(3u << (2 * (lid & 15))));
            if ((lid & (C - 1)) == rank) {
                const uint32_t v = f < kSmallThreads ? fv : in[lid];   // read when the frontier was marked
                core[v] = k;
                state[v] = 0;
            }
        }
    };
    while (cont) {
        // this CTA's minimum (scan of 8 slots per thread) and candidates, published to every CTA
        const uint4 t0 = reinterpret_cast<const uint4*>(s.tri)[threadIdx.x];
        const uint4 t1 = reinterpret_cast<const uint4*>(s.tri)[threadIdx.x + kSmallThreads];
        const uint32_t mine = min(min(min(t0.x, t0.y), min(t0.z, t0.w)), min(min(t1.x, t1.y), min(t1.z, t1.w)));
        const uint32_t wm = __reduce_min_sync(GA_FULL_MASK, mine);
        if (lane == 0) s.wmin[warp] = wm;
        __syncthreads();
        const uint32_t bmin = __reduce_min_sync(GA_FULL_MASK, s.wmin[lane]);
        const uint32_t thr = max(kcur, bmin);
        if (bmin != kSmallDead && mine <= thr) {
            const uint32_t ts[8] = {t0.x, t0.y, t0.z, t0.w, t1.x, t1.y, t1.z, t1.w};
#pragma unroll
            for (int j = 0; j < 8; j++) {
                if (ts[j] > thr) continue;
                const uint32_t slot = 4 * threadIdx.x + (j & 3) + (j >> 2) * 4 * kSmallThreads;
                const uint32_t at = atomicAdd(&s.count, 1u);
                if (at >= room) continue;   // counted: the round goes to the grid kernels
                const uint32_t lh = s.len_hi[slot], bl = s.beg_lo[slot];
                s.inbox[rank * room + at] = SmallEntry{slot * C + rank, lh, bl, 0};
                // its list is wanted in this round or in one soon after: from DRAM to L2 while the level is agreed on
                const uint32_t bytes = min(lh & kSmallLenMask, kSmallPrefetch) * 8u & ~15u;
                const char* list = (const char*)(inc + ((unsigned long long)(lh >> 30) << 32 | bl));
                if (bytes)
                    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"((uint64_t)list & ~15ull), "r"(bytes)
                                 : "memory");
            }
        }
        __syncthreads();
        const uint32_t mycount = s.count;
        for (uint32_t i = threadIdx.x; i < min(mycount, room) * C; i += kSmallThreads) {   // (candidate, CTA)
            if ((i & (C - 1)) == rank) continue;
            const SmallEntry* at = &s.inbox[rank * room + (i >> cbits)];
            const SmallEntry e = *at;
            asm volatile("st.shared::cluster.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(
                             remote_addr(smem_addr(at), i & (C - 1))),
                         "r"(e.lid), "r"(e.len_hi), "r"(e.beg_lo), "r"(0u)
                         : "memory");
        }
        if (threadIdx.x < C)
            asm volatile("st.shared::cluster.v2.u32 [%0], {%1, %2};" ::"r"(
                             remote_addr(smem_addr(&s.head[rank]), threadIdx.x)),
                         "r"(bmin), "r"(mycount)
                         : "memory");
        cluster.barrier_arrive();
        retire(fprev, kcur);   // while the others arrive
        fprev = 0;
        cluster.barrier_wait();
        // level, frontier and size of the round: the same in every warp of the cluster
        if (threadIdx.x == 0) s.count = 0;
        const SmallHead h = lane < C ? s.head[lane] : SmallHead{kSmallDead, 0};
        const uint32_t gmin = __reduce_min_sync(GA_FULL_MASK, h.mn);
        const uint32_t k = max(kcur, gmin);
        // every count <= k is a candidate of its CTA exactly when the CTA's minimum is <= k
        const uint32_t cnt = h.mn <= k && h.mn != kSmallDead ? h.count : 0u;
        if (__any_sync(GA_FULL_MASK, cnt > room)) break;   // the grid kernels take this round
        const uint32_t incl = warp_incl_scan(cnt, lane);
        const uint32_t F = __shfl_sync(GA_FULL_MASK, incl, 31);
        const uint32_t taking = __ballot_sync(GA_FULL_MASK, cnt != 0);
        uint32_t* flid = s.flid[done & 1];
        // the frontier's inbox positions, in order. Up to 32 vertices (almost every round) every warp finds them for
        // itself; more are spread over the block.
        const bool wide = F > 32;
        SmallEntry e = {0, 0, 0, 0};
        uint32_t work = 0;   // capped lengths: a sum over at most kSmallFront lists fits 32 bits
        for (uint32_t f0 = wide ? 32 * warp : 0; f0 < F; f0 += kSmallThreads) {   // warp-uniform
            const uint32_t f = f0 + lane;
            uint32_t c = 0, before = 0;   // the CTA of candidate f: the last taking one whose range starts at or below f
            for (uint32_t left = taking; left; left &= left - 1) {
                const uint32_t q = __ffs(left) - 1, start = __shfl_sync(GA_FULL_MASK, incl - cnt, q);
                if (start <= f) { c = q; before = start; }
            }
            if (f < F) {
                const uint32_t at = c * room + (f - before);
                e = s.inbox[at];
                work += min(e.len_hi & kSmallLenMask, kSmallWork + 1);
                if (wide || warp == 0) {
                    s.front[f] = (uint16_t)at;
                    flid[f] = e.lid;
                }
            }
        }
        work = __reduce_add_sync(GA_FULL_MASK, work);
        if (wide) {
            if (lane == 0) s.wwork[warp] = work;
            __syncthreads();
            work = __reduce_add_sync(GA_FULL_MASK, min(s.wwork[lane], kSmallWork + 1));
        }
        if (work > kSmallWork) break;    // the grid kernels take this round
        const bool last = F == nalive;   // nothing survives: no count is left to update
        // mark the frontier in this CTA's copy; its owner also takes it out of the counts
        for (uint32_t f = threadIdx.x; f < F; f += kSmallThreads) {
            const uint32_t lid = wide ? flid[f] : e.lid;
            atomicXor(&s.st[lid >> 4], 3u << (2 * (lid & 15)));   // 1 -> 2
            if ((lid & (C - 1)) == rank) {
                s.tri[lid >> cbits] = kSmallDead;
                if (f < kSmallThreads) fv = in[lid];   // in flight during the update
            }
        }
        __syncthreads();
        // update (k_frontier_update_list): each destroyed triangle once, by its smallest frontier corner
        if (!last) {
            const uint32_t per = (work + nthr - 1) / nthr;   // entries per lane
            const uint32_t chunk = 32 * min(max(per, 1u), 8u);
            uint32_t destroyed = 0, base = 0;
            for (uint32_t f0 = 0; f0 < F; f0 += 32) {
                if (wide) {
                    e = SmallEntry{0, 0, 0, 0};
                    if (f0 + lane < F) e = s.inbox[s.front[f0 + lane]];
                }
                const uint32_t len = e.len_hi & kSmallLenMask;
                const uint32_t nc = (len + chunk - 1) / chunk;
                const uint32_t ci = warp_incl_scan(nc, lane);
                const uint32_t tot = __shfl_sync(GA_FULL_MASK, ci, 31);
                // this warp's slices j (numbered over the whole frontier): j = gwarp mod nwarps
                for (uint32_t j = (gwarp - base) & (nwarps - 1); j < tot; j += nwarps) {
                    const uint32_t o = __ffs(__ballot_sync(GA_FULL_MASK, ci > j)) - 1;
                    const uint32_t x = __shfl_sync(GA_FULL_MASK, e.lid, o);
                    const uint32_t xl = __shfl_sync(GA_FULL_MASK, len, o);
                    const uint32_t first = (j - __shfl_sync(GA_FULL_MASK, ci - nc, o)) * chunk;
                    const uint32_t hi = __shfl_sync(GA_FULL_MASK, e.len_hi, o) >> 30;
                    const unsigned long long b = (unsigned long long)hi << 32 | __shfl_sync(GA_FULL_MASK, e.beg_lo, o);
                    const uint2* list = inc + b;
                    const uint32_t end = min(xl, first + chunk);
                    for (uint32_t i = first + lane; i < end; i += 128) {
                        uint2 yw[4];
                        uint32_t ly[4], lw[4];
#pragma unroll
                        for (int q = 0; q < 4; q++)
                            if (i + 32 * q < end) yw[q] = __ldcs(list + i + 32 * q);
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            const bool in_list = i + 32 * q < end;
                            ly[q] = in_list ? __ldca(loc + yw[q].x) : GA_EMPTY;
                            lw[q] = in_list ? __ldca(loc + yw[q].y) : GA_EMPTY;
                        }
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            if (ly[q] == GA_EMPTY || lw[q] == GA_EMPTY) continue;   // removed before the cluster began
                            const uint32_t sy = (s.st[ly[q] >> 4] >> (2 * (ly[q] & 15))) & 3;
                            const uint32_t sw = (s.st[lw[q] >> 4] >> (2 * (lw[q] & 15))) & 3;
                            if (!sy || !sw) continue;
                            if ((sy == 2 && ly[q] < x) || (sw == 2 && lw[q] < x)) continue;
                            destroyed++;
                            if (sy == 1) small_dec(s, tri0, ly[q], C, cbits);
                            if (sw == 1) small_dec(s, tri0, lw[q], C, cbits);
                        }
                    }
                }
                base += tot;
            }
            destroyed = __reduce_add_sync(GA_FULL_MASK, destroyed);
            if (lane == 0 && destroyed) atomicAdd(&s.destroyed, (unsigned long long)destroyed);
            __syncthreads();
            // send the sums and clear the table
            if (threadIdx.x < kSmallSums / 4) {
                uint4* keys = reinterpret_cast<uint4*>(s.sum_key) + threadIdx.x;
                const uint4 kq = *keys;
                if ((kq.x & kq.y & kq.z & kq.w) != GA_EMPTY) {
                    uint4* cnts = reinterpret_cast<uint4*>(s.sum_cnt) + threadIdx.x;
                    const uint4 cq = *cnts;
                    const uint32_t ks[4] = {kq.x, kq.y, kq.z, kq.w}, cs[4] = {cq.x, cq.y, cq.z, cq.w};
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        if (ks[q] != GA_EMPTY)
                            remote_sub(remote_addr(tri0 + 4 * (ks[q] >> cbits), ks[q] & (C - 1)), cs[q]);
                    *keys = make_uint4(GA_EMPTY, GA_EMPTY, GA_EMPTY, GA_EMPTY);
                    *cnts = make_uint4(0, 0, 0, 0);
                }
            }
        }
        cluster.sync();
        // close (close_round_if_last for LOOP_CORE), the same in every thread
        if (F == 0 && nalive > 0) status = LS_NO_PROGRESS;
        if (F > nalive) status = LS_OVER_REMOVED;
        nalive -= min((unsigned long long)F, nalive);
        iters++;
        if (iters > max_rounds + 1) status = LS_ROUND_LIMIT;   // count_iteration's bound
        if (status == LS_OK && nalive > 0 && round + 1 >= max_rounds) status = LS_ROUND_LIMIT;
        cont = (status == LS_OK && nalive > 0 && iters <= max_rounds) ? 1u : 0u;
        kcur = k;
        round++;
        done++;
        fprev = F;
    }
    retire(fprev, kcur);
    // leave: local ids end; with rounds run, the survivors' counts, list and the loop state go back to global memory
    uint32_t* survivors = cluster.map_shared_rank(&s.survivors, 0);
    for (uint32_t s0 = 32 * warp; s0 * C < na0; s0 += kSmallThreads) {   // warp-uniform
        const uint32_t slot = s0 + lane;
        const bool used = slot * C + rank < na0;
        const uint32_t v = used ? in[slot * C + rank] : 0u, t = used ? s.tri[slot] : kSmallDead;
        if (used) loc[v] = GA_EMPTY;
        const bool keep = done && t != kSmallDead;
        const uint32_t bal = __ballot_sync(GA_FULL_MASK, keep);
        uint32_t at = 0;
        if (lane == 0 && bal) at = atomicAdd(survivors, (uint32_t)__popc(bal));
        at = __shfl_sync(GA_FULL_MASK, at, 0);
        if (keep) {
            tri[v] = t;
            outl[at + __popc(bal & ((1u << lane) - 1))] = v;
        }
    }
    __syncthreads();
    if (done && threadIdx.x == 0 && rank != 0 && s.destroyed)
        atomicAdd(cluster.map_shared_rank(&s.destroyed, 0), s.destroyed);
    cluster.sync();   // the sums are complete; no CTA leaves while another may still write its shared memory
    if (writer && done) {
        const unsigned long long T = sc->T, des = s.destroyed;
        if (des > T) status = LS_OVER_REMOVED;
        if (status == LS_OK && s.survivors != (uint32_t)nalive) status = LS_OVER_REMOVED;
        if (status != LS_OK) cont = 0;
        sc->nalive = nalive;
        sc->T = nalive == 0 ? 0ull : T - min(des, T);   // the last round takes what is left
        sc->kcur = kcur;
        sc->kround = kcur;
        sc->round = round;
        sc->parity = p ^ 1;
        sc->alive_count[p] = 0;
        sc->alive_count[p ^ 1] = s.survivors;
        sc->fprev = 0;   // every frontier of these rounds is retired
        sc->iters = iters;
        sc->status = status;
        sc->cont = cont;
        if (!cont && use_handle) cudaGraphSetConditional(handle, 0);
    }
}

// Cluster size for k_core_small_rounds: 16 CTAs where 16 can be co-scheduled, else 8 (0: neither).
static int small_round_cluster(int device) {
    static int cached[64] = {};
    static std::mutex mu;
    if (device < 0 || device >= 64) return 0;
    std::lock_guard<std::mutex> lock(mu);
    if (cached[device]) return cached[device] > 0 ? cached[device] : 0;
    int best = -1;
    cudaFuncSetAttribute(k_core_small_rounds, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    cudaFuncSetAttribute(k_core_small_rounds, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmallShared));
    for (int c : {16, 8}) {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = c;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3(c);
        cfg.blockDim = dim3(kSmallThreads);
        cfg.dynamicSmemBytes = sizeof(SmallShared);
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, k_core_small_rounds, &cfg) == cudaSuccess && clusters > 0) {
            best = c;
            break;
        }
    }
    (void)cudaGetLastError();
    cached[device] = best;
    return best > 0 ? best : 0;
}

static ga_status launch_small_rounds(ga_graph* g, cudaStream_t st, uint32_t ctas, cudaGraphConditionalHandle h,
                                     int use_h) {
    ga_loops* L = g->loops;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ctas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(kSmallThreads);
    cfg.dynamicSmemBytes = sizeof(SmallShared);
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    GA_CUDA(cudaLaunchKernelEx(&cfg, k_core_small_rounds, L->sc, L->tri, L->state, L->out, L->alive[0], L->alive[1],
                               (const uint32_t*)L->frontier[0], (const uint32_t*)L->frontier[1], L->loc,
                               (const uint2*)L->inc, (const unsigned long long*)L->inc_ptr, h, use_h));
    return GA_OK;
}

// Per graph: T0 = (sum of its vertices' triangle counts) / 3, from the ends of its incidence lists when they exist
// (sums = inc_ptr), else from the prefix sums of tri[].
__global__ void k_seg_T(const unsigned long long* __restrict__ sums, Segs sg) {
    for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < sg.count; s += gridDim.x * blockDim.x)
        sg.T0[s] = (sums[sg.off[s + 1]] - sums[sg.off[s]]) / 3;
}

// Per graph: the state a lone batch_peel_loop starts from (densest.h:284-297): peel_arith_ok refusal, alive = n,
// T = T0, and round 0 recorded as the best so far (peel_improves with nothing recorded).
__global__ void k_seg_init(Segs sg, unsigned long long num, unsigned long long den) {
    for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < sg.count; s += gridDim.x * blockDim.x) {
        const unsigned long long n = sg.off[s + 1] - sg.off[s], T0 = sg.T0[s];
        const bool ok = peel_arith_fits(n, T0, num, den);
        sg.status[s] = ok ? LS_OK : LS_ARITH;
        sg.T[s] = T0;
        sg.nalive[s] = ok ? n : 0;
        sg.removed[s] = 0;
        sg.destroyed[s] = 0;
        sg.rounds[s] = 0;
        sg.best_num[s] = ok && n ? T0 : 0;
        sg.best_den[s] = ok && n ? n : 0;
        sg.best_round[s] = 0;
    }
}

// ---- host side --------------------------------------------------------------------------------------------------

// 64-bit words of a batch's results: T0, best_num, best_den, then best_round, rounds, status.
static size_t seg_result_words(size_t graphs) { return 3 * graphs + (3 * graphs + 1) / 2; }

static ga_status make_loops(ga_graph* g) {
    ga_loops* L = new ga_loops();
    g->loops = L;
    const uint32_t n = g->n;
    GA_TRY(dalloc(g, &L->tri, n));
    GA_TRY(dalloc(g, &L->state, n));
    GA_TRY(dalloc(g, &L->out, n));
    GA_TRY(dalloc(g, &L->alive[0], n));
    GA_TRY(dalloc(g, &L->alive[1], n));
    GA_TRY(dalloc(g, &L->frontier[0], n));
    GA_TRY(dalloc(g, &L->frontier[1], n));
    // every vertex enters one frontier per run and brings ceil(deg / kChunk) items
    L->item_cap = (uint64_t)n + (2ull * g->m) / kChunk + 1;
    GA_TRY(dalloc(g, &L->item_x, L->item_cap));
    GA_TRY(dalloc(g, &L->item_c, L->item_cap));
    GA_TRY(dalloc(g, &L->sc, 1));
    if (g->seg_count) {   // per-graph state of a batch
        Segs& sg = L->segs;
        const uint32_t c = g->seg_count;
        sg.count = c;
        sg.off = g->seg_off;
        GA_TRY(dalloc(g, &sg.T, c));
        GA_TRY(dalloc(g, &sg.nalive, c));
        GA_TRY(dalloc(g, &sg.removed, c));
        GA_TRY(dalloc(g, &sg.destroyed, c));
        GA_TRY(dalloc(g, &sg.T0, seg_result_words(c)));   // what a call returns is one block
        sg.best_num = sg.T0 + c;
        sg.best_den = sg.best_num + c;
        sg.best_round = (uint32_t*)(sg.best_den + c);
        sg.rounds = sg.best_round + c;
        sg.status = sg.rounds + c;
    }
    // fixed launch shapes (the graph body is captured once): grid-stride scans, persistent update grid
    int occ = 0;
    GA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_frontier_update, kUpdWarps * 32, 0));
    L->grid_scan = (unsigned)g->sm_count * 8;
    L->grid_update = (unsigned)g->sm_count * (unsigned)std::max(occ, 1);
    GA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_frontier_update_list, 256, 0));
    L->grid_list = (unsigned)g->sm_count * (unsigned)std::max(occ, 1);
    return GA_OK;
}

// The loop state, whole or not at all.
static ga_status ensure_loops(ga_graph* g) {
    if (g->loops) return GA_OK;
    const ga_status s = make_loops(g);
    if (s != GA_OK) reset_loops(g);
    return s;
}

// Releases the captured loop graphs. A captured round holds the addresses of the buffers it was captured with, so
// this runs whenever one of them is replaced (the next loop captures again). An executable graph still running is
// freed by CUDA when it completes.
static void drop_captured(ga_loops* L) {
    for (int k = 0; k < 2; k++) {
        if (L->exec[k]) cudaGraphExecDestroy(L->exec[k]);
        if (L->graph[k]) cudaGraphDestroy(L->graph[k]);
        L->exec[k] = nullptr;
        L->graph[k] = nullptr;
    }
    if (L->exec_seg) cudaGraphExecDestroy(L->exec_seg);
    if (L->graph_seg) cudaGraphDestroy(L->graph_seg);
    L->exec_seg = nullptr;
    L->graph_seg = nullptr;
}

void destroy_loops(ga_graph* g) {
    ga_loops* L = g->loops;
    if (!L) return;
    drop_captured(L);
    delete L;   // device buffers belong to g->allocations
    g->loops = nullptr;
}

void reset_loops(ga_graph* g) {
    ga_loops* L = g->loops;
    if (!L) return;
    cudaStreamSynchronize(g->stream);
    void* bufs[] = {L->tri, L->state, L->out, L->alive[0], L->alive[1], L->frontier[0], L->frontier[1], L->loc,
                    L->item_x, L->item_c, L->sc,
                    L->inc, L->inc_ptr, L->segs.T, L->segs.nalive, L->segs.removed, L->segs.destroyed,
                    L->segs.T0};
    for (void* b : bufs) dfree(g, b);
    destroy_loops(g);
}

static ga_status segment_counts(ga_graph* g);

__global__ void k_widen_counts(const uint32_t* __restrict__ tri, unsigned long long* __restrict__ out, uint32_t n) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v <= n; v += gridDim.x * blockDim.x)
        out[v] = v < n ? tri[v] : 0ull;
}

// T0 of every graph of a batch (tri[] holds the per-vertex counts).
static ga_status segment_counts(ga_graph* g) {
    ga_loops* L = g->loops;
    cudaStream_t st = g->stream;
    Scratch tmp(st);
    unsigned long long* sums = nullptr;
    if (L->lists != 1) {
        GA_TRY(tmp.alloc(&sums, (size_t)g->n + 1));
        k_widen_counts<<<grid_for((uint64_t)g->n + 1, 256), 256, 0, st>>>(L->tri, sums, g->n);
        GA_CUDA(cudaGetLastError());
        GA_TRY(scan_u64(g, sums, (uint64_t)g->n + 1));
    }
    k_seg_T<<<grid_for(L->segs.count, 256), 256, 0, st>>>(sums ? sums : L->inc_ptr, L->segs);
    GA_CUDA(cudaGetLastError());
    return GA_OK;
}

// Fills the lists (inc_ptr and inc allocated, tri[] the vertices' counts).
static ga_status fill_lists(ga_graph* g) {
    ga_loops* L = g->loops;
    cudaStream_t st = g->stream;
    const uint32_t n = g->n;
    Scratch tmp(st);
    uint32_t* fill;   // n cursors + the overflow counter
    GA_TRY(tmp.alloc(&fill, (size_t)n + 1));
    k_widen_counts<<<grid_for((uint64_t)n + 1, 256), 256, 0, st>>>(L->tri, L->inc_ptr, n);
    GA_CUDA(cudaGetLastError());
    GA_TRY(scan_u64(g, L->inc_ptr, (uint64_t)n + 1));
    GA_CUDA(cudaMemsetAsync(fill, 0, ((size_t)n + 1) * 4, st));
    TcArgs<unsigned int> a{};
    a.total = g->d_scalars + 1;
    a.inc = L->inc;
    a.inc_ptr = L->inc_ptr;
    a.fill = fill;
    a.overflow = fill + n;
    GA_TRY((run_tc<TC_LIST, false, unsigned int>(g, a, true)));
    uint32_t overflow = 0;
    if (cudaMemcpyAsync(&overflow, fill + n, 4, cudaMemcpyDeviceToHost, st) != cudaSuccess)
        return fail(GA_ERR_CUDA, "overflow read failed");
    GA_CUDA(cudaStreamSynchronize(st));
    if (overflow) return fail(GA_ERR_DEVICE_CHECK, "triangle listing disagreed with the count (%u entries)", overflow);
    return GA_OK;
}

// Decides the update method once per graph. With GA_OPT_UPDATE_MODE 0 (auto) or 2, the incidence lists are built
// when their 24 * T bytes (plus 8 (n + 1)) can be allocated; auto falls back to the enumeration update otherwise.
// tri[] must hold the per-vertex triangle counts of the whole graph and T0 their total / 3.
static ga_status build_lists(ga_graph* g, uint64_t T0) {
    ga_loops* L = g->loops;
    if (L->lists >= 0) return GA_OK;
    if (g->opt_update_mode == 1 || g->n == 0) { L->lists = 0; return GA_OK; }
    const uint32_t n = g->n;
    const uint64_t entries = 3 * T0;
    const uint64_t need_items = (uint64_t)n + entries / kListChunk + 1;
    ga_status s = dalloc(g, &L->inc_ptr, (size_t)n + 1);
    if (s == GA_OK) s = dalloc(g, &L->inc, entries ? entries : 1);
    uint32_t *ix = nullptr, *ic = nullptr;
    if (s == GA_OK && need_items > L->item_cap) {
        s = dalloc(g, &ix, need_items);
        if (s == GA_OK) s = dalloc(g, &ic, need_items);
    }
    if (s == GA_OK) s = fill_lists(g);
    if (s != GA_OK) {   // no half-made lists: the next call would take them for whole ones
        dfree(g, L->inc_ptr); dfree(g, L->inc); dfree(g, ix); dfree(g, ic);
        L->inc_ptr = nullptr; L->inc = nullptr;
        if (g->opt_update_mode == 2 || s != GA_ERR_OUT_OF_MEMORY) return s;
        clear_error();
        L->lists = 0;
        return GA_OK;
    }
    if (ix) {
        // a loop captured before (its update then enumerated: incidence_lists builds the lists later, for the
        // densest-subgraph stages) points at the old item buffers
        drop_captured(L);
        dfree(g, L->item_x); dfree(g, L->item_c);
        L->item_x = ix; L->item_c = ic; L->item_cap = need_items;
    }
    L->lists = 1;
    L->list_T = T0;
    return GA_OK;
}

// Enqueues one round on `st` (kernel parameters are fixed, everything per-round lives in *sc).
template <int KIND>
static ga_status enqueue_round(ga_graph* g, cudaStream_t st, cudaGraphConditionalHandle h, int use_h) {
    ga_loops* L = g->loops;
    const unsigned long long* inc_ptr = L->lists == 1 ? L->inc_ptr : nullptr;
    const Segs sg = KIND == LOOP_PEEL ? L->segs : Segs{};
    if (KIND == LOOP_PEEL) {
        k_peel_mark<<<L->grid_scan, kMarkThreads, 0, st>>>(L->sc, L->tri, L->state, L->out, L->alive[0], L->alive[1],
                                                  L->frontier[0], L->frontier[1], L->item_x, L->item_c, g->deg,
                                                  inc_ptr, sg);
    } else {
        // the small rounds first, in one cluster; the grid kernels below take the first large one
        const uint32_t ctas = use_h && L->lists == 1 ? (uint32_t)small_round_cluster(g->device) : 0;
        if (ctas) GA_TRY(launch_small_rounds(g, st, ctas, h, 1));
        k_core_min<<<L->grid_scan, 256, 0, st>>>(L->sc, L->tri, L->alive[0], L->alive[1], L->state, L->frontier[0],
                                                 L->frontier[1], h, use_h);
        k_core_mark<<<L->grid_scan, kMarkThreads, 0, st>>>(L->sc, L->tri, L->state, L->out, L->alive[0], L->alive[1],
                                                  L->frontier[0], L->frontier[1], L->item_x, L->item_c, g->deg,
                                                  inc_ptr);
    }
    // the update kernel's last block closes the round and sets the loop condition
    if (L->lists == 1)
        k_frontier_update_list<<<L->grid_list, 256, 0, st>>>(L->sc, L->inc, L->inc_ptr, L->item_x, L->item_c,
                                                               L->state, L->tri, sg, KIND, h, use_h);
    else
        k_frontier_update<<<L->grid_update, kUpdWarps * 32, 0, st>>>(L->sc, g->rowptr, g->col, g->deg, tc_index(g),
                                                                L->item_x, L->item_c, L->state, L->tri, sg, KIND,
                                                                h, use_h);
    GA_CUDA(cudaGetLastError());
    return GA_OK;
}

// Builds (once per graph and loop kind) the CUDA graph: a conditional WHILE node whose body is one round.
template <int KIND>
static ga_status ensure_graph(ga_graph* g) {
    ga_loops* L = g->loops;
    const bool seg = KIND == LOOP_PEEL && L->segs.count > 0;   // a batch peel has its own graph
    cudaGraphExec_t& exec = seg ? L->exec_seg : L->exec[KIND];
    if (exec) return GA_OK;
    cudaGraph_t graph;
    GA_CUDA(cudaGraphCreate(&graph, 0));
    (seg ? L->graph_seg : L->graph[KIND]) = graph;
    cudaGraphConditionalHandle handle;
    GA_CUDA(cudaGraphConditionalHandleCreate(&handle, graph, 1, cudaGraphCondAssignDefault));
    cudaGraphNodeParams params = {};
    params.type = cudaGraphNodeTypeConditional;
    params.conditional.handle = handle;
    params.conditional.type = cudaGraphCondTypeWhile;
    params.conditional.size = 1;
    cudaGraphNode_t node;
    GA_CUDA(cudaGraphAddNode(&node, graph, nullptr, 0, &params));
    cudaGraph_t body = params.conditional.phGraph_out[0];
    if (KIND == LOOP_CORE) (void)small_round_cluster(g->device);   // decided before the capture starts
    cudaStream_t cap;
    GA_CUDA(cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking));
    ga_status s = GA_OK;
    if (cudaStreamBeginCaptureToGraph(cap, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal) !=
        cudaSuccess) {
        s = fail(GA_ERR_CUDA, "cudaStreamBeginCaptureToGraph failed");
    } else {
        s = enqueue_round<KIND>(g, cap, handle, 1);
        cudaGraph_t out = nullptr;
        const cudaError_t e = cudaStreamEndCapture(cap, &out);
        if (s == GA_OK && e != cudaSuccess) s = fail(GA_ERR_CUDA, "cudaStreamEndCapture: %s", cudaGetErrorString(e));
    }
    cudaStreamDestroy(cap);
    GA_TRY(s);
    GA_CUDA(cudaGraphInstantiate(&exec, graph, 0));
    return GA_OK;
}

// Common driver: init (full per-vertex count, state), then the round loop in the selected mode.
template <int KIND>
static ga_status run_loop(ga_graph* g, uint64_t num, uint64_t den, LoopScalars* result) {
    GA_TRY(not_captured(g));
    GA_TRY(ready(g));
    GA_TRY(ensure_loops(g));
    ga_loops* L = g->loops;
    cudaStream_t st = g->stream;
    L->cores_in_out = false;   // out[] is rewritten below
    const uint32_t n = g->n;
    if (KIND == LOOP_CORE && !L->loc) GA_TRY(dalloc(g, &L->loc, n));
    // tri[] = triangles per vertex on the whole graph (uint32 counters; T < 2^32 is checked below): the list lengths
    // when the incidence lists exist (whose size is T's), else one per-vertex triangle pass
    uint64_t T0 = L->list_T;
    if (L->lists != 1) {
        TcArgs<unsigned int> a{};
        a.total = g->d_scalars;
        a.host_total = g->h_scalars;
        a.vsup = L->tri;
        GA_TRY((run_tc<TC_VSUP, false, unsigned int>(g, a, true)));
        GA_CUDA(cudaStreamSynchronize(st));
        T0 = g->h_scalars[0];
    }
    const bool seg = KIND == LOOP_PEEL && L->segs.count > 0;
    if (seg) {
        // a batch: every graph is checked on its own (peel_arith_ok with its own n and T0)
        GA_TRY(segment_counts(g));
        k_seg_init<<<grid_for(L->segs.count, 256), 256, 0, st>>>(L->segs, num, den);
        GA_CUDA(cudaGetLastError());
    } else if (T0 >= (1ull << 32)) {
        return fail(GA_ERR_ARITH, "triangle count %llu >= 2^32: uint32 tri[] counters could overflow",
                    (unsigned long long)T0);
    }
    if (KIND == LOOP_PEEL && !seg) {
        // peel_arith_ok (densest.h:65-72) with the device count as T0
        if (n > 0 && T0 > UINT64_MAX / ((uint64_t)n * den))
            return fail(GA_ERR_ARITH, "tri*nalive*den could overflow uint64");
        if (T0 > UINT64_MAX / (3ull * (den + num))) return fail(GA_ERR_ARITH, "3*(den+num)*T could overflow uint64");
    }
    GA_TRY(build_lists(g, T0));
    const uint64_t cap = g->opt_max_rounds ? (uint64_t)g->opt_max_rounds : (uint64_t)n + 1;
    const uint32_t max_rounds = (uint32_t)std::min<uint64_t>(cap, UINT32_MAX);
    k_loop_init<<<grid_for(n, 256), 256, 0, st>>>(L->state, L->out, L->alive[0],
                                                  KIND == LOOP_CORE ? L->loc : nullptr,
                                                  L->lists == 1 ? L->inc_ptr : nullptr, L->tri, g->d_scalars, L->sc, n,
                                                  num, den, max_rounds);
    GA_CUDA(cudaGetLastError());
    LoopScalars* h_sc = reinterpret_cast<LoopScalars*>(g->h_scalars + 32);   // page-locked
    static_assert(sizeof(LoopScalars) <= 32 * 8, "fits the second half of the handle's slot");
    bool more = true;   // the final state is still to be read
    if (n > 0) {
        const bool graph_mode = g->opt_loop_mode != 1;
        // A core loop whose vertices fit the cluster from the start is mostly one launch of it: where the mode is left
        // to the library, the launches are made here, with a grid round between them where a round is too large, and
        // only a loop that keeps alternating is captured as a graph, which costs more to make and release (about 0.3
        // ms) than such a loop takes
        const uint32_t ctas = KIND == LOOP_CORE && g->opt_loop_mode == 0 && L->lists == 1
                                  ? (uint32_t)small_round_cluster(g->device)
                                  : 0;
        if (ctas && (uint64_t)kSmallSlots * ctas >= n && !L->exec[LOOP_CORE]) {
            for (int i = 0; i < 4 && more; i++) {
                if (i) GA_TRY(enqueue_round<KIND>(g, st, 0, 0));
                GA_TRY(launch_small_rounds(g, st, ctas, 0, 0));
                GA_CUDA(cudaMemcpyAsync(h_sc, L->sc, sizeof(LoopScalars), cudaMemcpyDeviceToHost, st));
                GA_CUDA(cudaStreamSynchronize(st));
                more = h_sc->cont != 0;
            }
        }
        if (!more) {
        } else if (graph_mode) {
            GA_TRY(ensure_graph<KIND>(g));
            GA_CUDA(cudaGraphLaunch(seg ? L->exec_seg : L->exec[KIND], st));
        } else {
            for (uint64_t r = 0;; r++) {
                GA_TRY(enqueue_round<KIND>(g, st, 0, 0));
                GA_CUDA(cudaMemcpyAsync(h_sc, L->sc, sizeof(LoopScalars), cudaMemcpyDeviceToHost, st));
                GA_CUDA(cudaStreamSynchronize(st));
                if (!h_sc->cont) break;
                if (r > (uint64_t)max_rounds + 1) return fail(GA_ERR_ROUND_LIMIT, "host loop bound reached");
            }
        }
    }
    if (more) {
        GA_CUDA(cudaMemcpyAsync(h_sc, L->sc, sizeof(LoopScalars), cudaMemcpyDeviceToHost, st));
        GA_CUDA(cudaStreamSynchronize(st));
    }
    *result = *h_sc;
    switch (result->status) {
        case LS_OK: break;
        case LS_ROUND_LIMIT: return fail(GA_ERR_ROUND_LIMIT, "round cap %u reached", result->max_rounds);
        case LS_NO_PROGRESS: return fail(GA_ERR_DEVICE_CHECK, "no vertex removed in round %u", result->round - 1);
        case LS_LEVEL_DOWN: return fail(GA_ERR_DEVICE_CHECK, "core level decreased in round %u", result->round - 1);
        default: return fail(GA_ERR_DEVICE_CHECK, "removed more vertices than alive (round %u)", result->round - 1);
    }
    return GA_OK;
}

ga_status core_numbers(ga_graph* g, const uint32_t** d_core, uint32_t* kmax) {
    if (!g->loops || !g->loops->cores_in_out) {
        LoopScalars s;
        GA_TRY(run_loop<LOOP_CORE>(g, 0, 1, &s));
        g->loops->cores_in_out = true;
        g->loops->cores_kmax = s.kcur;
    }
    *d_core = g->loops->out;
    *kmax = g->loops->cores_kmax;
    return GA_OK;
}

ga_status incidence_lists(ga_graph* g, const uint2** inc, const unsigned long long** inc_ptr, uint64_t* T) {
    GA_TRY(not_captured(g));
    GA_TRY(ready(g));
    GA_TRY(ensure_loops(g));
    ga_loops* L = g->loops;
    cudaStream_t st = g->stream;
    if (!L->inc && g->n) {
        // per-vertex counts size the lists (the list build's input)
        TcArgs<unsigned int> a{};
        a.total = g->d_scalars;
        a.host_total = g->h_scalars;
        a.vsup = L->tri;
        GA_TRY((run_tc<TC_VSUP, false, unsigned int>(g, a, true)));
        GA_CUDA(cudaStreamSynchronize(st));
        const uint64_t T0 = g->h_scalars[0];
        if (T0 >= (1ull << 32))
            return fail(GA_ERR_ARITH, "triangle count %llu >= 2^32: uint32 tri[] counters could overflow",
                        (unsigned long long)T0);
        // build them even where the loops were told to enumerate; the loops keep the update they had chosen
        const int prev = L->lists;
        const int64_t mode = g->opt_update_mode;
        L->lists = -1;
        g->opt_update_mode = 2;
        const ga_status s = build_lists(g, T0);
        g->opt_update_mode = mode;
        if (s != GA_OK) {
            L->lists = prev;
            return s;
        }
        if (prev == 0) L->lists = 0;
        else if (mode == 1) L->lists = -1;
    }
    *inc = L->inc;
    *inc_ptr = L->inc_ptr;
    *T = 0;
    if (g->n) {
        GA_CUDA(cudaMemcpyAsync(g->h_scalars, L->inc_ptr + g->n, 8, cudaMemcpyDeviceToHost, st));
        GA_CUDA(cudaStreamSynchronize(st));
        *T = g->h_scalars[0] / 3;
    }
    return GA_OK;
}

ga_status set_segments(ga_graph* g, const unsigned long long* d_off, uint32_t count) {
    reset_loops(g);
    g->seg_off = d_off;
    g->seg_count = count;
    return ensure_loops(g);
}

ga_status count_segments(ga_graph* g, uint64_t* triangles) {
    if (!g->seg_count) return fail(GA_ERR_INVALID_ARGUMENT, "graph has no segments");
    GA_TRY(ready(g));
    GA_TRY(ensure_loops(g));
    ga_loops* L = g->loops;
    cudaStream_t st = g->stream;
    TcArgs<unsigned int> a{};
    a.total = g->d_scalars;
    a.vsup = L->tri;
    GA_TRY((run_tc<TC_VSUP, false, unsigned int>(g, a, true)));
    GA_TRY(segment_counts(g));
    GA_CUDA(cudaMemcpyAsync(triangles, L->segs.T0, (size_t)L->segs.count * 8, cudaMemcpyDeviceToHost, st));
    GA_CUDA(cudaStreamSynchronize(st));
    return GA_OK;
}

ga_status peel_segments(ga_graph* g, uint64_t num, uint64_t den, uint64_t* triangles, ga_peel_result* res,
                        uint32_t* status, uint32_t* removed_round) {
    if (!g->seg_count) return fail(GA_ERR_INVALID_ARGUMENT, "graph has no segments");
    LoopScalars s;
    GA_TRY(run_loop<LOOP_PEEL>(g, num, den, &s));
    const Segs& sg = g->loops->segs;
    const uint32_t G = sg.count;
    // T0 and the results are one block on the device (ensure_loops)
    std::vector<unsigned long long> block(seg_result_words(G));
    GA_TRY(download(g, block.data(), sg.T0, block.size() * 8));
    const unsigned long long *T0 = block.data(), *bn = T0 + G, *bd = bn + G;
    const uint32_t *br = (const uint32_t*)(bd + G), *rounds = br + G, *st = rounds + G;
    if (removed_round && g->n) GA_TRY(download(g, removed_round, g->loops->out, (size_t)g->n * 4));
    for (uint32_t i = 0; i < G; i++) {
        if (triangles) triangles[i] = T0[i];
        if (res) res[i] = ga_peel_result{bn[i], bd[i], br[i], rounds[i]};
        if (status)
            status[i] = st[i] == LS_OK ? GA_OK
                        : st[i] == LS_ARITH ? GA_ERR_ARITH
                        : st[i] == LS_ROUND_LIMIT ? GA_ERR_ROUND_LIMIT
                                                  : GA_ERR_DEVICE_CHECK;
    }
    return GA_OK;
}

}  // namespace ga

using namespace ga;

extern "C" {

ga_status ga_batch_peel(ga_graph* g, uint64_t num, uint64_t den, ga_peel_result* res, uint32_t* removed_round) {
    if (!g || !res) return fail(GA_ERR_INVALID_ARGUMENT, "null argument");
    GA_GRAPH_LOCK(g);
    if (den < 1 || den > (1ull << 20) || num > (1ull << 20))
        return fail(GA_ERR_INVALID_ARGUMENT, "eps = num/den needs 1 <= den <= 2^20 and num <= 2^20");
    GA_TRY(use_device(g));
    LoopScalars s;
    GA_TRY(run_loop<LOOP_PEEL>(g, num, den, &s));
    res->best_num = s.best_num;
    res->best_den = s.best_den;
    res->best_round = s.best_round;
    res->rounds = s.round;
    if (removed_round && g->n) {
        GA_TRY(download(g, removed_round, g->loops->out, (size_t)g->n * 4));
    }
    return GA_OK;
}

ga_status ga_core_decomposition(ga_graph* g, uint32_t* core, ga_core_result* res) {
    if (!g || !res) return fail(GA_ERR_INVALID_ARGUMENT, "null argument");
    GA_GRAPH_LOCK(g);
    GA_TRY(use_device(g));
    LoopScalars s;
    GA_TRY(run_loop<LOOP_CORE>(g, 0, 1, &s));
    g->loops->cores_in_out = true;   // the densest-subgraph stages start from these core numbers
    g->loops->cores_kmax = s.kcur;
    res->kmax = s.kcur;
    res->rounds = s.round;
    if (core && g->n) {
        GA_TRY(download(g, core, g->loops->out, (size_t)g->n * 4));
    }
    return GA_OK;
}

}  // extern "C"
