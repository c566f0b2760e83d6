// ga_tc.cu - triangle counting and triangle support on the oriented CSR (sm_100a).
//
// What is computed is the reference's sum (graph.h:15-18, kernels.cuh:3): T = sum over oriented edges u->v of
// |N+(u) ∩ N+(v)|, every triangle {a,b,c} with a->b, a->c, b->c found exactly once. The reference's kernels v1-v9
// (kernels.cuh:53-358) walk that sum edge by edge. Here it is reorganised around the MIDDLE vertex b of each
// triangle (the "anchor"):
//
//     T = sum over anchors v of sum over in-edges u->v of |N+(u) ∩ N+(v)|
//
// N+(v) is loaded ONCE into a shared-memory set and the in-neighbours' lists are streamed past it (probe). A common
// neighbour x of u and v has v->x, so it comes after v in the orientation order; the index (ga_graph.cu) numbers the
// vertices in that order (places) and keeps every row ascending, so the probe list of in-edge u->v is just the part of
// u's row after v. Probe work is sum_u d+(u)(d+(u)-1)/2, half of sum_u d+(u)^2 and a quarter or less of the merge sum's
// sum_{u->v} (d+(u) + d+(v)) on power-law graphs, and each probe is one shared-memory load instead of a merge step
// or a binary search in global memory. Rows are padded to octs (8 places, one 32-byte sector) with a value that is in
// no set: a lane reads one oct and does eight probes without testing where the list starts or ends, so the search for
// the list an oct belongs to and the loop around it are paid once per eight probes (once per four, with two range tests
// a probe, when rows were unpadded ids: R-MAT 22 count 2.56 ms against 2.23, R-MAT 20 0.79 against 0.49; 2.00 ms since
// an oct is one 256-bit load).
//
// Scheduler (degree-binned, one persistent launch):
//   * work items = slices of an anchor's in-edge list with bounded probe work (built in ga_graph.cu);
//   * HEAVY bin: anchors with out-degree > light_max_deg. The whole block (8 warps) shares one set of N+(v) in dynamic
//     shared memory - for counts a bitmap over places, else a hash set - and splits the in-edges; anchors whose set
//     does not fit fall back to binary search in their row;
//   * LIGHT bin: every warp owns a 512-slot hash set and takes items on its own;
//   * TINY bin: anchors of at most 16 out-neighbours and 32 in-edges; a count takes 32 consecutive ones at a time, one
//     lane per in-edge, without any set (other passes run them like light ones);
//   * blocks drain the heavy queue first, then the light queue, then the tiny one (one atomic per fetch).
// Inside an item a warp processes 32 in-edges at a time: lane l loads the l-th record, a warp scan of the list
// lengths flattens the 32 lists into one sequence of octs, and lane p takes octs p, p+32, ... so lanes stay busy
// whatever the list lengths are (load-balanced search: each lane advances its owner index monotonically).
//
// Results per triangle (u->v in-edge, x common, x at position e of N+(u) and j of N+(v)):
//   COUNT: T only, one 64-bit atomic per block at the end.
//   VSUP : per-vertex counts: x through a per-slot shared counter (flushed once per item), u through a per-in-edge
//          shared counter (flushed once per 32 in-edges), v through a warp reduction (once per item).
//   ESUP : per-edge counts (for_each_triangle's (e_uv, e_ux, e_vx), dsg.h:67-79): e_uv and e_vx through shared
//          counters as above, e_ux with one global atomic per triangle, all at the entries' positions in colr; moved
//          to col order after the pass.
//   ALIVE: restricts everything to the subgraph induced by alive[] (tc_per_vertex_alive, kernels.cuh:399-425).
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <mutex>

#include "ga_device.cuh"
#include "ga_tc.cuh"

namespace ga {

#ifndef GA_TC_MIN_BLOCKS
#define GA_TC_MIN_BLOCKS 6                // resident blocks per SM the support and list passes are compiled for (8:
                                          // R-MAT 16 vertex supports 186 us, 6: 177)
#endif

constexpr int kCountBlocks = 8;           // ... and counts (R-MAT 22: 1.99 ms; 6: 2.12, 5: 2.31)
constexpr int kWarps = 8;                 // warps per block of the hash kernel
constexpr int kThreads = kWarps * 32;
// Per-warp hash set of the light bin: 512 slots for counts and lists; 256 in the support modes, whose slots carry
// counters too (2-3 words each): the smaller set keeps 7-8 blocks resident per SM instead of 4 (an anchor of up to
// 128 out-neighbours then has up to 2 keys per 4-slot bucket).
template <int MODE>
constexpr int light_slots() { return (MODE == TC_VSUP || MODE == TC_ESUP) ? 256 : 512; }
template <int MODE>
constexpr uint32_t light_bits() { return (MODE == TC_VSUP || MODE == TC_ESUP) ? 6 : 7; }

// VSUP and ESUP book per-slot and per-in-edge counters; COUNT and LIST do not.
__host__ __device__ constexpr bool counters(int mode) { return mode == TC_VSUP || mode == TC_ESUP; }

template <int MODE>
struct SlotLayout {   // 32-bit words per hash slot: key, +count (VSUP/ESUP), +position (ESUP)
    static constexpr int words = 1 + (counters(MODE) ? 1 : 0) + (MODE == TC_ESUP ? 1 : 0);
};

// Per-warp batch area: incl[32], base[32], ecnt[32], u[32].
constexpr int kBatchWords = 128;

// Shared memory of the light phase per warp: slots * words + the batch area.
template <int MODE>
constexpr int light_warp_words() { return light_slots<MODE>() * SlotLayout<MODE>::words + kBatchWords; }

// Slots per hash bucket. A table of 2^bits "units" holds 4 * 2^bits slots either way: 2^(bits+1) buckets of 2 slots
// (counts and lists: one 64-bit shared load per lookup, half the shared-memory traffic of a 4-slot bucket; measured
// 3.88 vs 4.24 ms on R-MAT 22) or 2^bits buckets of 4 slots (supports, whose slots carry counters: 11.9 vs 12.5 ms).
template <int MODE>
constexpr uint32_t bucket_slots() { return counters(MODE) ? 4u : 2u; }
template <int MODE>
constexpr uint32_t bucket_shift() { return bucket_slots<MODE>() == 4 ? 0u : 1u; }

// Table slots hold vertex ids below kTabEmpty (the hash kernel takes graphs of at most kTabEmpty vertices; larger
// ones count with the merge kernel). A bucket fills its slots in order, so a search can stop at a bucket whose last
// slot is free. 2-slot buckets (counts, lists) are full often enough at a load of 1/2 key per bucket (about 9 % of
// them) that a miss would go on to the next bucket for every tenth probe; there a key that found its bucket full while
// the table was built set kTabSpill in the last slot of every bucket it passed, and a search goes past a bucket only
// when that flag is set (R-MAT 22: count 3.55 vs 3.88 ms). 4-slot buckets are rarely full, and the flag's masking
// costs more than it saves there (supports 12.2 vs 11.5 ms), so they keep the free-slot rule alone.
constexpr uint32_t kTabEmpty = 0x7FFFFFFFu, kTabSpill = 0x80000000u;

template <int MODE>
constexpr bool spill_flags() { return bucket_slots<MODE>() == 2; }
static_assert(!spill_flags<TC_VSUP>() && !spill_flags<TC_ESUP>(), "flush_counts reads the support modes' keys as ids");

// Slots of bucket b that hold x (bit i = slot i); *open when the search for x ends at this bucket.
template <int MODE>
__device__ __forceinline__ uint32_t bucket_match(const uint32_t* key, uint32_t b, uint32_t x, bool* open) {
    if constexpr (bucket_slots<MODE>() == 4) {
        const uint4 t = reinterpret_cast<const uint4*>(key)[b];
        *open = t.w == kTabEmpty;
        return (t.x == x ? 1u : 0u) | (t.y == x ? 2u : 0u) | (t.z == x ? 4u : 0u) | (t.w == x ? 8u : 0u);
    } else {
        const uint2 t = reinterpret_cast<const uint2*>(key)[b];
        *open = (t.y & kTabSpill) == 0;
        return (t.x == x ? 1u : 0u) | ((t.y & ~kTabSpill) == x ? 2u : 0u);
    }
}

// Writes the triangle (u lowest, v middle, x highest; ids) into the incidence list of each corner. A list is sized by
// the counting pass; an entry that would land past its list's end is dropped and counted in *overflow instead.
template <class CT>
__device__ __forceinline__ void list_at(const TcArgs<CT>& a, uint32_t c, uint32_t at, uint32_t p, uint32_t q) {
    const unsigned long long pos = a.inc_ptr[c] + at;
    if (pos < a.inc_ptr[c + 1]) a.inc[pos] = make_uint2(p, q);
    else atomicAdd(a.overflow, 1u);
}
template <class CT>
__device__ __forceinline__ void list_one(const TcArgs<CT>& a, uint32_t c, uint32_t p, uint32_t q) {
    list_at(a, c, atomicAdd(&a.fill[c], 1u), p, q);
}
template <class CT>
__device__ __forceinline__ void list_triangle(const TcArgs<CT>& a, uint32_t u, uint32_t v, uint32_t x) {
    list_one(a, x, u, v);
    list_one(a, u, v, x);
    list_one(a, v, u, x);
}

// An anchor and the set of its members as the probe loops see them: a bitmap (counts and, with ranks, supports), a hash
// table (bits > 0), or nothing but its row (bits 0: binary search).
struct Anchor {
    uint32_t v, id, row, dv;   // place, id (LIST, VSUP), first oct of the row, out-degree
    uint32_t bits;             // table size
    uint32_t span;             // bitmap: places above v it covers (0: no bitmap)
};

// Finds place x among the members of anchor `an`: its counter's index - rank in the row (bitmap, row) or table slot -
// or GA_EMPTY. A row's padding is above every place, so it is never found. key: table or bitmap; pre: the bitmap's
// ranks (members below every word).
template <int MODE, bool ALIVE, class CT>
__device__ __forceinline__ uint32_t find_member(const TcArgs<CT>& a, const Anchor& an, uint32_t x,
                                                const uint32_t* key, const uint16_t* pre) {
    if (an.span) {
        const uint32_t o = x - an.v - 1;
        if (o >= an.span) return GA_EMPTY;
        const uint32_t w = key[o >> 5], bit = 1u << (o & 31);
        if (!(w & bit)) return GA_EMPTY;
        return counters(MODE) ? pre[o >> 5] + __popc(w & (bit - 1)) : 0u;
    }
    if (an.bits) {
        // bucketed set (bucket_slots<MODE>() slots per bucket); a bucket fills its slots in order, so an empty last
        // slot ends the search. One shared load resolves almost every lookup.
        const uint32_t nb = an.bits + bucket_shift<MODE>(), mask = (1u << nb) - 1;
        uint32_t b = hash_slot(x, nb);
        for (;;) {
            bool open;
            const uint32_t m = bucket_match<MODE>(key, b, x, &open);
            if (m) return bucket_slots<MODE>() * b + (__ffs(m) - 1);
            if (open) return GA_EMPTY;
            b = (b + 1) & mask;
        }
    }
    const uint32_t* row = a.ix.colr + (size_t)an.row * 8;
    const uint32_t j = lower_bound_u32(row, 0, an.dv, x);
    return j < an.dv && row[j] == x && (!ALIVE || a.alive[x]) ? j : GA_EMPTY;
}

// The end of a pass, called by all 256 threads of every block. In a synchronous call the blocks' triangles meet in
// sync->acc, and the last block writes the total where the caller wants it (device, and the handle's page-locked slot
// when the host waits for it) and leaves the counters zero for the next pass - so a count is one launch, with nothing
// to clear before it and nothing to copy after it (901 vertices: 20 us a call with two clears and a copy around the
// kernel). An enqueued pass adds to the total cleared before it: replays of captured passes overlap, and would take
// each other's blocks for their own in counters they share.
template <class CT>
__device__ __forceinline__ void finish_pass(unsigned long long local, const TcArgs<CT>& a) {
    __shared__ unsigned long long s_red[8];
    local = warp_sum_u64(local);
    if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = local;
    __syncthreads();
    if (threadIdx.x != 0) return;
    unsigned long long t = 0;
    for (int w = 0; w < 8; w++) t += s_red[w];
    if (!a.sync) {
        if (t) atomicAdd(a.total, t);
        return;
    }
    if (t) atomicAdd(&a.sync->acc, t);
    __threadfence();
    if (atomicInc(&a.sync->ticket, gridDim.x - 1) != gridDim.x - 1) return;   // wraps to zero with the last block
    __threadfence();
    t = atomicExch(&a.sync->acc, 0ull);
    for (int q = 0; q < 4; q++) a.work->queue[q] = 0;   // every block is done with the queues
    *a.total = t;
    if (a.host_total) *a.host_total = t;
}

// Oct q of colr, in one 256-bit load (a scattered request costs the load unit the same for 4 bytes as for 32).
__device__ __forceinline__ void load_oct(const uint32_t* __restrict__ colr, size_t q, uint32_t (&x)[8]) {
    asm("ld.global.nc.v8.u32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3]), "=r"(x[4]), "=r"(x[5]), "=r"(x[6]), "=r"(x[7])
        : "l"(colr + 8 * q));
}

// The probe lists of a batch of up to 32 in-edges [kb, kend) (one warp): lane l takes the l-th in-edge's suffix of its
// source's row, a run of whole octs, from in_rng. A warp scan of the oct counts flattens the lists into one sequence:
// oct p of it is oct s_base[owner] + p of colr, owner the first with s_incl[owner] > p. Entries of the first oct before
// the suffix are at or below the anchor's place and the last oct's padding is above every place, so neither is a member
// of N+(anchor) and the probes test no ends. Returns the octs of the batch; *r this lane's record (0: none).
template <bool ALIVE, class IX>
__device__ __forceinline__ uint32_t open_batch(const IX& ix, const uint8_t* alive, uint32_t kb, uint32_t kend,
                                               uint32_t lane, uint32_t* s_incl, uint32_t* s_base,
                                               unsigned long long* rec) {
    const uint32_t k = kb + lane;
    unsigned long long r = k < kend ? ix.in_rng[k] : 0ull;
    uint32_t nq = rng_octs(r);
    if (ALIVE && nq && !alive[ix.osrc[rng_at(r) >> 3]]) nq = 0;
    const uint32_t incl = warp_incl_scan(nq, lane);
    s_incl[lane] = incl;
    s_base[lane] = rng_oct(r) - (incl - nq);
    *rec = nq ? r : 0ull;
    __syncwarp();
    return __shfl_sync(GA_FULL_MASK, incl, 31);
}

// The members of the anchor among the eight entries of oct q: their number, and their positions in the oct three bits
// each in *list. Without branches for a bitmap or a table; buckets that are full without a match (rare) are followed
// afterwards.
template <int MODE, bool ALIVE, class CT>
__device__ __forceinline__ uint32_t oct_members(const TcArgs<CT>& a, const Anchor& an, uint32_t q, const uint32_t* key,
                                                uint32_t* list) {
    uint32_t xs[8];
    load_oct(a.ix.colr, q, xs);
    uint32_t l = 0, c3 = 0;   // c3: three times the number found
    if (an.span) {
        const uint32_t base = an.v + 1;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const uint32_t o = xs[i] - base;
            const uint32_t w = o < an.span ? key[o >> 5] : 0u;
            const bool m = (w >> (o & 31)) & 1u;
            l |= m ? i << c3 : 0;
            c3 += m ? 3 : 0;
        }
    } else if (an.bits) {
        const uint32_t nb = an.bits + bucket_shift<MODE>();
        uint32_t more = 0;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            bool open;
            const bool m = bucket_match<MODE>(key, hash_slot(xs[i], nb), xs[i], &open) != 0;
            l |= m ? i << c3 : 0;
            c3 += m ? 3 : 0;
            more |= (uint32_t)(!m & !open) << i;
        }
        while (more) {
            const uint32_t i = __ffs(more) - 1;
            more &= more - 1;
            if (find_member<MODE, ALIVE, CT>(a, an, __ldg(a.ix.colr + 8 * (size_t)q + i), key, nullptr) != GA_EMPTY) {
                l |= i << c3;
                c3 += 3;
            }
        }
    } else {
        for (uint32_t i = 0; i < 8; i++)
            if (find_member<MODE, ALIVE, CT>(a, an, a.ix.colr[8 * (size_t)q + i], key, nullptr) != GA_EMPTY) {
                l |= i << c3;
                c3 += 3;
            }
    }
    *list = l;
    return c3 / 3;
}

// Probes one batch of anchor `an` and books what MODE (supports, lists) asks for. A lane takes an oct and finds all its
// members; the hits of the 32 octs, a fifth to a quarter of the entries and unevenly spread, are then dealt out to the
// lanes 32 at a time, so the booking runs with full warps, and neighbouring lanes hold hits of one oct (their
// increments of the edges u->x share a sector; the entries of the anchor's list are consecutive). What an oct's
// triangles have in common (the edge u->v, u's list) is booked once per oct. Returns this lane's hits. (R-MAT 22 edge
// supports: booking inside the probe of each entry 7.4 ms; a loop over a lane's own hits 7.8 ms, 290 instructions a
// hit, most lanes idle.)
template <int MODE, bool ALIVE, class CT>
__device__ __forceinline__ uint32_t probe_batch(const TcArgs<CT>& a, uint32_t kb, uint32_t kend, const uint32_t* key,
                                                const uint16_t* pre, uint32_t* cnt, const Anchor& an, uint32_t* s_incl,
                                                uint32_t* s_base, uint32_t lane) {
    uint32_t *s_ecnt = s_base + 32, *s_u = s_base + 64;   // the caller's batch area: incl, base, ecnt, u
    unsigned long long rec;
    const uint32_t tot = open_batch<ALIVE>(a.ix, a.alive, kb, kend, lane, s_incl, s_base, &rec);
    uint32_t u = 0;
    if ((MODE == TC_LIST || MODE == TC_VSUP) && rec) u = a.ix.order[a.ix.osrc[rng_at(rec) >> 3]];   // the source's id
    if (MODE == TC_LIST) {
        s_u[lane] = u;
        __syncwarp();
    }
    uint32_t owner = 0, end = s_incl[0], hits = 0;
    for (uint32_t p0 = 0; p0 < tot; p0 += 32) {   // warp-uniform
        const uint32_t p = p0 + lane;
        uint32_t list = 0, c = 0, q = 0;
        if (p < tot) {
            while (end <= p) end = s_incl[++owner];
            q = s_base[owner] + p;
            c = oct_members<MODE, ALIVE, CT>(a, an, q, key, &list);
        }
        __syncwarp();
        const uint32_t incl = warp_incl_scan(c, lane), excl = incl - c, all = __shfl_sync(GA_FULL_MASK, incl, 31);
        if (!all) continue;
        hits += c;
        uint32_t bv = 0, bu = 0, uid = 0;
        if (MODE == TC_LIST) {
            if (lane == 0) bv = atomicAdd(&a.fill[an.id], all);
            bv = __shfl_sync(GA_FULL_MASK, bv, 0);
            if (c) {
                uid = s_u[owner];
                bu = atomicAdd(&a.fill[uid], c);
            }
        } else if (c) {
            atomicAdd(&s_ecnt[owner], c);
        }
        for (uint32_t h0 = 0; h0 < all; h0 += 32) {   // hit h0 + lane: the k-th of lane `from`
            const uint32_t h = h0 + lane;
            uint32_t from = 0;
#pragma unroll
            for (uint32_t step = 16; step > 0; step >>= 1)
                if (__shfl_sync(GA_FULL_MASK, excl, from + step) <= h) from += step;
            const uint32_t k = h - __shfl_sync(GA_FULL_MASK, excl, from);
            const uint32_t i = (__shfl_sync(GA_FULL_MASK, list, from) >> (3 * (k & 7))) & 7;
            const size_t e = (size_t)__shfl_sync(GA_FULL_MASK, q, from) * 8 + i;
            uint32_t hu = 0, hb = 0;
            if (MODE == TC_LIST) {
                hu = __shfl_sync(GA_FULL_MASK, uid, from);
                hb = __shfl_sync(GA_FULL_MASK, bu, from) + k;
            }
            if (h >= all) continue;
            const uint32_t x = __ldg(a.ix.colr + e);
            if (MODE == TC_LIST) {   // (u, v, x), lowest to highest
                const uint32_t xid = a.ix.order[x];
                list_at(a, an.id, bv + h, hu, xid);
                list_at(a, hu, hb, an.id, xid);
                list_at(a, xid, atomicAdd(&a.fill[xid], 1u), hu, an.id);
            } else {
                const uint32_t slot = find_member<MODE, ALIVE, CT>(a, an, x, key, pre);
                if (an.span || an.bits) atomicAdd(&cnt[slot], 1u);
                else if (MODE == TC_VSUP) red_add(&a.vsup[a.ix.order[x]], (CT)1);
                else red_add(&a.esupk[(size_t)an.row * 8 + slot], 1u);
                if (MODE == TC_ESUP) red_add(&a.esupk[e], 1u);   // u->x at its place in u's row
            }
        }
        __syncwarp();
    }
    __syncwarp();
    if (counters(MODE)) {
        const uint32_t c = s_ecnt[lane];
        if (c) {
            if (MODE == TC_VSUP) red_add(&a.vsup[u], (CT)c);
            else red_add(&a.esupk[rng_at(rec)], c);
            s_ecnt[lane] = 0;
        }
    }
    __syncwarp();
    return hits;
}

// Probes one batch of anchor `an` for a count, one lane per oct, in the anchor's table (or, without one, by binary
// search in its row). Returns this lane's hits.
template <bool ALIVE, class CT>
__device__ __forceinline__ uint32_t count_batch(const TcArgs<CT>& a, uint32_t kb, uint32_t kend, const uint32_t* key,
                                                const Anchor& an, uint32_t* s_incl, uint32_t* s_base, uint32_t lane) {
    unsigned long long rec;
    const uint32_t tot = open_batch<ALIVE>(a.ix, a.alive, kb, kend, lane, s_incl, s_base, &rec);
    uint32_t owner = 0, end = s_incl[0], hits = 0;
    if (!an.bits) {
        const uint32_t* row = a.ix.colr + (size_t)an.row * 8;
        for (uint32_t p = lane; p < tot; p += 32) {
            while (end <= p) end = s_incl[++owner];
            const uint32_t q = s_base[owner] + p;
#pragma unroll 1
            for (int i = 0; i < 8; i++) {
                const uint32_t x = a.ix.colr[8 * (size_t)q + i], j = lower_bound_u32(row, 0, an.dv, x);
                hits += j < an.dv && row[j] == x && (!ALIVE || a.alive[x]);
            }
        }
        __syncwarp();
        return hits;
    }
    // the eight lookups of an oct are issued without branches, so they overlap; a bucket that is full without a match
    // (rare) continues in the next buckets afterwards
    const uint32_t nb = an.bits + bucket_shift<TC_COUNT>(), bmask = (1u << nb) - 1;
    for (uint32_t p = lane; p < tot; p += 32) {
        while (end <= p) end = s_incl[++owner];
        const size_t q = s_base[owner] + p;
        uint32_t xs[8];
        load_oct(a.ix.colr, q, xs);
        uint32_t more = 0;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const uint32_t x = xs[i];
            bool open;
            const bool m = bucket_match<TC_COUNT>(key, hash_slot(x, nb), x, &open) != 0;
            hits += m;
            more |= (uint32_t)(!m & !open) << i;
        }
        while (more) {
            const int i = __ffs(more) - 1;
            more &= more - 1;
            const uint32_t x = __ldg(a.ix.colr + 8 * q + i);
            uint32_t b = hash_slot(x, nb);
            for (;;) {
                b = (b + 1) & bmask;
                bool open;
                if (bucket_match<TC_COUNT>(key, b, x, &open)) { hits++; break; }
                if (open) break;
            }
        }
    }
    __syncwarp();
    return hits;
}

// Buckets (log2) for an anchor with dv out-neighbours: 2^b >= dv (at most one key per bucket on average), at least
// 8 buckets, at most `cap` bits; an oversized anchor accepts up to 2 keys per bucket. Returns 0 when even that does
// not fit (the caller then binary-searches the global row).
__device__ __forceinline__ uint32_t table_bits(uint32_t dv, uint32_t cap) {
    uint32_t b = 3;
    while ((1u << b) < dv) b++;
    if (b <= cap) return b;
    return (2u << cap) >= dv ? cap : 0;
}

// Clears the table's 4 * 2^bits slots and inserts the (alive) members of N+(v): a key takes the first free slot of its
// bucket, or moves on to the next bucket when all of them are taken, flagging the full one where the mode keeps spill
// flags (kTabSpill in its last slot, which holds a key by then). tid/nthr cover the cooperating threads.
template <int MODE, bool ALIVE, class CT>
__device__ __forceinline__ void build_table(const TcArgs<CT>& a, const Anchor& an, uint32_t* key, uint32_t* cnt,
                                            uint32_t* pos, uint32_t tid, uint32_t nthr, bool sync_block) {
    constexpr uint32_t B = bucket_slots<MODE>();
    const uint32_t S = 4u << an.bits, nb = an.bits + bucket_shift<MODE>(), mask = (1u << nb) - 1;
    for (uint32_t s = tid; s < S / 4; s += nthr) {
        reinterpret_cast<uint4*>(key)[s] = make_uint4(kTabEmpty, kTabEmpty, kTabEmpty, kTabEmpty);
        if (counters(MODE)) reinterpret_cast<uint4*>(cnt)[s] = make_uint4(0, 0, 0, 0);
    }
    if (sync_block) __syncthreads(); else __syncwarp();
    const uint32_t* row = a.ix.colr + (size_t)an.row * 8;
    for (uint32_t i = tid; i < an.dv; i += nthr) {
        const uint32_t x = row[i];
        if (ALIVE && !a.alive[x]) continue;
        uint32_t b = hash_slot(x, nb), slot = B * b;
        while (atomicCAS(&key[slot], kTabEmpty, x) != kTabEmpty) {
            slot++;
            if ((slot & (B - 1)) == 0) {
                if (spill_flags<MODE>()) atomicOr(&key[slot - 1], kTabSpill);
                b = (b + 1) & mask;
                slot = B * b;
            }
        }
        if (MODE == TC_ESUP) pos[slot] = i;
    }
    if (sync_block) __syncthreads(); else __syncwarp();
}

// Heavy anchors use a bitmap of N+(v) instead of a hash set when it fits the table's shared memory: every
// out-neighbour's place is above v's own, and for the anchors of many out-neighbours (high degree) they lie in a short
// range (R-MAT 22: under 65,536 places for every anchor of more than 128 out-neighbours, against 4.2M vertices). Bit o
// of the bitmap is set iff place v + 1 + o is an (alive) out-neighbour of v; span = the largest out-neighbour - v
// bounds o. A probe is then one shared 32-bit load and a bit test, with no collisions and nothing to continue; the
// entries before the suffix and the padding fall outside [0, span). Supports also need which member it is: pre[w], the
// members below word w, plus a population count: the rank among the row's (alive) members, which the flush goes through
// again.
template <int MODE, bool ALIVE, class CT>
__device__ __forceinline__ void build_bitmap(const TcArgs<CT>& a, const Anchor& an, uint32_t* bm, uint16_t* pre,
                                             uint32_t* cnt) {
    const uint32_t quads = (an.span + 127) >> 7;
    for (uint32_t w = threadIdx.x; w < quads; w += kThreads) reinterpret_cast<uint4*>(bm)[w] = make_uint4(0, 0, 0, 0);
    if (counters(MODE))
        for (uint32_t i = threadIdx.x; i < an.dv; i += kThreads) cnt[i] = 0;
    __syncthreads();
    const uint32_t* row = a.ix.colr + (size_t)an.row * 8;
    for (uint32_t i = threadIdx.x; i < an.dv; i += kThreads) {
        const uint32_t x = row[i];
        if (ALIVE && !a.alive[x]) continue;
        const uint32_t o = x - an.v - 1;
        atomicOr(&bm[o >> 5], 1u << (o & 31));
    }
    __syncthreads();
    if (counters(MODE)) {
        // exclusive scan of the words' population counts: every warp scans a stretch, then adds the stretches before
        __shared__ uint32_t s_part[kWarps];
        const uint32_t words = (an.span + 31) >> 5, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const uint32_t per = ((words + kWarps - 1) / kWarps + 31) & ~31u, w0 = warp * per, w1 = min(words, w0 + per);
        uint32_t run = 0;
        for (uint32_t w = w0; w < w1; w += 32)
            run += __reduce_add_sync(GA_FULL_MASK, w + lane < w1 ? __popc(bm[w + lane]) : 0);
        if (lane == 0) s_part[warp] = run;
        __syncthreads();
        run = 0;
        for (uint32_t q = 0; q < warp; q++) run += s_part[q];
        for (uint32_t w = w0; w < w1; w += 32) {
            const uint32_t c = w + lane < w1 ? __popc(bm[w + lane]) : 0u;
            const uint32_t incl = warp_incl_scan(c, lane);
            if (w + lane < w1) pre[w + lane] = (uint16_t)(run + incl - c);
            run += __shfl_sync(GA_FULL_MASK, incl, 31);
        }
        __syncthreads();
    }
}

// A batch of a count against the bitmap of a heavy anchor. Returns this lane's hits.
template <bool ALIVE, class CT>
__device__ __forceinline__ uint32_t count_batch_bitmap(const TcArgs<CT>& a, uint32_t kb, uint32_t kend,
                                                       const uint32_t* bm, uint32_t base, uint32_t span,
                                                       uint32_t* s_incl, uint32_t* s_base, uint32_t lane) {
    unsigned long long rec;
    const uint32_t tot = open_batch<ALIVE>(a.ix, a.alive, kb, kend, lane, s_incl, s_base, &rec);
    uint32_t owner = 0, end = s_incl[0], hits = 0;
    for (uint32_t p = lane; p < tot; p += 32) {
        while (end <= p) end = s_incl[++owner];
        const size_t q = s_base[owner] + p;
        uint32_t xs[8];
        load_oct(a.ix.colr, q, xs);
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const uint32_t o = xs[i] - base;
            const uint32_t w = o < span ? bm[o >> 5] : 0u;
            hits += (w >> (o & 31)) & 1u;
        }
    }
    __syncwarp();
    return hits;
}

// Common entries of octs x and y of ascending rows, calling hit(place) for each when the caller books them.
// Padding must not match padding: y's is replaced by its first entry, which a row's every oct has.
template <bool BOOK, class F>
__device__ __forceinline__ uint32_t oct_common(const uint32_t (&x)[8], const uint32_t (&y)[8], F hit) {
    uint32_t z[8], c = 0;
#pragma unroll
    for (int j = 0; j < 8; j++) z[j] = y[j] == kPad ? y[0] : y[j];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        bool f = false;
#pragma unroll
        for (int j = 0; j < 8; j++) f |= x[i] == z[j];
        c += f;
        if (BOOK && f) hit(x[i]);
    }
    return c;
}

// Common places of an in-edge's suffix (x: its first oct, q, of `octs`) and its anchor's row (octs r.. up to rend):
// both ascend, so the oct with the smaller last entry is done after one comparison of all pairs. hit(place) as above.
template <bool BOOK, class F>
__device__ __forceinline__ uint32_t suffix_common(const uint32_t* __restrict__ colr, uint32_t (&x)[8], size_t q,
                                                  uint32_t octs, size_t r, size_t rend, F hit) {
    const size_t qend = q + octs;
    uint32_t y[8], c = 0;
    load_oct(colr, r, y);
    for (;;) {
        if (x[7] >= y[0])   // else the whole oct is below the row (padding counts as above)
            c += oct_common<BOOK>(x, y, hit);
        if (x[7] <= y[7]) {
            if (++q >= qend) return c;
            load_oct(colr, q, x);
        } else {
            if (++r >= rend) return c;
            load_oct(colr, r, y);
        }
    }
}

// The tiny bin of a count: one warp takes 32 consecutive places, flattens the in-edges of the tiny anchors among them,
// and every lane intersects one in-edge's suffix with its anchor's row, oct against oct in registers. An anchor of the
// light bin costs a warp some thousand cycles of item, table and batch set-up whatever its size; Holme-Kim graphs and
// the tails of R-MAT graphs are mostly anchors with a handful of probes. Rows are whole 32-byte sectors, so an in-edge
// of a short row is one sector.
template <class CT>
__device__ __forceinline__ uint32_t tiny_group(const TcArgs<CT>& a, uint32_t p0, uint32_t pend, uint32_t light_max_deg,
                                               uint32_t* s_incl, uint32_t* s_base, uint32_t* s_row, uint32_t* s_deg,
                                               uint32_t lane) {
    const uint32_t v = p0 + lane;
    uint32_t in = 0, k0 = 0, row = 0, d = 0;
    if (v < pend) {
        const uint32_t w = a.ix.work[v];
        d = a.ix.dout[v];
        if (w && d && d <= kTinyDeg) {
            const uint2 b = a.ix.pos[v];
            k0 = b.x;
            row = b.y;
            in = a.ix.pos[v + 1].x - k0;
            if (!is_tiny(d, in, w, light_max_deg)) in = 0;
        }
    }
    const uint32_t incl = warp_incl_scan(in, lane);
    const uint32_t tot = __shfl_sync(GA_FULL_MASK, incl, 31);
    if (!tot) return 0;
    s_incl[lane] = incl;
    s_base[lane] = k0 - (incl - in);
    s_row[lane] = row;
    s_deg[lane] = d;
    __syncwarp();
    uint32_t owner = 0, end = s_incl[0], hits = 0;
    for (uint32_t p = lane; p < tot; p += 32) {
        while (end <= p) end = s_incl[++owner];
        const unsigned long long r = a.ix.in_rng[s_base[owner] + p];
        if (!rng_octs(r)) continue;
        uint32_t x[8];
        load_oct(a.ix.colr, rng_oct(r), x);
        hits += suffix_common<false>(a.ix.colr, x, rng_oct(r), rng_octs(r), s_row[owner],
                                     s_row[owner] + ((s_deg[owner] + 7) >> 3), [](uint32_t) {});
    }
    __syncwarp();
    return hits;
}

// Adds an item's counters to the outputs (x's vertex count or edge v->x's count): by table slot, or by rank among the
// (alive) members of the row for a bitmap.
template <int MODE, bool ALIVE, class CT>
__device__ __forceinline__ void flush_counts(const TcArgs<CT>& a, const Anchor& an, const uint32_t* key,
                                             const uint16_t* pre, const uint32_t* cnt, const uint32_t* pos,
                                             uint32_t tid, uint32_t nthr) {
    if (!counters(MODE)) return;
    if (an.span) {
        const uint32_t* row = a.ix.colr + (size_t)an.row * 8;
        for (uint32_t j = tid; j < an.dv; j += nthr) {
            const uint32_t x = row[j];
            if (ALIVE && !a.alive[x]) continue;
            const uint32_t o = x - an.v - 1;
            const uint32_t c = cnt[ALIVE ? pre[o >> 5] + __popc(key[o >> 5] & ((1u << (o & 31)) - 1)) : j];
            if (!c) continue;
            if (MODE == TC_VSUP) red_add(&a.vsup[a.ix.order[x]], (CT)c);
            else red_add(&a.esupk[(size_t)an.row * 8 + j], c);
        }
        return;
    }
    const uint32_t S = 4u << an.bits;
    for (uint32_t s = tid; s < S; s += nthr) {
        const uint32_t c = cnt[s];
        if (c) {
            if (MODE == TC_VSUP) red_add(&a.vsup[a.ix.order[key[s]]], (CT)c);   // 4-slot buckets: no spill flags
            else red_add(&a.esupk[(size_t)an.row * 8 + pos[s]], c);
        }
    }
}

// esup[e] = esupk at the padded position of edge e's entry in its row: the place of col[e], found in the (short,
// sorted) row. Every edge is written, so esup needs no clearing.
__global__ void k_esup_fold(TcIndex ix, const uint32_t* __restrict__ src, const uint32_t* __restrict__ col, uint32_t m,
                            const uint32_t* __restrict__ esupk, uint32_t* __restrict__ esup) {
    for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < m; e += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t a = ix.vrank[src[e]], x = ix.vrank[col[e]];
        const size_t b = (size_t)ix.pos[a].y * 8;
        const uint32_t j = lower_bound_u32(ix.colr + b, 0, ix.dout[a], x);
        esup[e] = esupk[b + j];
    }
}

// alive mask by id -> by place.
__global__ void k_alive_places(const uint8_t* __restrict__ alive, const uint32_t* __restrict__ order, uint32_t n,
                               uint8_t* __restrict__ out) {
    for (uint64_t a = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; a < n; a += (uint64_t)gridDim.x * blockDim.x)
        out[a] = alive[order[a]];
}
// bounds (optional, device): this launch's item ranges (a shard), [bounds[2b], bounds[2b + 1]) of the items of bin b
// (heavy, light, tiny); null means every item. tiny_groups: counts of the whole graph take the tiny bin in groups of 32
// places from tiny_first on; otherwise its items are run like light ones.
template <int MODE, bool ALIVE, class CT>
__global__ void __launch_bounds__(kThreads, MODE == TC_COUNT ? kCountBlocks : GA_TC_MIN_BLOCKS)
k_tc_hash(ga_items items, const uint32_t* __restrict__ bounds, uint32_t heavy_bits_max, uint32_t tiny_first,
          uint32_t tiny_end, uint32_t light_max_deg, TcArgs<CT> a) {
    extern __shared__ __align__(16) uint32_t smem[];
    __shared__ uint32_t s_item, s_next;
    constexpr int W = SlotLayout<MODE>::words;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long hits = 0;
    const uint32_t H = items.info[0], L = items.info[1], T = items.info[2];
    const uint32_t h0 = bounds ? bounds[0] : 0u, h1 = bounds ? bounds[1] : H;
    const uint32_t l0 = bounds ? bounds[2] : H, l1 = bounds ? bounds[3] : H + L;
    const uint32_t t0 = bounds ? bounds[4] : H + L, t1 = bounds ? bounds[5] : H + L + T;
    const bool groups = MODE == TC_COUNT && !ALIVE && tiny_first < tiny_end;

    // ---- heavy bin: the block shares one set of N+(v) per item; its warps pull 32-in-edge batches from a shared
    //      counter, so no warp waits for another until the item is exhausted ----
    {
        const uint32_t Smax = 4u << heavy_bits_max;
        uint32_t* key = smem;
        uint32_t* cnt = key + Smax;
        uint32_t* pos = cnt + (counters(MODE) ? Smax : 0);
        uint32_t* wbase = smem + (size_t)Smax * W + warp * kBatchWords;
        uint32_t *s_incl = wbase, *s_base = wbase + 32;
        wbase[64 + lane] = 0;   // ecnt
        for (;;) {
            if (threadIdx.x == 0) s_item = h0 + atomicAdd(&a.work->queue[0], 1u);
            __syncthreads();
            const uint32_t item = s_item;
            if (item >= h1) break;
            Anchor an;
            an.v = items.v[item];
            if (ALIVE && !a.alive[an.v]) {
                __syncthreads();          // everyone has read s_item before thread 0 overwrites it
                continue;
            }
            an.row = a.ix.pos[an.v].y;
            an.dv = a.ix.dout[an.v];
            an.id = MODE == TC_LIST || MODE == TC_VSUP ? a.ix.order[an.v] : 0u;
            const uint32_t k0 = items.k0[item], k1 = items.k1[item];
            // the last entry of the row has the largest place; the bitmap takes the table's place, with the ranks and
            // counters of the support modes behind it
            const uint32_t span = a.ix.colr[(size_t)an.row * 8 + an.dv - 1] - an.v;
            const uint32_t words = (span + 127) >> 7 << 2, ranks = counters(MODE) ? words / 2 : 0;
            const bool bitmap =
                a.bitmaps && words + ranks + (counters(MODE) ? an.dv : 0u) <= Smax * W && an.dv <= 0xFFFFu;
            an.span = bitmap ? span : 0u;
            an.bits = bitmap ? 0u : table_bits(an.dv, heavy_bits_max);
            uint16_t* pre = reinterpret_cast<uint16_t*>(key + words);
            uint32_t* cn = bitmap ? key + words + ranks : cnt;
            if (threadIdx.x == 0) s_next = k0;
            if (bitmap) build_bitmap<MODE, ALIVE, CT>(a, an, key, pre, cn);
            else if (an.bits) build_table<MODE, ALIVE, CT>(a, an, key, cnt, pos, threadIdx.x, kThreads, true);
            else __syncthreads();
            unsigned long long h = 0;
            for (;;) {
                uint32_t kb = 0;
                if (lane == 0) kb = atomicAdd(&s_next, 32u);
                kb = __shfl_sync(GA_FULL_MASK, kb, 0);
                if (kb >= k1) break;
                if constexpr (MODE == TC_COUNT) {
                    if (bitmap) h += count_batch_bitmap<ALIVE, CT>(a, kb, min(kb + 32, k1), key, an.v + 1, span, s_incl,
                                                                   s_base, lane);
                    else h += count_batch<ALIVE, CT>(a, kb, min(kb + 32, k1), key, an, s_incl, s_base, lane);
                } else {
                    h += probe_batch<MODE, ALIVE, CT>(a, kb, min(kb + 32, k1), key, pre, cn, an, s_incl, s_base, lane);
                }
            }
            hits += h;
            if (MODE == TC_VSUP) {
                const unsigned long long t = warp_sum_u64(h);
                if (lane == 0 && t) red_add(&a.vsup[an.id], (CT)t);
            }
            __syncthreads();
            if (an.span || an.bits) flush_counts<MODE, ALIVE, CT>(a, an, key, pre, cn, pos, threadIdx.x, kThreads);
            __syncthreads();
        }
    }
    // ---- light bin (and the tiny one, unless it is taken in groups): one warp per item, private hash set of
    //      light_slots<MODE>() slots ----
    constexpr int PW = light_warp_words<MODE>();
    constexpr int LS = light_slots<MODE>();
    uint32_t* key = smem + warp * PW;
    uint32_t* cnt = key + LS;
    uint32_t* pos = cnt + (counters(MODE) ? LS : 0);
    uint32_t* s_incl = key + LS * W;
    uint32_t* s_base = s_incl + 32;
    s_incl[64 + lane] = 0;   // ecnt
    __syncwarp();
    const uint32_t nl = l1 - l0, total = nl + (groups ? 0u : t1 - t0);
    for (;;) {
        uint32_t i = 0;
        if (lane == 0) i = atomicAdd(&a.work->queue[1], 1u);
        i = __shfl_sync(GA_FULL_MASK, i, 0);
        if (i >= total) break;
        const uint32_t item = i < nl ? l0 + i : t0 + (i - nl);
        Anchor an;
        an.v = items.v[item];
        if (ALIVE && !a.alive[an.v]) continue;
        an.row = a.ix.pos[an.v].y;
        an.dv = a.ix.dout[an.v];
        an.id = MODE == TC_LIST || MODE == TC_VSUP ? a.ix.order[an.v] : 0u;
        // a table unless the anchor is too large for this mode's set (GA_OPT_LIGHT_MAX_DEG above 128 in the
        // support modes): then binary search in the row
        an.span = 0;
        an.bits = table_bits(an.dv, light_bits<MODE>());
        if (an.bits) build_table<MODE, ALIVE, CT>(a, an, key, cnt, pos, lane, 32, false);
        unsigned long long h = 0;
        const uint32_t k1 = items.k1[item];
        for (uint32_t kb = items.k0[item]; kb < k1; kb += 32) {
            if constexpr (MODE == TC_COUNT)
                h += count_batch<ALIVE, CT>(a, kb, min(kb + 32, k1), key, an, s_incl, s_base, lane);
            else
                h += probe_batch<MODE, ALIVE, CT>(a, kb, min(kb + 32, k1), key, nullptr, cnt, an, s_incl, s_base, lane);
        }
        hits += h;
        if (MODE == TC_VSUP) {
            const unsigned long long t = warp_sum_u64(h);
            if (lane == 0 && t) red_add(&a.vsup[an.id], (CT)t);
        }
        __syncwarp();
        if (an.bits) flush_counts<MODE, ALIVE, CT>(a, an, key, nullptr, cnt, pos, lane, 32);
        __syncwarp();
    }
    // ---- tiny bin of a whole count: groups of 32 places ----
    if constexpr (MODE == TC_COUNT && !ALIVE) {
        if (groups) {
            const uint32_t ngroups = (uint32_t)(((uint64_t)tiny_end - tiny_first + 31) / 32);
            // four groups a fetch, but no more than a warp's share: a group is a chain of up to 32 rounds of loads, and
            // on small graphs four of them were the kernel (R-MAT 16 count 61.7 -> 49.7 us, R-MAT 18 127.7 -> 122.1)
            const uint32_t take = min(kTinyGroups, max(1u, ngroups / (gridDim.x * kWarps)));
            for (;;) {
                uint32_t g0 = 0;
                if (lane == 0) g0 = atomicAdd(&a.work->queue[2], take);
                g0 = __shfl_sync(GA_FULL_MASK, g0, 0);
                if (g0 >= ngroups) break;
                const uint32_t g1 = min(g0 + take, ngroups);
                for (uint32_t g = g0; g < g1; g++)
                    hits += tiny_group<CT>(a, tiny_first + 32 * g, tiny_end, light_max_deg, s_incl, s_base, s_incl + 64,
                                           s_incl + 96, lane);
            }
        }
    }
    finish_pass(hits, a);
}

// The one-thread-per-edge form on the index: thread k takes in-edge k, whose record names its suffix and, one entry
// before it, its anchor; suffix and anchor's row are intersected oct against oct in registers. For graphs of short rows
// (Holme-Kim), where an anchor's set costs more than its probes: there an in-edge is two 32-byte sectors and some 70
// compares, against two unaligned rows merged entry by entry, each step waiting for the last, in k_tc_plain.
// VSUP: consecutive in-edges share their anchor, so a warp adds up its lanes' triangles by anchor before the atomic.
template <int MODE, bool ALIVE, class CT>
__global__ void __launch_bounds__(256) k_tc_octs(uint32_t m, TcArgs<CT> a) {
    static_assert(MODE == TC_COUNT || MODE == TC_VSUP, "the modes this form serves");
    const uint32_t lane = threadIdx.x & 31;
    unsigned long long local = 0;
    for (uint64_t k0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x - lane; k0 < m;
         k0 += (uint64_t)gridDim.x * blockDim.x) {   // warp-uniform
        const unsigned long long r = k0 + lane < m ? a.ix.in_rng[k0 + lane] : 0ull;
        const uint32_t octs = rng_octs(r);
        uint32_t c = 0, v = 0, u = 0;
        if (octs) {
            const size_t at = rng_at(r);
            uint32_t x[8];
            load_oct(a.ix.colr, rng_oct(r), x);
            // the anchor is the entry before the suffix: in its first oct, unless that starts one
            const uint32_t j = at & 7;
            v = x[0];
#pragma unroll
            for (int i = 1; i < 7; i++) v = j == i ? x[i] : v;
            if (j == 7) v = __ldg(a.ix.colr + at);
            const uint32_t row = a.ix.pos[v].y, rend = a.ix.pos[v + 1].y;
            if (ALIVE || MODE == TC_VSUP) u = a.ix.osrc[at >> 3];
            if (row != rend && (!ALIVE || (a.alive[u] && a.alive[v]))) {
                const uint32_t all = suffix_common<(ALIVE || MODE != TC_COUNT)>(
                    a.ix.colr, x, rng_oct(r), octs, row, rend, [&](uint32_t w) {
                        if (ALIVE && !a.alive[w]) return;
                        c++;
                        if (MODE == TC_VSUP) red_add(&a.vsup[a.ix.order[w]], (CT)1);
                    });
                if (MODE == TC_COUNT && !ALIVE) c = all;
            }
        }
        local += c;
        if (MODE == TC_VSUP && __any_sync(GA_FULL_MASK, c != 0)) {
            if (c) red_add(&a.vsup[a.ix.order[u]], (CT)c);
            const uint32_t peers = __match_any_sync(GA_FULL_MASK, c ? v : kPad);
            const uint32_t sum = __reduce_add_sync(peers, c);
            if (c && lane == (uint32_t)__ffs(peers) - 1) red_add(&a.vsup[a.ix.order[v]], (CT)sum);
        }
    }
    finish_pass(local, a);
}

// Plain form (GA_OPT_TC_KERNEL = 1): one thread per oriented edge, two-pointer merge of N+(u) and N+(v), one
// atomic per triangle and corner - the structure of the reference's v1 / tc_per_vertex_alive (kernels.cuh:53-69,
// 399-425), kept as the one-kernel-per-launch baseline.
template <int MODE, bool ALIVE, class CT>
__global__ void __launch_bounds__(256) k_tc_plain(const uint32_t* __restrict__ rowptr,
                                                  const uint32_t* __restrict__ col,
                                                  const uint32_t* __restrict__ src, uint32_t e_begin, uint32_t e_end,
                                                  TcArgs<CT> a) {
    unsigned long long local = 0;
    for (uint32_t e = e_begin + blockIdx.x * blockDim.x + threadIdx.x; e < e_end; e += gridDim.x * blockDim.x) {
        const uint32_t u = src[e], v = col[e];
        if (ALIVE && (!a.alive[u] || !a.alive[v])) continue;
        uint32_t i = rowptr[u], iend = rowptr[u + 1], j = rowptr[v], jend = rowptr[v + 1];
        while (i < iend && j < jend) {
            const uint32_t x = col[i], y = col[j];
            if (x < y) i++;
            else if (x > y) j++;
            else {
                if (!ALIVE || a.alive[x]) {
                    local++;
                    if (MODE == TC_VSUP) {
                        red_add(&a.vsup[u], (CT)1);
                        red_add(&a.vsup[v], (CT)1);
                        red_add(&a.vsup[x], (CT)1);
                    }
                    if (MODE == TC_ESUP) {
                        red_add(&a.esup[e], 1u);
                        red_add(&a.esup[i], 1u);
                        red_add(&a.esup[j], 1u);
                    }
                    if (MODE == TC_LIST) list_triangle(a, u, v, x);
                }
                i++;
                j++;
            }
        }
    }
    finish_pass(local, a);
}

// ---- host launchers ---------------------------------------------------------------------------------------------

template <int MODE>
static size_t hash_smem_bytes(uint32_t heavy_bits) {
    const size_t heavy = ((size_t)SlotLayout<MODE>::words << (heavy_bits + 2)) + kWarps * kBatchWords;
    const size_t light = (size_t)kWarps * light_warp_words<MODE>();
    return 4 * std::max(heavy, light);
}

// log2 buckets of the heavy (block-wide) set: enough for the largest heavy anchor at one key per bucket, capped by
// 200 KB of dynamic shared memory (and by GA_OPT_HEAVY_TABLE_BITS).
static uint32_t heavy_bits_for(const ga_graph* g, int mode) {
    const int words = 1 + (mode >= TC_VSUP) + (mode == TC_ESUP);
    uint32_t cap = 3;
    while ((((size_t)words << (cap + 3)) + kWarps * kBatchWords) * 4 <= 200 * 1024) cap++;
    if (g->heavy_bits_cap) cap = std::min(cap, g->heavy_bits_cap);
    // support modes: at most 512 buckets (anchors of up to 1,024 out-neighbours keep a table), so that the block's
    // shared memory stays near the light bin's and 7-8 blocks stay resident per SM
    if (mode == TC_VSUP || mode == TC_ESUP) cap = std::min(cap, 9u);
    uint32_t need = 3;
    const uint32_t largest = g->max_out_degree > g->light_max_deg ? g->max_out_degree : 0u;   // of the heavy bin
    while (need < cap && (1u << need) < largest) need++;
    return std::min(need, cap);
}

// Item ranges of shard `shard` of `nshards` in the three bins ([lo, hi) each, into out[6], as indexes of the whole item
// array). A shard is a range of anchors cut by their cumulative probe work (anchor_work[a] = work of the anchors below
// place a): an anchor goes to the shard its work starts in. Per-anchor work depends only on the graph - not on the bin
// cutoff or item work the autotuner picked for this copy, nor on the order a build left an in-list in - so copies of a
// graph prepared independently on several GPUs cut the same anchors, and the shards partition the triangles (each is
// counted at its middle vertex). The items of an anchor range are found by binary search (each bin ascends).
__global__ void k_shard_bounds(const unsigned long long* __restrict__ anchor_work, uint32_t n, ga_items items,
                               uint32_t shard, uint32_t nshards, uint32_t* __restrict__ out) {
    const uint32_t t = threadIdx.x;   // 6 threads: lo and hi of each bin
    if (t >= 6) return;
    const uint32_t part = shard + (t & 1), bin = t >> 1;
    uint32_t first = n;               // first anchor of shard `part` (n for the end)
    if (part < nshards) {
        const unsigned long long W = anchor_work[n];
        const unsigned long long goal = (W * part + nshards - 1) / nshards;   // ceil(W * part / nshards)
        uint32_t lo = 0, hi = n;      // first v with anchor_work[v] >= goal
        while (lo < hi) {
            const uint32_t mid = lo + ((hi - lo) >> 1);
            if (anchor_work[mid] < goal) lo = mid + 1; else hi = mid;
        }
        first = part == 0 ? 0u : lo;
    }
    uint32_t lo = 0;
    for (uint32_t b = 0; b < bin; b++) lo += items.info[b];
    uint32_t hi = lo + items.info[bin];
    while (lo < hi) {                 // first item of the bin whose anchor is >= first
        const uint32_t mid = lo + ((hi - lo) >> 1);
        if (items.v[mid] < first) lo = mid + 1; else hi = mid;
    }
    out[t] = lo;
}

// Blocks of a kernel resident per SM. The driver's answer for a shared-memory size does not change, so the last one is
// kept per kernel and device (`memo`: size << 8 | blocks) instead of asking before every launch; the kernel's limit is
// raised once to all it may use, never to one launch's size, which another thread's launch could exceed.
static ga_status resident_blocks(const void* kern, int threads, size_t smem, std::atomic<uint64_t>& memo, int* occ) {
    const uint64_t seen = memo.load(std::memory_order_relaxed);
    if (seen && seen >> 8 == smem) {
        *occ = (int)(seen & 0xFF);
        return GA_OK;
    }
    if (smem > 40 * 1024)
        GA_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 224 * 1024));
    int o = 0;
    GA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, kern, threads, smem));
    *occ = std::max(o, 1);
    memo.store((uint64_t)smem << 8 | (uint64_t)*occ, std::memory_order_relaxed);
    return GA_OK;
}

template <int MODE, bool ALIVE, class CT>
static ga_status launch_hash(ga_graph* g, const TcArgs<CT>& a) {
    cudaStream_t st = g->stream;
    const uint32_t hb = heavy_bits_for(g, MODE);
    const size_t smem = hash_smem_bytes<MODE>(hb);
    auto kern = k_tc_hash<MODE, ALIVE, CT>;
    static std::atomic<uint64_t> memo[64];
    int occ = 1;
    GA_TRY(resident_blocks((const void*)kern, kThreads, smem, memo[g->device], &occ));
    const uint32_t* bounds = nullptr;
    uint64_t want = (g->items.bound + kWarps - 1) / kWarps;
    uint32_t tiny_first = g->isolated, tiny_end = g->n;
    if (a.nshards > 1) {   // this shard's anchors (cut on the device)
        uint32_t* b = a.work->bounds;
        k_shard_bounds<<<1, 32, 0, st>>>(g->anchor_work, g->n, g->items, a.shard, a.nshards, b);
        GA_CUDA(cudaGetLastError());
        bounds = b;
        want = (want + a.nshards - 1) / a.nshards + 1;
        tiny_end = tiny_first;
    }
    want = std::max<uint64_t>(want, (uint64_t)g->max_out_degree > g->light_max_deg ? (uint64_t)g->sm_count * occ : 1);
    const unsigned grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((uint64_t)g->sm_count * occ, want));
    kern<<<grid, kThreads, smem, st>>>(g->items, bounds, hb, tiny_first, tiny_end, g->light_max_deg, a);
    GA_CUDA(cudaGetLastError());
    return GA_OK;
}

// One pass on the index (octs: one thread per in-edge, else the hash kernel). Per-vertex outputs are the caller's, by
// id: by place the hubs' counters would be neighbours, and the atomics on them meet in a few L2 sectors (vertex
// supports of R-MAT 18: 1.06 ms against 0.78). Per-edge outputs are by position in colr and moved to the caller's col
// order.
template <int MODE, bool ALIVE, class CT>
static ga_status launch_index(ga_graph* g, const TcArgs<CT>& a0, bool octs) {
    cudaStream_t st = g->stream;
    TcArgs<CT> a = a0;
    a.ix = tc_index(g);
    a.bitmaps = !g->opt_count_bitmap;
    Scratch tmp(st);   // supports by position in colr, or the mask by place
    if (MODE == TC_ESUP) {
        GA_TRY(tmp.alloc(&a.esupk, (size_t)g->octs * 8));
        GA_CUDA(cudaMemsetAsync(a.esupk, 0, (size_t)g->octs * 8 * 4, st));
    }
    if (ALIVE) {
        uint8_t* al;
        GA_TRY(tmp.alloc(&al, g->n));
        k_alive_places<<<grid_for(g->n, 256), 256, 0, st>>>(a0.alive, g->order, g->n, al);
        GA_CUDA(cudaGetLastError());
        a.alive = al;
    }
    if constexpr (MODE == TC_COUNT || MODE == TC_VSUP) {
        if (octs) {
            k_tc_octs<MODE, ALIVE, CT><<<grid_for(g->m, 256, (unsigned)g->sm_count * 16), 256, 0, st>>>(g->m, a);
            GA_CUDA(cudaGetLastError());
        }
    }
    static_assert(MODE != TC_ESUP || !ALIVE, "one temporary");
    if (!octs) GA_TRY((launch_hash<MODE, ALIVE, CT>(g, a)));
    if (MODE == TC_ESUP)
        k_esup_fold<<<grid_for(g->m, 256), 256, 0, st>>>(a.ix, g->src, g->col, g->m, a.esupk, a0.esup);
    GA_CUDA(cudaGetLastError());
    return GA_OK;
}

template <int MODE, bool ALIVE, class CT>
static ga_status launch_plain(ga_graph* g, const TcArgs<CT>& a) {
    static std::atomic<uint64_t> memo[64];
    int occ = 1;
    GA_TRY(resident_blocks((const void*)k_tc_plain<MODE, ALIVE, CT>, 256, 0, memo[g->device], &occ));
    uint32_t e0 = 0, e1 = g->m;
    if (a.nshards > 1) {   // this shard's equal part of the edges
        e0 = (uint32_t)((uint64_t)g->m * a.shard / a.nshards);
        e1 = (uint32_t)((uint64_t)g->m * (a.shard + 1) / a.nshards);
    }
    // an empty shard still runs one block, which writes the total
    const unsigned grid = grid_for(e1 > e0 ? e1 - e0 : 1, 256, (unsigned)g->sm_count * occ * 4);
    k_tc_plain<MODE, ALIVE, CT><<<grid, 256, 0, g->stream>>>(g->rowptr, g->col, g->src, e0, e1, a);
    GA_CUDA(cudaGetLastError());
    return GA_OK;
}

template <int MODE, bool ALIVE, class CT>
ga_status run_tc(ga_graph* g, const TcArgs<CT>& a0, bool zero_outputs) {
    // Automatic choice: the autotuned kernel for counts. Supports take the one-thread-per-edge form too when it counts
    // faster and rows are short (row_work / m, the octs of an edge's row on average, at most 2.5: Holme-Kim graphs have
    // 1 to 2.1; edge supports of the 1.7M one take 400 us against 2,010 us, vertex supports of a 200,003-vertex one 380
    // against 510), else the hash kernel: with longer rows there are more triangles an edge, whose increments contend
    // on hub vertices (R-MAT 14, 4.3 octs: vertex supports 334 us against 139). Incidence lists always take the hash
    // kernel (Holme-Kim 1.7M: 154 ms plain vs 4 ms hash).
    // A sharded count always uses the hash kernel unless one is forced: every GPU must cut the same partition, and
    // an autotuned choice could differ between GPUs.
    TcArgs<CT> a = a0;
    GA_TRY(a.nshards > 1 ? prepare_shards(g) : prepare(g));
    int64_t kernel = g->opt_tc_kernel ? g->opt_tc_kernel
                                      : (MODE == TC_COUNT || (MODE != TC_LIST && g->row_work * 2 <= 5ull * g->m)) &&
                                                a.nshards <= 1
                                            ? g->tuned_kernel
                                            : 2;
    if (g->n > kTabEmpty) kernel = 1;   // ids of kTabEmpty and above do not fit the hash kernel's table slots
    // the one-thread-per-edge form on the index for counts of any kind (per-edge supports are written in col's own
    // order by the plain form, without a pass to move them: 400 us vs 590); shards cut the edges themselves
    const bool octs = kernel == 1 && (MODE == TC_COUNT || MODE == TC_VSUP) && a.nshards <= 1 && g->n <= kTabEmpty;
    const bool index = (kernel != 1 || octs) && g->m;
    cudaStream_t st = g->stream;
    if (zero_outputs) {   // on the index, edge supports are written whole from the kernels' own array
        if (MODE == TC_VSUP && g->n) GA_CUDA(cudaMemsetAsync(a.vsup, 0, (size_t)g->n * sizeof(CT), st));
        if (!index && MODE == TC_ESUP && g->m) GA_CUDA(cudaMemsetAsync(a.esup, 0, (size_t)g->m * sizeof(uint32_t), st));
    }
    if (!g->m || a.enqueued) GA_CUDA(cudaMemsetAsync(a.total, 0, sizeof(unsigned long long), st));
    if (!g->m) {   // no kernel: the total is zero
        if (a.host_total) *a.host_total = 0;
        return GA_OK;
    }
    a.work = g->sync->work;
    if (!a.enqueued) {
        a.sync = g->sync;
    } else if (index && !octs) {   // the hash kernel's queues
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
        GA_CUDA(cudaStreamIsCapturing(st, &capture));
        if (capture == cudaStreamCaptureStatusNone) {
            a.work++;
        } else {
            GA_TRY(captured_work(g, &a.work));
            g->items_captured = true;
        }
        GA_CUDA(cudaMemsetAsync(a.work->queue, 0, sizeof a.work->queue, st));
    }
    return index ? launch_index<MODE, ALIVE, CT>(g, a, octs) : launch_plain<MODE, ALIVE, CT>(g, a);
}

// ---- autotuner ----------------------------------------------------------------------------------------------------
// What runs fastest depends on the degree distribution: on graphs whose out-lists are all short (Holme-Kim with a
// handful of edges per vertex) the one-thread-per-in-edge form (k_tc_octs, choice 1) can win, on skewed graphs with
// long lists (R-MAT) the degree-binned hash kernel wins by several times, and within the hash kernel the bin cutoff
// between per-warp and block-wide sets (light_max_deg) and the probe work per item (item_work, which sets how many
// warps share an anchor) move the time by some percent. The choice - kernel, cutoff, item work - is cached per
// degree-distribution signature: log2 of n and m and the fraction of edges whose source has out-degree in each log2
// bucket, in sixteenths. A signature seen before is answered from the cache (process-wide; also kept in the file named
// by GA_TUNE_CACHE when that is set); a new one is decided by timing candidates on the graph: both forms at the current
// options, then the cutoffs {32, 64, 128, 256} and the item works {1024, 4096, 16384} (coordinate-wise; options the
// caller set explicitly stay as set). Every candidate gives the same count.

struct TuneChoice {
    int kernel = 2;
    uint32_t light_max_deg = 128, item_work = 4096;
};

static std::mutex g_tune_mu;
static std::map<uint64_t, TuneChoice> g_tune_cache;
static bool g_tune_loaded = false;

static void tune_cache_load_locked() {
    if (g_tune_loaded) return;
    g_tune_loaded = true;
    const char* path = std::getenv("GA_TUNE_CACHE");
    if (!path) return;
    FILE* f = std::fopen(path, "r");
    if (!f) return;
    unsigned long long key;
    TuneChoice c;
    while (std::fscanf(f, "%llx %d %u %u", &key, &c.kernel, &c.light_max_deg, &c.item_work) == 4)
        if ((c.kernel == 1 || c.kernel == 2) && c.light_max_deg >= 1 && c.light_max_deg <= 256 && c.item_work >= 1)
            g_tune_cache[key] = c;
    std::fclose(f);
}

static void tune_cache_store_locked(uint64_t key, const TuneChoice& c) {
    g_tune_cache[key] = c;
    const char* path = std::getenv("GA_TUNE_CACHE");
    if (!path) return;
    FILE* f = std::fopen(path, "a");
    if (!f) return;
    std::fprintf(f, "%llx %d %u %u\n", (unsigned long long)key, c.kernel, c.light_max_deg, c.item_work);
    std::fclose(f);
}

// Degree-distribution signature of g (from the histogram the upload checks made).
static uint64_t tune_key(const ga_graph* g) {
    uint64_t key = mix64(32 - __builtin_clz(g->n | 1)) ^ mix64(0x100 + 32 - __builtin_clz(g->m)) ^ mix64(0x5e2);
    for (int b = 0; b < 33; b++) {
        const uint64_t q = (g->row_hist[b] * 16 + g->m / 2) / g->m;   // sixteenths of the edges
        key = mix64(key ^ (q << 8) ^ (uint64_t)b);
    }
    return key;
}

// Takes the choice of a signature seen before, if there is one, for a handle without work items.
static void choice_from_cache(ga_graph* g) {
    if (g->opt_tc_kernel || g->tuned_kernel || g->prepared || !g->m) return;
    const uint64_t key = tune_key(g);
    std::lock_guard<std::mutex> lock(g_tune_mu);
    tune_cache_load_locked();
    auto it = g_tune_cache.find(key);
    if (it == g_tune_cache.end()) return;
    if (!g->light_max_deg_set) g->light_max_deg = it->second.light_max_deg;
    if (!g->item_work_set) g->item_work = it->second.item_work;
    g->tuned_kernel = it->second.kernel;
    g->tune_key = key;
    g->tune_ms = 0;
}

ga_status ready(ga_graph* g) {
    choice_from_cache(g);   // before the work items are built, so they are built once
    GA_TRY(prepare(g));
    if (g->opt_tc_kernel == 0) GA_TRY(autotune(g));
    return GA_OK;
}

// Applies a choice (leaving options the caller set) and rebuilds the work items when the cutoff or item work moved.
static ga_status apply_choice(ga_graph* g, const TuneChoice& c) {
    const uint32_t light = g->light_max_deg_set ? g->light_max_deg : c.light_max_deg;
    const uint32_t work = g->item_work_set ? g->item_work : c.item_work;
    if (light != g->light_max_deg || work != g->item_work) {
        g->light_max_deg = light;
        g->item_work = work;
        g->prepared = false;
    }
    return prepare(g);
}

ga_status autotune(ga_graph* g) {
    if (g->tuned_kernel) return GA_OK;
    cudaStream_t st = g->stream;
    if (g->m == 0) { g->tuned_kernel = 2; return GA_OK; }
    if (g->n > kTabEmpty) { g->tuned_kernel = 1; return GA_OK; }   // beyond the hash kernel's ids
    const uint64_t key = tune_key(g);
    {
        std::lock_guard<std::mutex> lock(g_tune_mu);
        tune_cache_load_locked();
        auto it = g_tune_cache.find(key);
        if (it != g_tune_cache.end()) {
            const TuneChoice c = it->second;
            GA_TRY(apply_choice(g, c));
            g->tuned_kernel = c.kernel;
            g->tune_key = key;
            g->tune_ms = 0;
            return GA_OK;
        }
    }
    // time the candidates on this graph (count only); every kernel's code is loaded first (lazy module loading
    // would otherwise charge the load to the first candidate)
    cudaEvent_t e0, e1;
    GA_CUDA(cudaEventCreate(&e0));
    GA_CUDA(cudaEventCreate(&e1));
    TcArgs<unsigned int> a{};
    a.total = g->d_scalars + 2;
    cudaFuncAttributes fa;
    cudaFuncGetAttributes(&fa, k_tc_hash<TC_COUNT, false, unsigned int>);
    cudaFuncGetAttributes(&fa, k_tc_octs<TC_COUNT, false, unsigned int>);
    ga_status s = GA_OK;
    // best of two launches of candidate c
    auto time_of = [&](const TuneChoice& c, float* ms) -> ga_status {
        GA_TRY(apply_choice(g, c));
        g->tuned_kernel = c.kernel;
        float best = 1e30f;
        for (int rep = 0; rep < 2; rep++) {
            cudaEventRecord(e0, st);
            GA_TRY((run_tc<TC_COUNT, false, unsigned int>(g, a, true)));
            cudaEventRecord(e1, st);
            if (cudaEventSynchronize(e1) != cudaSuccess) return fail(GA_ERR_CUDA, "autotune timing failed");
            float t = 0;
            cudaEventElapsedTime(&t, e0, e1);
            best = std::min(best, t);
        }
        *ms = best;
        return GA_OK;
    };
    TuneChoice hash{2, g->light_max_deg, g->item_work}, plain{1, g->light_max_deg, g->item_work};
    float hash_ms = 0, plain_ms = 0;
    s = time_of(hash, &hash_ms);
    if (s == GA_OK) s = time_of(plain, &plain_ms);   // this form does not use the items
    for (uint32_t light : {32u, 64u, 128u, 256u}) {   // the bin cutoff, at the current item work
        if (s != GA_OK || g->light_max_deg_set || light == hash.light_max_deg) continue;
        TuneChoice c = hash;
        c.light_max_deg = light;
        float t = 0;
        s = time_of(c, &t);
        if (s == GA_OK && t < hash_ms) { hash = c; hash_ms = t; }
    }
    for (uint32_t work : {1024u, 4096u, 16384u}) {    // the item work, at the best cutoff
        if (s != GA_OK || g->item_work_set || work == hash.item_work) continue;
        TuneChoice c = hash;
        c.item_work = work;
        float t = 0;
        s = time_of(c, &t);
        if (s == GA_OK && t < hash_ms) { hash = c; hash_ms = t; }
    }
    // the items stay at the best hash configuration either way (supports and incidence lists use them)
    TuneChoice best = hash;
    float best_ms = hash_ms;
    if (plain_ms < hash_ms) { best.kernel = 1; best_ms = plain_ms; }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    g->tuned_kernel = 0;
    GA_TRY(s);
    GA_TRY(apply_choice(g, best));
    {
        std::lock_guard<std::mutex> lock(g_tune_mu);
        tune_cache_store_locked(key, best);
    }
    g->tuned_kernel = best.kernel;
    g->tune_key = key;
    g->tune_ms = best_ms;
    return GA_OK;
}

// The first count of a graph that nothing has prepared, when the one-thread-per-edge form is known to be its choice (by
// option or from the signature cache): counted straight from the CSR, since that form's plain version needs no index
// and building one costs more than a single count saves. The choice was made for k_tc_octs and this runs k_tc_plain,
// which loses more on longer rows; but where it loses to index + octs, the choice is the hash form. First calls on a
// new handle, us, k_tc_plain / index + k_tc_octs / index + hash, with row_work / m (octs to an edge's row):
//   chosen:     Holme-Kim 8,298 vertices 17-24 / 117-153 / 154-198 (1.0-2.5), 1.7M vertices 155 / 600 / 782 (1.0),
//               381 / 946 / 1,202 (1.1), 1,718 / 2,860 / 3,119 (2.5); R-MAT 10 18-25 / 85-92 / 102-117 (1.1-3.1),
//               R-MAT 14 25-39 / 148-169 / 183-211 (1.7-4.1), R-MAT 16 51 / 181 / 231 (3.4), R-MAT 18 77 / 239 / 284
//               (2.7)
//   not chosen: R-MAT 18 589 / 617 / 433 (8.0), 1,874 / 1,416 / 605 (14.0); Holme-Kim 1.7M 7,755 / 6,902 / 5,579 (4.9)
// A second count shows that the graph stays in use and builds the index. Misoriented graphs go on to ready(), which
// refuses them.
static bool counts_without_index(ga_graph* g) {
    if (g->index_ready || g->counted_bare || g->misoriented || !g->m) return false;
    choice_from_cache(g);   // kept: a later _async call counts with the same kernel
    return (g->opt_tc_kernel ? g->opt_tc_kernel : g->tuned_kernel) == 1;
}

template ga_status run_tc<TC_COUNT, false, unsigned int>(ga_graph*, const TcArgs<unsigned int>&, bool);
template ga_status run_tc<TC_COUNT, true, unsigned int>(ga_graph*, const TcArgs<unsigned int>&, bool);
template ga_status run_tc<TC_VSUP, false, unsigned long long>(ga_graph*, const TcArgs<unsigned long long>&, bool);
template ga_status run_tc<TC_VSUP, false, unsigned int>(ga_graph*, const TcArgs<unsigned int>&, bool);
template ga_status run_tc<TC_VSUP, true, unsigned int>(ga_graph*, const TcArgs<unsigned int>&, bool);
template ga_status run_tc<TC_ESUP, false, unsigned int>(ga_graph*, const TcArgs<unsigned int>&, bool);
template ga_status run_tc<TC_LIST, false, unsigned int>(ga_graph*, const TcArgs<unsigned int>&, bool);

}  // namespace ga

using namespace ga;

namespace {

// alive[v] = core[v] >= k; the number of such vertices is added to *cnt (one atomic per warp).
__global__ void k_core_mask(const uint32_t* __restrict__ core, uint32_t n, uint32_t k, uint8_t* __restrict__ alive,
                            unsigned long long* cnt) {
    uint32_t c = 0;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        const uint8_t in = core[v] >= k;
        alive[v] = in;
        c += in;
    }
    c = __reduce_add_sync(GA_FULL_MASK, c);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(cnt, (unsigned long long)c);
}

// Waits for the stream; the pass (whose host_total is the handle's slot) has left its total there.
ga_status read_total(ga_graph* g, uint64_t* out) {
    GA_CUDA(cudaStreamSynchronize(g->stream));
    if (out) *out = g->h_scalars[0];
    return GA_OK;
}

}  // namespace

extern "C" {

ga_status ga_tc_count(ga_graph* g, uint64_t* triangles) {
    if (!g || !triangles) return fail(GA_ERR_INVALID_ARGUMENT, "null argument");
    GA_GRAPH_LOCK(g);
    GA_TRY(use_device(g));
    TcArgs<unsigned int> a{};
    a.total = g->d_scalars;
    a.host_total = g->h_scalars;
    if (!counts_without_index(g)) {
        GA_TRY(ready(g));
        GA_TRY((run_tc<TC_COUNT, false, unsigned int>(g, a, true)));
        return read_total(g, triangles);
    }
    a.sync = g->sync;
    a.work = g->sync->work;
    GA_TRY((launch_plain<TC_COUNT, false, unsigned int>(g, a)));
    GA_TRY(read_total(g, triangles));
    g->counted_bare = true;
    return GA_OK;
}

ga_status ga_tc_count_shard(ga_graph* g, uint32_t shard, uint32_t nshards, uint64_t* partial) {
    if (!g || !partial) return fail(GA_ERR_INVALID_ARGUMENT, "null argument");
    if (nshards == 0 || shard >= nshards) return fail(GA_ERR_INVALID_ARGUMENT, "need shard < nshards");
    GA_GRAPH_LOCK(g);
    GA_TRY(use_device(g));
    GA_TRY(ready(g));
    TcArgs<unsigned int> a{};
    a.total = g->d_scalars;
    a.host_total = g->h_scalars;
    a.shard = shard;
    a.nshards = nshards;
    GA_TRY((run_tc<TC_COUNT, false, unsigned int>(g, a, true)));
    return read_total(g, partial);
}

ga_status ga_tc_count_shard_async(ga_graph* g, uint32_t shard, uint32_t nshards, uint64_t* d_partial) {
    if (!g || !d_partial) return fail(GA_ERR_INVALID_ARGUMENT, "null argument");
    if (nshards == 0 || shard >= nshards) return fail(GA_ERR_INVALID_ARGUMENT, "need shard < nshards");
    GA_GRAPH_LOCK(g);
    GA_TRY(use_device(g));
    TcArgs<unsigned int> a{};
    a.total = (unsigned long long*)d_partial;
    a.enqueued = true;
    a.shard = shard;
    a.nshards = nshards;
    GA_TRY(prepare_enqueued(g, nshards > 1));
    return run_tc<TC_COUNT, false, unsigned int>(g, a, true);
}

ga_status ga_tc_count_async(ga_graph* g, uint64_t* d_triangles) {
    if (!g || !d_triangles) return fail(GA_ERR_INVALID_ARGUMENT, "null argument");
    GA_GRAPH_LOCK(g);
    GA_TRY(use_device(g));
    TcArgs<unsigned int> a{};
    a.total = (unsigned long long*)d_triangles;
    a.enqueued = true;
    GA_TRY(prepare_enqueued(g, false));
    return run_tc<TC_COUNT, false, unsigned int>(g, a, true);
}

ga_status ga_tc_support_edges_device(ga_graph* g, uint32_t* d_sup, uint64_t* triangles) {
    if (!g || (!d_sup && g->m)) return fail(GA_ERR_INVALID_ARGUMENT, "null argument");
    GA_GRAPH_LOCK(g);
    GA_TRY(use_device(g));
    GA_TRY(ready(g));
    TcArgs<unsigned int> a{};
    a.total = g->d_scalars;
    a.host_total = g->h_scalars;
    a.esup = d_sup;
    GA_TRY((run_tc<TC_ESUP, false, unsigned int>(g, a, true)));
    return read_total(g, triangles);
}

ga_status ga_tc_support_edges(ga_graph* g, uint32_t* sup, uint64_t* triangles) {
    if (!g || (!sup && g->m)) return fail(GA_ERR_INVALID_ARGUMENT, "null argument");
    GA_GRAPH_LOCK(g);
    GA_TRY(use_device(g));
    Scratch s(g->stream);
    uint32_t* d_sup;
    GA_TRY(s.alloc(&d_sup, (size_t)g->m + 1));
    GA_TRY(ga_tc_support_edges_device(g, d_sup, triangles));
    return download(g, sup, d_sup, (size_t)g->m * 4);
}

ga_status ga_tc_support_vertices(ga_graph* g, uint64_t* deg, uint64_t* triangles) {
    if (!g || (!deg && g->n)) return fail(GA_ERR_INVALID_ARGUMENT, "null argument");
    GA_GRAPH_LOCK(g);
    GA_TRY(use_device(g));
    GA_TRY(ready(g));
    Scratch s(g->stream);
    TcArgs<unsigned long long> a{};
    GA_TRY(s.alloc(&a.vsup, (size_t)g->n + 1));
    a.total = g->d_scalars;
    a.host_total = g->h_scalars;
    GA_TRY((run_tc<TC_VSUP, false, unsigned long long>(g, a, true)));
    GA_TRY(download(g, deg, a.vsup, (size_t)g->n * 8));
    return read_total(g, triangles);
}

ga_status ga_tc_participation(ga_graph* g, const uint8_t* alive, uint32_t* tri, uint64_t* triangles) {
    if (!g || ((!alive || !tri) && g->n)) return fail(GA_ERR_INVALID_ARGUMENT, "null argument");
    GA_GRAPH_LOCK(g);
    GA_TRY(use_device(g));
    GA_TRY(ready(g));
    // T of the alive subgraph is at most T of the graph; refuse when uint32 counters could overflow (densest.h:68). T
    // is at most sum over u of C(d+(u), 2), and that at most 4 * row_work: only above 2^32 does it take a count to know
    if (g->row_work >= (1ull << 30)) {
        uint64_t T_full = 0;
        GA_TRY(ga_tc_count(g, &T_full));
        if (T_full >= (1ull << 32))
            return fail(GA_ERR_ARITH, "triangle count >= 2^32: uint32 tri[] counters could overflow");
    }
    Scratch s(g->stream);
    uint8_t* d_alive;   // the mask behind the counts
    GA_TRY(s.alloc(&d_alive, ((size_t)g->n + 1) * 5));
    uint32_t* d_tri = (uint32_t*)d_alive;
    d_alive += ((size_t)g->n + 1) * 4;
    if (g->n) GA_CUDA(cudaMemcpyAsync(d_alive, alive, g->n, cudaMemcpyHostToDevice, g->stream));
    TcArgs<unsigned int> a{};
    a.total = g->d_scalars;
    a.host_total = g->h_scalars;
    a.vsup = d_tri;
    a.alive = d_alive;
    GA_TRY((run_tc<TC_VSUP, true, unsigned int>(g, a, true)));
    GA_TRY(download(g, tri, d_tri, (size_t)g->n * 4));
    return read_total(g, triangles);
}

ga_status ga_graph_tuning(ga_graph* g, ga_tuning* out) {
    if (!g || !out) return fail(GA_ERR_INVALID_ARGUMENT, "null argument");
    GA_GRAPH_LOCK(g);
    GA_TRY(use_device(g));
    GA_TRY(ready(g));
    out->kernel = (uint32_t)(g->opt_tc_kernel ? g->opt_tc_kernel : g->tuned_kernel);
    out->light_max_deg = g->light_max_deg;
    out->item_work = g->item_work;
    out->signature = g->tune_key;
    out->measured_ms = g->opt_tc_kernel ? 0.0 : (double)g->tune_ms;
    out->heavy_items = out->light_items = 0;
    if (g->items.info && g->prepared) {
        uint32_t info[3];
        GA_CUDA(cudaMemcpyAsync(info, g->items.info, sizeof info, cudaMemcpyDeviceToHost, g->stream));
        GA_CUDA(cudaStreamSynchronize(g->stream));
        out->heavy_items = info[0];
        out->light_items = (uint64_t)info[1] + info[2];
    }
    return GA_OK;
}

ga_status ga_core_level_density(ga_graph* g, const uint32_t* core, uint32_t k, uint64_t* triangles,
                                uint64_t* vertices) {
    if (!g || (!core && g->n) || !triangles || !vertices) return fail(GA_ERR_INVALID_ARGUMENT, "null argument");
    GA_GRAPH_LOCK(g);
    GA_TRY(use_device(g));
    GA_TRY(ready(g));
    Scratch s(g->stream);
    const size_t n = g->n;
    uint8_t* d_alive;   // the mask behind the core numbers
    GA_TRY(s.alloc(&d_alive, (n + 1) * 5));
    uint32_t* d_core = (uint32_t*)d_alive;
    d_alive += (n + 1) * 4;
    unsigned long long* d_cnt = g->d_scalars + 1;
    GA_CUDA(cudaMemsetAsync(d_cnt, 0, 8, g->stream));
    if (n) {
        GA_CUDA(cudaMemcpyAsync(d_core, core, n * 4, cudaMemcpyHostToDevice, g->stream));
        k_core_mask<<<grid_for(n, 256), 256, 0, g->stream>>>(d_core, g->n, k, d_alive, d_cnt);
        GA_CUDA(cudaGetLastError());
    }
    TcArgs<unsigned int> a{};
    a.total = g->d_scalars;
    a.host_total = g->h_scalars;
    a.alive = d_alive;
    GA_TRY((run_tc<TC_COUNT, true, unsigned int>(g, a, true)));
    GA_CUDA(cudaMemcpyAsync(g->h_scalars + 1, g->d_scalars + 1, 8, cudaMemcpyDeviceToHost, g->stream));
    GA_CUDA(cudaStreamSynchronize(g->stream));
    *triangles = g->h_scalars[0];
    *vertices = g->h_scalars[1];
    return GA_OK;
}

}  // extern "C"
