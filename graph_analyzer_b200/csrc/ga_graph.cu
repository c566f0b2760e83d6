// ga_graph.cu - device-resident graph handle: upload, validation, and the derived structures every query shares.
//
// Derived structures (built on the device, kept resident). The orientation order (degree, id) numbers the vertices; a
// vertex's number is its PLACE, and everything the triangle kernels read is kept in places:
//   src[m], deg[n]         row owner and degree of every edge / vertex, by id (made with the checks at upload)
//   vrank[n] / order[n]    place of every id and id of every place
//   pos[n+1]               by place: where its in-edges start (x) and where its row starts in colr (y, in octs)
//   colr                   every row as ascending places, padded to whole octs (8 entries, one 32-byte sector) with
//                          kPad, which no place reaches: a probe loop reads whole octs and tests no ends
//   osrc                   place of the row every oct belongs to
//   in_rng[m]              for every in-edge u->v, laid out anchor by anchor (v): where v sits in u's row and how many
//                          octs of that row hold entries after v (its probe suffix)
//   dout[n], work[n]       by place: out-degree, and octs its in-edges have to probe
//   items                  work lists of the triangle kernels: one item = a slice of an anchor's in-edges whose probe
//                          work is bounded; anchors of a large out-degree are "heavy" (a block each), others "light"
//                          (a warp each), the smallest "tiny" (counts take 32 of them at a time)
#include <algorithm>
#include <cstring>
#include <mutex>
#include <vector>

#include "ga_device.cuh"

namespace ga {

// ---- exclusive scan: tiles of 512 threads x 8 elements, two launches ------------------------------------------------
// k_scan_sums writes every tile's sum; k_scan_tiles adds up the sums of the tiles before its own itself (a few KB from
// L2 for the sizes here) and scans its tile from registers, so there is no third launch for the sums. Above
// kScanDirect tiles the sums are scanned first.
constexpr int kScanThreads = 512, kScanItems = 8, kScanTile = kScanThreads * kScanItems;
constexpr uint64_t kScanDirect = 8192;
constexpr unsigned long long kHeavyItemFactor = 64;   // heavy items carry 64x the probe work of light items

// Sum over the block (every thread gets it). s_w: kScanThreads / 32 slots.
template <class T>
__device__ __forceinline__ T block_sum(T x, T* s_w) {
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(GA_FULL_MASK, x, o);
    if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = x;
    __syncthreads();
    T t = 0;
    for (int w = 0; w < kScanThreads / 32; w++) t += s_w[w];
    __syncthreads();
    return t;
}

template <class T>
__global__ void __launch_bounds__(kScanThreads) k_scan_sums(const T* __restrict__ in, uint64_t n, T* __restrict__ sums) {
    __shared__ T s_w[kScanThreads / 32];
    const uint64_t base = (uint64_t)blockIdx.x * kScanTile + threadIdx.x;
    T acc = 0;
#pragma unroll
    for (int j = 0; j < kScanItems; j++) {
        const uint64_t k = base + (uint64_t)j * kScanThreads;
        if (k < n) acc += in[k];
    }
    acc = block_sum(acc, s_w);
    if (threadIdx.x == 0) sums[blockIdx.x] = acc;
}

// sums: the tiles' sums (scanned = false) or their exclusive prefix (true); null for a single tile. In place allowed.
template <class T>
__global__ void __launch_bounds__(kScanThreads) k_scan_tiles(const T* in, T* out, uint64_t n, const T* __restrict__ sums,
                                                             bool scanned) {
    __shared__ T s_w[kScanThreads / 32];
    T before = 0;
    if (sums && scanned) before = sums[blockIdx.x];
    else if (sums) {
        T acc = 0;
        for (uint32_t b = threadIdx.x; b < blockIdx.x; b += kScanThreads) acc += sums[b];
        before = block_sum(acc, s_w);
    }
    // thread t scans elements 8t .. 8t + 7 of the tile
    const uint64_t k0 = (uint64_t)blockIdx.x * kScanTile + (uint64_t)threadIdx.x * kScanItems;
    T v[kScanItems], run = 0;
#pragma unroll
    for (int j = 0; j < kScanItems; j++) {
        v[j] = k0 + j < n ? in[k0 + j] : (T)0;
        run += v[j];
    }
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    T x = run;
    for (int o = 1; o < 32; o <<= 1) {
        const T t = __shfl_up_sync(GA_FULL_MASK, x, o);
        if (lane >= (uint32_t)o) x += t;
    }
    if (lane == 31) s_w[w] = x;
    __syncthreads();
    T pre = before + x - run;
    for (uint32_t q = 0; q < w; q++) pre += s_w[q];
#pragma unroll
    for (int j = 0; j < kScanItems; j++) {
        if (k0 + j < n) out[k0 + j] = pre;
        pre += v[j];
    }
}

template <class T>
static ga_status scan_impl(cudaStream_t st, const T* in, T* out, uint64_t n) {
    if (n == 0) return GA_OK;
    const uint64_t nb = (n + kScanTile - 1) / kScanTile;
    if (nb == 1) {
        k_scan_tiles<T><<<1, kScanThreads, 0, st>>>(in, out, n, nullptr, false);
        GA_CUDA(cudaGetLastError());
        return GA_OK;
    }
    Scratch tmp(st);
    T* sums;
    GA_TRY(tmp.alloc(&sums, nb));
    k_scan_sums<T><<<(unsigned)nb, kScanThreads, 0, st>>>(in, n, sums);
    GA_CUDA(cudaGetLastError());
    const bool scanned = nb > kScanDirect;
    if (scanned) GA_TRY(scan_impl<T>(st, sums, sums, nb));
    k_scan_tiles<T><<<(unsigned)nb, kScanThreads, 0, st>>>(in, out, n, sums, scanned);
    GA_CUDA(cudaGetLastError());
    return GA_OK;
}

ga_status scan_u64(ga_graph* g, unsigned long long* data, uint64_t n) {
    return scan_impl<unsigned long long>(g->stream, data, data, n);
}

// ---- validation and derived structures -------------------------------------------------------------------------

// d_scalars slots of the upload checks.
enum : int { SC_HIST = 8, SC_ISOLATED = 55, SC_ORIENT = 56, SC_MAXDEG = 57, SC_WORK = 58, SC_OCTS = 59, SC_MAXOUT = 60,
             SC_ERR = 61 };

// One pass over the rows: the checks, src[], the in-degrees (indeg[] zeroed before) and the sums that size the index.
// A warp takes 32 consecutive rows, whose entries are consecutive: lanes read them coalesced and find their row among
// the 32 starts. Rows of a warp whose starts are not ascending within [0, m] are flagged and not read.
// Flags in sc[SC_ERR]: 1 rowptr not monotone / beyond m, 2 endpoint >= n, 4 self loop, 8 row not strictly ascending.
__global__ void __launch_bounds__(256) k_rows(const uint32_t* __restrict__ rowptr, const uint32_t* __restrict__ col,
                                              uint32_t n, uint32_t m, uint32_t* __restrict__ src,
                                              uint32_t* __restrict__ indeg, unsigned long long* __restrict__ sc) {
    // the block's sums: histogram, then SC_WORK .. SC_ERR (one atomic each per block: a per-warp one serialises)
    __shared__ unsigned long long s_hist[33], s_sum[4];
    if (threadIdx.x < 33) s_hist[threadIdx.x] = 0;
    if (threadIdx.x < 4) s_sum[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    uint32_t bad = 0, maxout = 0;
    unsigned long long octs = 0, work = 0;
    for (uint64_t v0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x - lane; v0 < n; v0 += stride) {
        const uint32_t v = (uint32_t)v0 + lane;
        const bool row = v0 + lane < n;
        const uint32_t b = row ? rowptr[v] : 0u;
        const uint32_t e = row ? rowptr[v + 1] : 0u;
        const bool wrong = row && (b > e || e > m);
        if (__any_sync(GA_FULL_MASK, wrong)) {
            bad |= wrong;
            continue;
        }
        const uint32_t d = e - b;
        maxout = max(maxout, d);
        octs += (d + 7) >> 3;
        work += (unsigned long long)d * ((d + 7) >> 3);
        {   // edges by log2 of the row's length (the autotuner's signature), one add per bucket and warp
            const uint32_t bucket = d ? 32 - __clz(d) : 0u;
            const uint32_t peers = __match_any_sync(GA_FULL_MASK, bucket);
            const uint32_t sum = __reduce_add_sync(peers, d);
            if (bucket && lane == (uint32_t)__ffs(peers) - 1) atomicAdd(&s_hist[bucket], (unsigned long long)sum);
        }
        const uint32_t nrows = (uint32_t)min((uint64_t)32, n - v0);
        const uint32_t first = __shfl_sync(GA_FULL_MASK, b, 0), last = __shfl_sync(GA_FULL_MASK, e, nrows - 1);
        const uint32_t start = row ? b : last;   // lanes past the last row start at the end: never found below it
        for (uint32_t i0 = first; i0 < last; i0 += 32) {
            const uint32_t i = i0 + lane;
            const bool in = i >= i0 && i < last;   // i >= i0: no wrap past 2^32
            // row of entry i: the last lane whose start is <= i (empty rows share their start with the next)
            uint32_t r = 0;
#pragma unroll
            for (uint32_t step = 16; step > 0; step >>= 1) {
                const uint32_t at = __shfl_sync(GA_FULL_MASK, start, r + step);
                if (in && at <= i) r += step;
            }
            const uint32_t rb = __shfl_sync(GA_FULL_MASK, b, r);
            const uint32_t x = in ? col[i] : 0u;
            uint32_t prev = __shfl_up_sync(GA_FULL_MASK, x, 1);
            if (lane == 0 && in && i > rb) prev = col[i - 1];
            if (in) {
                const uint32_t u = (uint32_t)v0 + r;
                src[i] = u;
                if (x >= n) bad |= 2;
                else atomicAdd(&indeg[x], 1u);
                if (x == u) bad |= 4;
                if (i > rb && prev >= x) bad |= 8;
            }
            if (last - i0 <= 32) break;   // no wrap of i0
        }
    }
    bad = __reduce_or_sync(GA_FULL_MASK, bad);
    maxout = __reduce_max_sync(GA_FULL_MASK, maxout);
    octs = warp_sum_u64(octs);
    work = warp_sum_u64(work);
    if (lane == 0) {
        if (bad) atomicOr(&s_sum[SC_ERR - SC_WORK], (unsigned long long)bad);
        if (maxout) atomicMax(&s_sum[SC_MAXOUT - SC_WORK], (unsigned long long)maxout);
        if (octs) atomicAdd(&s_sum[SC_OCTS - SC_WORK], octs);
        if (work) atomicAdd(&s_sum[0], work);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (s_sum[SC_ERR - SC_WORK]) atomicOr(&sc[SC_ERR], s_sum[SC_ERR - SC_WORK]);
        atomicMax(&sc[SC_MAXOUT], s_sum[SC_MAXOUT - SC_WORK]);
        atomicAdd(&sc[SC_OCTS], s_sum[SC_OCTS - SC_WORK]);
        atomicAdd(&sc[SC_WORK], s_sum[0]);
    }
    if (threadIdx.x < 33 && s_hist[threadIdx.x]) atomicAdd(&sc[SC_HIST + threadIdx.x], s_hist[threadIdx.x]);
}

// deg[v] += out-degree (deg holds the in-degrees): total degrees, their maximum and the number of isolated vertices.
__global__ void __launch_bounds__(256) k_degrees(const uint32_t* __restrict__ rowptr, uint32_t n,
                                                 uint32_t* __restrict__ deg, unsigned long long* __restrict__ sc) {
    __shared__ uint32_t s_mx, s_isolated;
    if (threadIdx.x == 0) s_mx = s_isolated = 0;
    __syncthreads();
    uint32_t mx = 0, isolated = 0;
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t d = deg[v] + rowptr[v + 1] - rowptr[v];
        deg[v] = d;
        mx = max(mx, d);
        isolated += d == 0;
    }
    mx = __reduce_max_sync(GA_FULL_MASK, mx);
    isolated = __reduce_add_sync(GA_FULL_MASK, isolated);
    if ((threadIdx.x & 31) == 0) {
        if (mx) atomicMax(&s_mx, mx);
        if (isolated) atomicAdd(&s_isolated, isolated);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (s_mx) atomicMax(&sc[SC_MAXDEG], (unsigned long long)s_mx);
        if (s_isolated) atomicAdd(&sc[SC_ISOLATED], (unsigned long long)s_isolated);
    }
}

// The orientation rule of graph.h:43-45 for every edge: from the smaller to the larger endpoint by (degree, id).
// sc[SC_ORIENT] != 0: an edge points the wrong way. (Endpoints >= n are skipped: k_rows has refused the graph.)
__global__ void __launch_bounds__(256) k_orient(const uint32_t* __restrict__ src, const uint32_t* __restrict__ col,
                                                const uint32_t* __restrict__ deg, uint32_t n, uint32_t m,
                                                unsigned long long* __restrict__ sc) {
    bool bad = false;
    for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < m; e += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t u = src[e], x = col[e];
        if (x >= n || u >= n) continue;
        const uint32_t du = deg[u], dx = deg[x];
        bad |= !(du != dx ? du < dx : u < x);
    }
    if (__any_sync(GA_FULL_MASK, bad) && (threadIdx.x & 31) == 0) atomicOr(&sc[SC_ORIENT], 1ull);
}

// ---- rows in places ----------------------------------------------------------------------------------------------
// Every row's entries become places (one gather of vrank), are sorted (places alone: the sort carries nothing else) and
// written as whole octs. A row is sorted by a bitonic network over E keys per lane, element l * E + i in register i of
// lane l: strides below E stay inside a thread (min / max), larger ones are one shuffle. k_in_lists then reads the
// octs once, in order, and writes every entry's in-list record; it is a kernel of its own because it only waits (an
// atomic with a result and a scattered write per entry) and wants all the warps an SM holds, which the sort's registers
// do not leave (both in one kernel: 2.64 ms for R-MAT 22's rows of more than 8 entries, apart 1.0 + 1.0). (64-bit
// (degree, id) keys counted against each other in shared memory with the entries' positions carried along, then a
// scatter and a gather of their own, took 4.0 ms of R-MAT 22's 5.4 ms of build kernels.)
template <int E, int LANES>
__device__ __forceinline__ void sort_keys(uint32_t (&k)[E], uint32_t l) {
#pragma unroll
    for (int size = 2; size <= E * LANES; size <<= 1) {
#pragma unroll
        for (int st = size >> 1; st > 0; st >>= 1) {
            if (st >= E) {
                const uint32_t xl = st / E;
                const bool lower = (l & xl) == 0;
                const bool up = size >= E * LANES || (l & (size / E)) == 0;
#pragma unroll
                for (int i = 0; i < E; i++) {
                    const uint32_t o = __shfl_xor_sync(GA_FULL_MASK, k[i], xl);
                    k[i] = lower == up ? min(k[i], o) : max(k[i], o);
                }
            } else {
#pragma unroll
                for (int i = 0; i < E; i++) {
                    if ((i & st) == 0) {
                        const bool up = size < E ? (i & size) == 0 : size >= E * LANES || (l & (size / E)) == 0;
                        const uint32_t a = k[i], b = k[i | st];
                        k[i] = up ? min(a, b) : max(a, b);
                        k[i | st] = up ? max(a, b) : min(a, b);
                    }
                }
            }
        }
    }
}

// Rows of at most 8 entries, four rows per warp, one per 8-lane group. Longer rows are appended to `listed`.
__global__ void __launch_bounds__(256) k_place_rows_small(const uint32_t* __restrict__ rowptr,
                                                          const uint32_t* __restrict__ col,
                                                          const uint32_t* __restrict__ vrank,
                                                          const uint32_t* __restrict__ order,
                                                          const uint2* __restrict__ pos, uint32_t first, uint32_t n,
                                                          uint32_t* __restrict__ colr, uint32_t* __restrict__ osrc,
                                                          uint32_t* __restrict__ listed,
                                                          uint32_t* __restrict__ nlisted) {
    const uint32_t lane = threadIdx.x & 31, sub = lane & 7;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t t0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x - lane; t0 < (uint64_t)(n - first) * 8;
         t0 += stride) {
        const uint64_t row = first + ((t0 + lane) >> 3);
        const bool valid = row < n;
        const uint32_t a = (uint32_t)row;
        uint32_t b = 0, d = 0;
        if (valid) {
            const uint32_t u = order[a];
            b = rowptr[u];
            d = rowptr[u + 1] - b;
        }
        const bool mine = d >= 1 && d <= 8;   // the whole group agrees (same row)
        uint32_t k[1] = {mine && sub < d ? vrank[col[b + sub]] : kPad};
        sort_keys<1, 8>(k, sub);
        if (mine) {
            const uint32_t o0 = pos[a].y;
            colr[(size_t)o0 * 8 + sub] = k[0];
            if (sub == 0) osrc[o0] = a;
        }
        const bool longer = valid && d > 8 && sub == 0;
        const uint32_t bal = __ballot_sync(GA_FULL_MASK, longer);
        if (bal) {
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(nlisted, (uint32_t)__popc(bal));
            base = __shfl_sync(GA_FULL_MASK, base, 0);
            if (longer) listed[base + __popc(bal & ((1u << lane) - 1))] = a;
        }
    }
}

template <int E>
__device__ __forceinline__ void place_row(const uint32_t* __restrict__ row, uint32_t d, uint32_t a, uint32_t lane,
                                          const uint32_t* __restrict__ vrank, const uint2* __restrict__ pos,
                                          uint32_t* __restrict__ colr, uint32_t* __restrict__ osrc) {
    uint32_t k[E];
#pragma unroll
    for (int i = 0; i < E; i++) k[i] = lane + 32 * i < d ? vrank[row[lane + 32 * i]] : kPad;   // any start order
    sort_keys<E, 32>(k, lane);
    const uint32_t o0 = pos[a].y, end = (d + 7) & ~7u;
#pragma unroll
    for (int i = 0; i < E; i++) {
        const uint32_t j = lane * E + i;
        if (E < 4 && j < end) colr[(size_t)o0 * 8 + j] = k[i];
        if (E >= 4 && (i & 3) == 0 && j < end)
            *reinterpret_cast<uint4*>(colr + (size_t)o0 * 8 + j) =
                make_uint4(k[i], k[E >= 4 ? i + 1 : 0], k[E >= 4 ? i + 2 : 0], k[E >= 4 ? i + 3 : 0]);
        if (j < end && (j & 7) == 0) osrc[o0 + (j >> 3)] = a;
    }
}

// The listed rows, one warp per row, the last (largest places, mostly the longest rows) first. Up to 512 entries: the
// register network; longer rows (rare: out-degrees are at most sqrt(2m) in this orientation) count smaller places.
__global__ void __launch_bounds__(128) k_place_rows_listed(const uint32_t* __restrict__ rowptr,
                                                           const uint32_t* __restrict__ col,
                                                           const uint32_t* __restrict__ vrank,
                                                           const uint32_t* __restrict__ order,
                                                           const uint2* __restrict__ pos,
                                                           uint32_t* __restrict__ colr, uint32_t* __restrict__ osrc,
                                                           const uint32_t* __restrict__ listed,
                                                           const uint32_t* __restrict__ nlisted) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t count = *nlisted;
    for (uint32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < count; r += nwarps) {
        const uint32_t a = listed[count - 1 - r], u = order[a];
        const uint32_t b = rowptr[u], d = rowptr[u + 1] - b;
        const uint32_t* row = col + b;
        if (d <= 32) place_row<1>(row, d, a, lane, vrank, pos, colr, osrc);
        else if (d <= 64) place_row<2>(row, d, a, lane, vrank, pos, colr, osrc);
        else if (d <= 128) place_row<4>(row, d, a, lane, vrank, pos, colr, osrc);
        else if (d <= 256) place_row<8>(row, d, a, lane, vrank, pos, colr, osrc);
        else if (d <= 512) place_row<16>(row, d, a, lane, vrank, pos, colr, osrc);
        else {
            const uint32_t o0 = pos[a].y, end = (d + 7) & ~7u;
            for (uint32_t i0 = lane; i0 < d; i0 += 256) {   // eight entries per lane per pass over the row
                uint32_t kq[8], rk[8];
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    kq[q] = i0 + 32 * q < d ? vrank[row[i0 + 32 * q]] : 0u;
                    rk[q] = 0;
                }
                for (uint32_t j = 0; j < d; j++) {
                    const uint32_t kj = vrank[row[j]];
#pragma unroll
                    for (int q = 0; q < 8; q++) rk[q] += kj < kq[q];
                }
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    if (i0 + 32 * q >= d) continue;
                    colr[(size_t)o0 * 8 + rk[q]] = kq[q];
                }
            }
            for (uint32_t j = d + lane; j < end; j += 32) colr[(size_t)o0 * 8 + j] = kPad;
            for (uint32_t j = lane; j < end >> 3; j += 32) osrc[o0 + j] = a;
        }
    }
}

// One lane per entry of colr: the entry x of place a's row is the in-edge a->x, whose record goes to the next free
// place of x's in-list. cur[x] holds that place in its low word and the octs x's in-edges have to probe in its high
// word, so one 64-bit atomic serves both (neither reaches 2^32: an in-edge with a suffix of s octs needs a row of
// 8(s-1) others).
__global__ void __launch_bounds__(256) k_in_lists(const uint32_t* __restrict__ colr, const uint32_t* __restrict__ osrc,
                                                  const uint2* __restrict__ pos, uint64_t entries,
                                                  unsigned long long* __restrict__ cur,
                                                  unsigned long long* __restrict__ in_rng) {
    for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < entries;
         e += (uint64_t)gridDim.x * blockDim.x) {   // entries is a multiple of 8: an oct's lanes are here together
        const uint32_t x = colr[e];
        if (x == kPad) continue;
        uint32_t octs = pos[osrc[e >> 3] + 1].y - (uint32_t)((e + 1) >> 3);
        if (((e + 1) & 7) && colr[e + 1] == kPad) octs = 0;   // the row's last entry: nothing to probe after it
        const unsigned long long at = atomicAdd(&cur[x], (unsigned long long)octs << 32 | 1u);
        in_rng[(uint32_t)at] = pack_rng(e, octs);
    }
}

// cur[a] = start of a's in-list.
__global__ void k_in_cursors(const uint2* __restrict__ pos, uint32_t n, unsigned long long* __restrict__ cur) {
    for (uint64_t a = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; a < n; a += (uint64_t)gridDim.x * blockDim.x)
        cur[a] = pos[a].x;
}

// ---- vertex places in the (degree, id) order ---------------------------------------------------------------------
// A stable LSD radix sort of the vertices by degree (out + in), 9 bits per pass, starting from id order, so that
// equal degrees stay in id order: the result is the (degree, id) order of graph.h:43-45. Each warp owns a chunk of
// `chunk` consecutive entries: k_rank_count counts the chunk's digits, an exclusive scan over (digit, chunk) gives
// every chunk its start in each digit's range, and k_rank_scatter writes the chunk's entries in order (lanes with the
// same digit ranked by __match_any_sync, a per-digit running count per warp in shared memory).
constexpr uint32_t kRankBits = 9, kRankDigits = 1u << kRankBits, kRankWarps = 8;
// entries per chunk: a warp walks its chunk serially (16 dependent steps), so small inputs take shorter ones
static uint32_t rank_chunk(uint32_t n) { return n <= 1u << 16 ? 128 : 512; }

// counts[d * nchunks + c] = entries of chunk c whose digit is d (cur == nullptr: the identity order).
__global__ void __launch_bounds__(kRankWarps * 32) k_rank_count(const uint32_t* __restrict__ cur,
                                                                const uint32_t* __restrict__ deg, uint32_t n,
                                                                uint32_t shift, uint32_t nchunks, uint32_t chunk,
                                                                uint32_t* __restrict__ counts) {
    __shared__ uint32_t s_h[kRankWarps][kRankDigits];
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t c = blockIdx.x * kRankWarps + w;
    if (c >= nchunks) return;   // warp-uniform; no block barrier below
    uint32_t* h = s_h[w];
    for (uint32_t d = lane; d < kRankDigits; d += 32) h[d] = 0;
    __syncwarp();
    const uint32_t b = c * chunk, e = (uint32_t)min((uint64_t)n, (uint64_t)b + chunk);
    for (uint32_t i = b + lane; i < e; i += 32) {
        const uint32_t x = cur ? cur[i] : i;
        atomicAdd(&h[(deg[x] >> shift) & (kRankDigits - 1)], 1u);
    }
    __syncwarp();
    for (uint32_t d = lane; d < kRankDigits; d += 32) counts[(size_t)d * nchunks + c] = h[d];
}

// Writes the chunk's entries to next[] at their digit's place (offs = exclusive scan of counts), in chunk order.
__global__ void __launch_bounds__(kRankWarps * 32) k_rank_scatter(const uint32_t* __restrict__ cur,
                                                                  const uint32_t* __restrict__ deg, uint32_t n,
                                                                  uint32_t shift, uint32_t nchunks, uint32_t chunk,
                                                                  const uint32_t* __restrict__ offs,
                                                                  uint32_t* __restrict__ next) {
    __shared__ uint32_t s_run[kRankWarps][kRankDigits];
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t c = blockIdx.x * kRankWarps + w;
    if (c >= nchunks) return;   // warp-uniform; no block barrier below
    uint32_t* run = s_run[w];
    for (uint32_t d = lane; d < kRankDigits; d += 32) run[d] = 0;
    __syncwarp();
    const uint32_t b = c * chunk, e = (uint32_t)min((uint64_t)n, (uint64_t)b + chunk);
    for (uint32_t i0 = b; i0 < e; i0 += 32) {
        const uint32_t i = i0 + lane;
        const bool valid = i < e;
        const uint32_t x = valid ? (cur ? cur[i] : i) : 0u;
        // lanes past the chunk get distinct digits outside the digit range, so they match no one
        const uint32_t d = valid ? (deg[x] >> shift) & (kRankDigits - 1) : kRankDigits + lane;
        const uint32_t peers = __match_any_sync(GA_FULL_MASK, d);
        const uint32_t leader = __ffs(peers) - 1;
        uint32_t base = 0;
        if (lane == leader && valid) base = run[d];
        base = __shfl_sync(GA_FULL_MASK, base, leader);
        if (valid) next[offs[(size_t)d * nchunks + c] + base + __popc(peers & ((1u << lane) - 1))] = x;
        __syncwarp();
        if (lane == leader && valid) run[d] = base + __popc(peers);
        __syncwarp();
    }
}

// By place: vrank[order[a]] = a, dout, and what pos[] is the scan of (in-degree in the low word, octs of the row in the
// high word: neither sum reaches 2^32, so one 64-bit scan gives both).
__global__ void k_places(const uint32_t* __restrict__ rowptr, const uint32_t* __restrict__ deg,
                         const uint32_t* __restrict__ order, uint32_t n, uint32_t* __restrict__ vrank,
                         uint32_t* __restrict__ dout, unsigned long long* __restrict__ pos) {
    for (uint64_t a = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; a <= n; a += (uint64_t)gridDim.x * blockDim.x) {
        if (a == n) { pos[n] = 0; continue; }
        const uint32_t u = order[a], d = rowptr[u + 1] - rowptr[u];
        vrank[u] = (uint32_t)a;
        dout[a] = d;
        pos[a] = (unsigned long long)((d + 7) >> 3) << 32 | (deg[u] - d);
    }
}

// work[a] = octs to probe for anchor a, from the cursors.
__global__ void k_work(const unsigned long long* __restrict__ cur, uint32_t n, uint32_t* __restrict__ work) {
    for (uint64_t a = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; a < n; a += (uint64_t)gridDim.x * blockDim.x)
        work[a] = (uint32_t)(cur[a] >> 32);
}

__global__ void k_widen(const uint32_t* __restrict__ in, uint32_t n, unsigned long long* __restrict__ out) {
    for (uint64_t a = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; a <= n; a += (uint64_t)gridDim.x * blockDim.x)
        out[a] = a < n ? in[a] : 0ull;
}

// Items of anchor a: none without out-neighbours or probe work, else ceil(work / target) (at most one per in-edge;
// heavy anchors have kHeavyItemFactor times the target, since the block-wide set is built once per item).
// cnt[a] = light items | heavy items << 32, tiny[a] = 1 for an anchor of the tiny bin (one item).
__global__ void k_count_items(const uint2* __restrict__ pos, const uint32_t* __restrict__ dout,
                              const uint32_t* __restrict__ work, uint32_t n, uint32_t light_max_deg,
                              unsigned long long target, unsigned long long* __restrict__ cnt,
                              uint32_t* __restrict__ tiny) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i <= n; i += (uint64_t)gridDim.x * blockDim.x) {
        unsigned long long c = 0;
        uint32_t t = 0;
        if (i < n) {
            const uint32_t a = (uint32_t)i, d = dout[a], in = pos[a + 1].x - pos[a].x;
            const unsigned long long w = (unsigned long long)work[a] * 8;
            if (d && w) {
                const bool heavy = d > light_max_deg;
                const unsigned long long tg = heavy ? target * kHeavyItemFactor : target;
                const unsigned long long want = min((w + tg - 1) / tg, (unsigned long long)in);
                t = is_tiny(d, in, work[a], light_max_deg);
                c = t ? 0ull : heavy ? want << 32 : want;
            }
        }
        cnt[i] = c;
        tiny[i] = t;
    }
}

// One thread per item, in the order heavy, light, tiny (each by ascending anchor): finds its anchor by binary search
// over the bin's offsets, then its part of the anchor's in-edges (equal numbers: the in-lists are in no order of work).
// Thread 0 leaves the bins' sizes in info[0..2].
__global__ void k_emit_items(const uint2* __restrict__ pos, const unsigned long long* __restrict__ off,
                             const uint32_t* __restrict__ toff, uint32_t n, uint32_t* __restrict__ it_v,
                             uint32_t* __restrict__ it_k0, uint32_t* __restrict__ it_k1, uint32_t* __restrict__ info) {
    const uint32_t H = (uint32_t)(off[n] >> 32), L = (uint32_t)off[n], T = toff[n];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        info[0] = H;
        info[1] = L;
        info[2] = T;
    }
    const uint64_t total = (uint64_t)H + L + T;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (uint64_t)gridDim.x * blockDim.x) {
        const int bin = i < H ? 0 : i < (uint64_t)H + L ? 1 : 2;
        const uint32_t q = (uint32_t)(bin == 0 ? i : bin == 1 ? i - H : i - H - L);
        auto at = [&](uint32_t a) -> uint32_t {
            return bin == 2 ? toff[a] : bin == 1 ? (uint32_t)off[a] : (uint32_t)(off[a] >> 32);
        };
        uint32_t lo = 0, hi = n;   // anchor = last a with at(a) <= q (one without items shares its offset with the next)
        while (lo < hi) {
            const uint32_t mid = lo + ((hi - lo) >> 1);
            if (at(mid) <= q) lo = mid + 1; else hi = mid;
        }
        const uint32_t a = lo - 1, o = at(a), c = at(a + 1) - o, j = q - o;
        const uint32_t b = pos[a].x, len = pos[a + 1].x - b;
        it_v[i] = a;
        it_k0[i] = b + (uint32_t)((uint64_t)len * j / c);
        it_k1[i] = b + (uint32_t)((uint64_t)len * (j + 1) / c);
    }
}

void dfree(ga_graph* g, void* p) {
    if (!p) return;
    for (size_t i = 0; i < g->allocations.size(); i++)
        if (g->allocations[i].first == p) {
            g->bytes -= g->allocations[i].second;
            g->allocations.erase(g->allocations.begin() + i);
            break;
        }
    cudaFreeAsync(p, g->stream);
}

ga_status use_device(const ga_graph* g) {
    GA_CUDA(cudaSetDevice(g->device));
    return GA_OK;
}

static std::mutex g_pool_mu;
static constexpr uint64_t kPoolKeepDefault = 8ull << 30;   // bytes the pool keeps cached after frees, by default
static cudaMemPool_t g_pools[64] = {};

ga_status init_pool(int device) {
    if (device < 0 || device >= 64) return fail(GA_ERR_INVALID_ARGUMENT, "device %d out of range", device);
    std::lock_guard<std::mutex> lock(g_pool_mu);
    if (g_pools[device]) return GA_OK;
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    cudaMemPool_t pool;
    GA_CUDA(cudaMemPoolCreate(&pool, &props));
    uint64_t keep = kPoolKeepDefault;
    GA_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
    g_pools[device] = pool;
    return GA_OK;
}

static uint32_t g_pool_holders[64] = {};   // servers keeping their budget mapped, per device

ga_status pool_keep_at_least(int device, uint64_t bytes) {
    GA_TRY(init_pool(device));
    std::lock_guard<std::mutex> lock(g_pool_mu);
    uint64_t keep = 0;
    GA_CUDA(cudaMemPoolGetAttribute(g_pools[device], cudaMemPoolAttrReleaseThreshold, &keep));
    if (bytes > keep) GA_CUDA(cudaMemPoolSetAttribute(g_pools[device], cudaMemPoolAttrReleaseThreshold, &bytes));
    g_pool_holders[device]++;
    return GA_OK;
}

void pool_keep_release(int device) {
    if (device < 0 || device >= 64) return;
    std::lock_guard<std::mutex> lock(g_pool_mu);
    if (!g_pools[device] || !g_pool_holders[device] || --g_pool_holders[device]) return;
    // the last holder is gone: back to the default and hand the rest of the cached memory back to the driver
    uint64_t keep = kPoolKeepDefault;
    cudaMemPoolSetAttribute(g_pools[device], cudaMemPoolAttrReleaseThreshold, &keep);
    cudaMemPoolTrimTo(g_pools[device], keep);
}

// Slots of one 64 KB slab (allocated with the first handle) in a free list; beyond it every handle has its own block.
static std::mutex g_slot_mu;
static std::vector<unsigned long long*> g_slots_free;
static unsigned long long* g_slab = nullptr;
constexpr size_t kSlotWords = 64, kSlabSlots = 128;

unsigned long long* host_slot_acquire() {
    std::lock_guard<std::mutex> lock(g_slot_mu);
    if (!g_slab) {
        void* p = nullptr;
        if (cudaHostAlloc(&p, kSlabSlots * kSlotWords * 8, cudaHostAllocPortable | cudaHostAllocMapped) == cudaSuccess) {
            g_slab = (unsigned long long*)p;
            for (size_t i = kSlabSlots; i > 0; i--) g_slots_free.push_back(g_slab + (i - 1) * kSlotWords);
        } else {
            (void)cudaGetLastError();
        }
    }
    if (!g_slots_free.empty()) {
        unsigned long long* s = g_slots_free.back();
        g_slots_free.pop_back();
        return s;
    }
    void* p = nullptr;
    if (cudaHostAlloc(&p, kSlotWords * 8, cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
        (void)cudaGetLastError();
        return nullptr;
    }
    return (unsigned long long*)p;
}

void host_slot_release(unsigned long long* s) {
    if (!s) return;
    std::lock_guard<std::mutex> lock(g_slot_mu);
    if (g_slab && s >= g_slab && s < g_slab + kSlabSlots * kSlotWords) g_slots_free.push_back(s);
    else cudaFreeHost(s);
}

// Streams of destroyed handles, kept for the next ones (at most 16 per device): creating and destroying one costs more
// than everything else a small handle does on the host.
static std::mutex g_stream_mu;
static std::vector<cudaStream_t> g_streams[64];

cudaError_t stream_acquire(int device, cudaStream_t* st) {
    {
        std::lock_guard<std::mutex> lock(g_stream_mu);
        if (!g_streams[device].empty()) {
            *st = g_streams[device].back();
            g_streams[device].pop_back();
            return cudaSuccess;
        }
    }
    return cudaStreamCreateWithFlags(st, cudaStreamNonBlocking);
}

void stream_release(int device, cudaStream_t st) {
    {
        std::lock_guard<std::mutex> lock(g_stream_mu);
        if (g_streams[device].size() < 16) {
            g_streams[device].push_back(st);
            return;
        }
    }
    cudaStreamDestroy(st);
}

// Results of half a megabyte and more go to pageable memory through two page-locked buffers: the next piece crosses the
// link while several threads copy the last one out, whose time is mostly the page faults of a fresh array (6.8 MB: 1.1
// ms by one cudaMemcpy). At most four pairs of buffers exist in a process; a fifth concurrent download copies directly.
constexpr size_t kStageBytes = 1u << 20, kStageMin = 512 * 1024;
constexpr int kStages = 4, kStageThreads = 6;
static std::mutex g_stage_mu;
static char* g_stage[kStages] = {};
static bool g_stage_busy[kStages] = {};

static int stage_acquire() {
    std::lock_guard<std::mutex> lock(g_stage_mu);
    for (int i = 0; i < kStages; i++) {
        if (g_stage_busy[i]) continue;
        if (!g_stage[i] && cudaHostAlloc((void**)&g_stage[i], 2 * kStageBytes, cudaHostAllocPortable) != cudaSuccess) {
            (void)cudaGetLastError();
            g_stage[i] = nullptr;
            return -1;
        }
        g_stage_busy[i] = true;
        return i;
    }
    return -1;
}

ga_status download(ga_graph* g, void* dst, const void* src, size_t bytes) {
    cudaStream_t st = g->stream;
    int slot = -1;
    if (bytes >= kStageMin) {
        cudaPointerAttributes at;
        const bool pageable = cudaPointerGetAttributes(&at, dst) != cudaSuccess || at.type == cudaMemoryTypeUnregistered;
        (void)cudaGetLastError();
        if (pageable) slot = stage_acquire();
    }
    if (slot < 0) {
        if (bytes) GA_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st));
        GA_CUDA(cudaStreamSynchronize(st));
        return GA_OK;
    }
    cudaEvent_t ev[2] = {nullptr, nullptr};
    cudaError_t e = cudaEventCreateWithFlags(&ev[0], cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ev[1], cudaEventDisableTiming);
    const size_t pieces = (bytes + kStageBytes - 1) / kStageBytes;
    auto size_of = [&](size_t i) { return std::min(kStageBytes, bytes - i * kStageBytes); };
    auto start = [&](size_t i) {
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(g_stage[slot] + (i & 1) * kStageBytes, (const char*)src + i * kStageBytes, size_of(i),
                                cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaEventRecord(ev[i & 1], st);
    };
    start(0);
    for (size_t i = 0; i < pieces && e == cudaSuccess; i++) {
        if (i + 1 < pieces) start(i + 1);
        if (e == cudaSuccess) e = cudaEventSynchronize(ev[i & 1]);
        if (e != cudaSuccess) break;
        const char* from = g_stage[slot] + (i & 1) * kStageBytes;
        char* to = (char*)dst + i * kStageBytes;
        const size_t n = size_of(i), part = (n / kStageThreads + 4096) & ~(size_t)4095;
#pragma omp parallel for schedule(static, 1) num_threads(kStageThreads)
        for (int t = 0; t < kStageThreads; t++) {
            const size_t a = std::min(n, t * part), b = std::min(n, a + part);
            if (b > a) std::memcpy(to + a, from + a, b - a);
        }
    }
    if (e != cudaSuccess) cudaStreamSynchronize(st);   // no copy into the buffers is left behind
    for (cudaEvent_t v : ev)
        if (v) cudaEventDestroy(v);
    {
        std::lock_guard<std::mutex> lock(g_stage_mu);
        g_stage_busy[slot] = false;
    }
    GA_CUDA(e);
    return GA_OK;
}

cudaMemPool_t pool_of_current() {
    int device = 0;
    cudaGetDevice(&device);
    std::lock_guard<std::mutex> lock(g_pool_mu);
    return device >= 0 && device < 64 ? g_pools[device] : nullptr;
}

// The derived index (built once per handle, on the stream, without a synchronisation: the upload checks left every size
// it needs on the host).
static ga_status prepare_index(ga_graph* g) {
    if (g->index_ready) return GA_OK;
    if (g->misoriented)
        return fail(GA_ERR_INVALID_GRAPH, "CSR is not oriented by (degree, id) (graph.h:43-45): an edge points from "
                                          "the larger to the smaller endpoint, or an undirected edge is stored twice");
    cudaStream_t st = g->stream;
    const uint32_t n = g->n, m = g->m;
    auto drop = [&](auto*& p) {   // left by a build that failed half way
        dfree(g, p);
        p = nullptr;
    };
    drop(g->vrank); drop(g->order); drop(g->dout); drop(g->work);
    drop(g->pos); drop(g->colr); drop(g->osrc); drop(g->in_rng);
    GA_TRY(dalloc(g, &g->vrank, n));
    GA_TRY(dalloc(g, &g->order, n));
    GA_TRY(dalloc(g, &g->dout, n));
    GA_TRY(dalloc(g, &g->work, n));
    GA_TRY(dalloc(g, &g->pos, (size_t)n + 1));
    GA_TRY(dalloc(g, &g->colr, (size_t)g->octs * 8));
    GA_TRY(dalloc(g, &g->osrc, g->octs));
    GA_TRY(dalloc(g, &g->in_rng, m));
    if (n) {
        // the vertices in (degree, id) order
        const unsigned gv = grid_for((uint64_t)n + 1, 256);
        const uint32_t chunk = rank_chunk(n);
        const uint32_t nchunks = (uint32_t)(((uint64_t)n + chunk - 1) / chunk);
        const uint64_t ncounts = (uint64_t)kRankDigits * nchunks;
        uint32_t passes = 1;
        while (passes * kRankBits < 32 && (g->max_degree >> (passes * kRankBits)) != 0) passes++;
        Scratch s_other(st), s_counts(st);
        uint32_t *other, *counts;
        GA_TRY(s_other.alloc(&other, n));
        GA_TRY(s_counts.alloc(&counts, ncounts));
        const unsigned gr = (nchunks + kRankWarps - 1) / kRankWarps;
        const uint32_t* cur = nullptr;   // the identity (id order) before the first pass
        for (uint32_t ps = 0; ps < passes; ps++) {
            uint32_t* next = ((passes - ps) & 1) ? g->order : other;   // the last pass ends in order
            k_rank_count<<<gr, kRankWarps * 32, 0, st>>>(cur, g->deg, n, ps * kRankBits, nchunks, chunk, counts);
            GA_CUDA(cudaGetLastError());
            GA_TRY(scan_impl<uint32_t>(st, counts, counts, ncounts));
            k_rank_scatter<<<gr, kRankWarps * 32, 0, st>>>(cur, g->deg, n, ps * kRankBits, nchunks, chunk, counts, next);
            GA_CUDA(cudaGetLastError());
            cur = next;
        }
        k_places<<<gv, 256, 0, st>>>(g->rowptr, g->deg, g->order, n, g->vrank, g->dout, (unsigned long long*)g->pos);
        GA_CUDA(cudaGetLastError());
        GA_TRY(scan_impl<unsigned long long>(st, (unsigned long long*)g->pos, (unsigned long long*)g->pos,
                                             (uint64_t)n + 1));
        if (m) {
            Scratch s_cur(st), s_listed(st);
            unsigned long long* cur;
            uint32_t* listed;   // rows longer than 8, then their count
            GA_TRY(s_cur.alloc(&cur, n));
            GA_TRY(s_listed.alloc(&listed, (size_t)n + 1));
            GA_CUDA(cudaMemsetAsync(listed + n, 0, 4, st));
            k_in_cursors<<<gv, 256, 0, st>>>(g->pos, n, cur);
            GA_CUDA(cudaGetLastError());
            k_place_rows_small<<<grid_for((uint64_t)(n - g->isolated) * 8, 256), 256, 0, st>>>(
                g->rowptr, g->col, g->vrank, g->order, g->pos, g->isolated, n, g->colr, g->osrc, listed, listed + n);
            GA_CUDA(cudaGetLastError());
            if (g->max_out_degree > 8)
                k_place_rows_listed<<<(unsigned)g->sm_count * 8, 128, 0, st>>>(
                    g->rowptr, g->col, g->vrank, g->order, g->pos, g->colr, g->osrc, listed, listed + n);
            GA_CUDA(cudaGetLastError());
            k_in_lists<<<grid_for(g->octs * 8, 256, (unsigned)g->sm_count * 64), 256, 0, st>>>(
                g->colr, g->osrc, g->pos, g->octs * 8, cur, g->in_rng);
            GA_CUDA(cudaGetLastError());
            k_work<<<gv, 256, 0, st>>>(cur, n, g->work);
            GA_CUDA(cudaGetLastError());
        } else {
            GA_CUDA(cudaMemsetAsync(g->work, 0, (size_t)n * 4, st));
        }
    }
    g->index_ready = true;
    return GA_OK;
}

// The work items for the current light_max_deg / item_work (rebuilt when those change, e.g. by the autotuner trying
// candidates). Their number stays on the device (it_info); the arrays are sized by a bound: one item per anchor plus
// one per `item_work` probes, at most one per in-edge.
static ga_status prepare_items(ga_graph* g) {
    cudaStream_t st = g->stream;
    const uint32_t n = g->n, m = g->m;
    if (!n || !m) return GA_OK;
    const uint64_t bound = std::min<uint64_t>(m, (uint64_t)std::min(n, m) + g->row_work * 8 / g->item_work + 1);
    if (g->items_captured) {   // replays read those lists: they stay until the handle ends
        g->items = ga_items{};
        g->items_captured = false;
    }
    if (bound > g->items.capacity) {
        dfree(g, g->items.v); dfree(g, g->items.k0); dfree(g, g->items.k1);
        g->items.v = g->items.k0 = g->items.k1 = nullptr;
        g->items.capacity = 0;
        GA_TRY(dalloc(g, &g->items.v, bound));
        GA_TRY(dalloc(g, &g->items.k0, bound));
        GA_TRY(dalloc(g, &g->items.k1, bound));
        g->items.capacity = bound;
    }
    if (!g->items.info) GA_TRY(dalloc(g, &g->items.info, 3));
    g->items.bound = bound;
    Scratch s_cnt(st), s_tiny(st);
    unsigned long long* cnt;
    uint32_t* tiny;
    GA_TRY(s_cnt.alloc(&cnt, (size_t)n + 1));
    GA_TRY(s_tiny.alloc(&tiny, (size_t)n + 1));
    k_count_items<<<grid_for((uint64_t)n + 1, 256), 256, 0, st>>>(g->pos, g->dout, g->work, n, g->light_max_deg,
                                                                  g->item_work, cnt, tiny);
    GA_CUDA(cudaGetLastError());
    GA_TRY(scan_impl<unsigned long long>(st, cnt, cnt, (uint64_t)n + 1));
    GA_TRY(scan_impl<uint32_t>(st, tiny, tiny, (uint64_t)n + 1));
    k_emit_items<<<grid_for(bound, 256), 256, 0, st>>>(g->pos, cnt, tiny, n, g->items.v, g->items.k0, g->items.k1,
                                                       g->items.info);
    GA_CUDA(cudaGetLastError());
    return GA_OK;
}

ga_status not_captured(const ga_graph* g) {
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    GA_CUDA(cudaStreamIsCapturing(g->stream, &capture));
    return capture == cudaStreamCaptureStatusNone
               ? GA_OK
               : fail(GA_ERR_CUDA, "the graph's stream is being captured and the call would build structures it keeps: "
                                   "call ga_graph_prepare before the capture");
}

ga_status prepare(ga_graph* g) {
    if (g->prepared) return GA_OK;
    GA_TRY(use_device(g));
    GA_TRY(not_captured(g));
    GA_TRY(prepare_index(g));
    GA_TRY(prepare_items(g));
    if (!g->built) GA_CUDA(cudaEventCreateWithFlags(&g->built, cudaEventDisableTiming));
    GA_CUDA(cudaEventRecord(g->built, g->stream));
    g->prepared = true;
    return GA_OK;
}

bool index_stands(const ga_graph* g) {
    GA_GRAPH_LOCK(g);
    return g->prepared;
}

ga_status prepare_shards(ga_graph* g) {
    GA_TRY(prepare(g));
    if (g->anchor_work) return GA_OK;
    GA_TRY(not_captured(g));
    unsigned long long* w = nullptr;
    GA_TRY(dalloc(g, &w, (size_t)g->n + 1));
    k_widen<<<grid_for((uint64_t)g->n + 1, 256), 256, 0, g->stream>>>(g->work, g->n, w);
    const ga_status s = scan_u64(g, w, (uint64_t)g->n + 1);
    if (s == GA_OK) g->anchor_work = w;
    else dfree(g, w);
    return s;
}

// Runs `make` with g on another stream, behind the last build, and waits for it: what it builds is complete before a pass
// that needs it is recorded in the capture of g's own stream.
template <class F>
static ga_status beside_capture(ga_graph* g, F make) {
    cudaStream_t own = g->stream, side = nullptr;
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    GA_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
    ga_status s = GA_OK;
    if (stream_acquire(g->device, &side) != cudaSuccess) s = fail(GA_ERR_CUDA, "cudaStreamCreate failed");
    if (s == GA_OK && g->built && cudaStreamWaitEvent(side, g->built, 0) != cudaSuccess)
        s = fail(GA_ERR_CUDA, "cudaStreamWaitEvent failed");
    if (s == GA_OK) {
        g->stream = side;
        s = make();
        g->stream = own;
    }
    if (side && cudaStreamSynchronize(side) != cudaSuccess && s == GA_OK)
        s = fail(GA_ERR_CUDA, "building beside a capture failed");
    if (side) stream_release(g->device, side);
    cudaThreadExchangeStreamCaptureMode(&mode);
    return s;
}

ga_status prepare_enqueued(ga_graph* g, bool shards) {
    if (g->prepared && (!shards || g->anchor_work)) return GA_OK;
    const bool counted = g->counted_bare && !g->index_ready;   // nothing of the handle is pending on its stream
    if ((!g->prepared && !counted) || not_captured(g) == GA_OK) return shards ? prepare_shards(g) : prepare(g);
    clear_error();
    return beside_capture(g, [&] { return shards ? prepare_shards(g) : prepare(g); });
}

ga_status captured_work(ga_graph* g, ga_work** work) {
    if (!g->captured_left) {
        constexpr uint32_t kSlab = 64;
        GA_TRY(beside_capture(g, [&] { return dalloc(g, &g->captured, kSlab); }));
        g->captured_left = kSlab;
    }
    *work = g->captured++;
    g->captured_left--;
    return GA_OK;
}

static ga_status create_common(const uint32_t* rowptr, const uint32_t* col, uint32_t n, uint32_t m, int device,
                               void* stream, bool from_device, ga_graph** out) {
    if (!out) return fail(GA_ERR_INVALID_ARGUMENT, "out is null");
    *out = nullptr;
    if (!rowptr || (m && !col)) return fail(GA_ERR_INVALID_ARGUMENT, "null CSR array");
    if (n == UINT32_MAX) return fail(GA_ERR_INVALID_ARGUMENT, "n must be < 2^32 - 1");
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || count == 0) {
        (void)cudaGetLastError();
        return fail(GA_ERR_NO_DEVICE, "no CUDA device");
    }
    if (device < 0 || device >= count) return fail(GA_ERR_INVALID_ARGUMENT, "device %d out of range", device);
    if (!from_device && (rowptr[0] != 0 || rowptr[n] != m))
        return fail(GA_ERR_INVALID_GRAPH, "rowptr[0] must be 0 and rowptr[n] must equal m");
    ga_graph* g = new ga_graph();
    g->device = device;
    g->n = n;
    g->m = m;
    auto bail = [&](ga_status s) { ga_graph_destroy(g); return s; };
    if (cudaSetDevice(device) != cudaSuccess) return bail(fail(GA_ERR_CUDA, "cudaSetDevice(%d) failed", device));
    cudaDeviceGetAttribute(&g->sm_count, cudaDevAttrMultiProcessorCount, device);
    ga_status s;
    if ((s = init_pool(device)) != GA_OK) return bail(s);
    if (stream) {
        g->stream = (cudaStream_t)stream;
    } else {
        if (stream_acquire(device, &g->stream) != cudaSuccess)
            return bail(fail(GA_ERR_CUDA, "cudaStreamCreate failed"));
        g->own_stream = true;
    }
    if ((s = dalloc(g, &g->rowptr, (size_t)n + 1)) != GA_OK) return bail(s);
    if ((s = dalloc(g, &g->col, m)) != GA_OK) return bail(s);
    if ((s = dalloc(g, &g->d_scalars, 64)) != GA_OK) return bail(s);
    if ((s = dalloc(g, &g->sync, 1)) != GA_OK) return bail(s);
    if (!(g->h_scalars = host_slot_acquire())) return bail(fail(GA_ERR_OUT_OF_MEMORY, "page-locked slot failed"));
    cudaMemsetAsync(g->sync, 0, sizeof(ga_sync), g->stream);
    const cudaMemcpyKind kind = from_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
    if (cudaMemcpyAsync(g->rowptr, rowptr, ((size_t)n + 1) * 4, kind, g->stream) != cudaSuccess ||
        (m && cudaMemcpyAsync(g->col, col, (size_t)m * 4, kind, g->stream) != cudaSuccess))
        return bail(fail(GA_ERR_CUDA, "CSR copy to the device failed"));
    // the checks, with everything the index will be sized by, in one pass (results: d_scalars, SC_*)
    if ((s = dalloc(g, &g->src, m)) != GA_OK) return bail(s);
    if ((s = dalloc(g, &g->deg, n)) != GA_OK) return bail(s);
    cudaMemsetAsync(g->d_scalars, 0, 64 * 8, g->stream);
    if (n) {
        cudaMemsetAsync(g->deg, 0, (size_t)n * 4, g->stream);
        const unsigned few = (unsigned)g->sm_count * 8;   // one wave: the kernels end in per-block sums
        k_rows<<<grid_for(n, 256, few), 256, 0, g->stream>>>(g->rowptr, g->col, n, m, g->src, g->deg, g->d_scalars);
        k_degrees<<<grid_for(n, 256, few), 256, 0, g->stream>>>(g->rowptr, n, g->deg, g->d_scalars);
        if (m) k_orient<<<grid_for(m, 256), 256, 0, g->stream>>>(g->src, g->col, g->deg, n, m, g->d_scalars);
    }
    uint32_t ends[2] = {0, 0};
    cudaMemcpyAsync(g->h_scalars, g->d_scalars, 64 * 8, cudaMemcpyDeviceToHost, g->stream);
    if (from_device) {
        cudaMemcpyAsync(&ends[0], g->rowptr, 4, cudaMemcpyDeviceToHost, g->stream);
        cudaMemcpyAsync(&ends[1], g->rowptr + n, 4, cudaMemcpyDeviceToHost, g->stream);
    }
    if (cudaStreamSynchronize(g->stream) != cudaSuccess) {
        const char* why = cudaGetErrorString(cudaGetLastError());
        return bail(fail(GA_ERR_CUDA, "validation failed: %s", why));
    }
    if (from_device && (ends[0] != 0 || ends[1] != m))
        return bail(fail(GA_ERR_INVALID_GRAPH, "rowptr[0] must be 0 and rowptr[n] must equal m"));
    if (g->h_scalars[SC_ERR])
        return bail(fail(GA_ERR_INVALID_GRAPH, "invalid CSR (flags 0x%llx: 1 rowptr, 2 endpoint >= n, 4 self loop, "
                                               "8 row not strictly ascending)", g->h_scalars[SC_ERR]));
    g->max_out_degree = (uint32_t)g->h_scalars[SC_MAXOUT];
    g->max_degree = (uint32_t)g->h_scalars[SC_MAXDEG];
    g->isolated = (uint32_t)g->h_scalars[SC_ISOLATED];
    g->octs = g->h_scalars[SC_OCTS];
    g->row_work = g->h_scalars[SC_WORK];
    g->misoriented = g->h_scalars[SC_ORIENT] != 0;
    for (int b = 0; b < 33; b++) g->row_hist[b] = g->h_scalars[SC_HIST + b];
    *out = g;
    return GA_OK;
}

}  // namespace ga

using namespace ga;

extern "C" {

ga_status ga_device_count(int* count) {
    if (!count) return fail(GA_ERR_INVALID_ARGUMENT, "null argument");
    *count = 0;
    if (cudaGetDeviceCount(count) != cudaSuccess) {
        (void)cudaGetLastError();
        *count = 0;
    }
    return GA_OK;
}

ga_status ga_host_pinned_alloc(uint64_t bytes, void** out) {
    if (!out) return fail(GA_ERR_INVALID_ARGUMENT, "null argument");
    *out = nullptr;
    if (cudaMallocHost(out, bytes ? bytes : 1) != cudaSuccess) {
        (void)cudaGetLastError();
        *out = nullptr;
        return fail(GA_ERR_OUT_OF_MEMORY, "page-locked allocation of %llu bytes failed", (unsigned long long)bytes);
    }
    return GA_OK;
}

ga_status ga_host_pinned_free(void* p) {
    if (p && cudaFreeHost(p) != cudaSuccess) {
        (void)cudaGetLastError();
        return fail(GA_ERR_CUDA, "cudaFreeHost failed");
    }
    return GA_OK;
}

ga_status ga_graph_create(const uint32_t* rowptr, const uint32_t* col, uint32_t n, uint32_t m, int device,
                          void* stream, ga_graph** out) {
    return create_common(rowptr, col, n, m, device, stream, false, out);
}

ga_status ga_graph_create_device(const uint32_t* d_rowptr, const uint32_t* d_col, uint32_t n, uint32_t m, int device,
                                 void* stream, ga_graph** out) {
    return create_common(d_rowptr, d_col, n, m, device, stream, true, out);
}

ga_status ga_graph_destroy(ga_graph* g) {
    if (!g) return GA_OK;
    { GA_GRAPH_LOCK(g); }   // calls in flight on other threads finish first (none may start after this one)
    cudaSetDevice(g->device);
    if (g->stream) cudaStreamSynchronize(g->stream);
    destroy_loops(g);
    for (auto& a : g->allocations) cudaFreeAsync(a.first, g->stream);
    if (g->stream) cudaStreamSynchronize(g->stream);
    if (g->own_stream && g->stream) stream_release(g->device, g->stream);
    host_slot_release(g->h_scalars);
    if (g->built) cudaEventDestroy(g->built);
    delete g;
    return GA_OK;
}

ga_status ga_graph_set_stream(ga_graph* g, void* stream) {
    if (!g) return fail(GA_ERR_INVALID_ARGUMENT, "null graph");
    GA_GRAPH_LOCK(g);
    GA_TRY(use_device(g));
    GA_CUDA(cudaStreamSynchronize(g->stream));
    if (g->own_stream) { stream_release(g->device, g->stream); g->own_stream = false; }
    if (stream) {
        g->stream = (cudaStream_t)stream;
    } else {
        GA_CUDA(stream_acquire(g->device, &g->stream));
        g->own_stream = true;
    }
    return GA_OK;
}

ga_status ga_graph_device_bytes(const ga_graph* g, uint64_t* bytes) {
    if (!g || !bytes) return fail(GA_ERR_INVALID_ARGUMENT, "null argument");
    GA_GRAPH_LOCK(g);
    *bytes = g->bytes;
    return GA_OK;
}

ga_status ga_graph_prepare(ga_graph* g) {
    if (!g) return fail(GA_ERR_INVALID_ARGUMENT, "null graph");
    GA_GRAPH_LOCK(g);
    GA_TRY(use_device(g));
    const bool builds = !g->prepared || (g->opt_tc_kernel == 0 && !g->tuned_kernel);
    GA_TRY(ready(g));
    if (builds) GA_CUDA(cudaStreamSynchronize(g->stream));   // the call ends with the structures built, not enqueued
    return GA_OK;
}

ga_status ga_graph_set_option(ga_graph* g, ga_option opt, int64_t value) {
    if (!g) return fail(GA_ERR_INVALID_ARGUMENT, "null graph");
    GA_GRAPH_LOCK(g);
    if (value < 0) return fail(GA_ERR_INVALID_ARGUMENT, "option values are >= 0");
    switch (opt) {
        case GA_OPT_TC_KERNEL:
            if (value > 2) return fail(GA_ERR_INVALID_ARGUMENT, "GA_OPT_TC_KERNEL is 0, 1 or 2");
            g->opt_tc_kernel = value;
            return GA_OK;
        case GA_OPT_LOOP_MODE:
            if (value > 2) return fail(GA_ERR_INVALID_ARGUMENT, "GA_OPT_LOOP_MODE is 0, 1 or 2");
            g->opt_loop_mode = value;
            return GA_OK;
        case GA_OPT_MAX_ROUNDS:
            g->opt_max_rounds = value;
            return GA_OK;
        case GA_OPT_UPDATE_MODE:
            if (value > 2) return fail(GA_ERR_INVALID_ARGUMENT, "GA_OPT_UPDATE_MODE is 0, 1 or 2");
            if (value != g->opt_update_mode) {
                GA_TRY(use_device(g));
                reset_loops(g);
                g->opt_update_mode = value;
            }
            return GA_OK;
        case GA_OPT_ITEM_WORK: {   // 0: the autotuner's choice (4096 until it has run)
            const uint32_t v = value ? (uint32_t)std::min<int64_t>(value, 1 << 30) : 4096;
            g->item_work_set = value != 0;
            if (v != g->item_work) { g->item_work = v; g->prepared = false; }
            g->tuned_kernel = 0;
            return GA_OK;
        }
        case GA_OPT_COUNT_BITMAP:
            if (value > 1) return fail(GA_ERR_INVALID_ARGUMENT, "GA_OPT_COUNT_BITMAP is 0 or 1");
            g->opt_count_bitmap = value;
            return GA_OK;
        case GA_OPT_HEAVY_TABLE_BITS:
            if (value != 0 && (value < 3 || value > 13))
                return fail(GA_ERR_INVALID_ARGUMENT, "GA_OPT_HEAVY_TABLE_BITS is 0 or 3..13");
            g->heavy_bits_cap = (uint32_t)value;
            return GA_OK;
        case GA_OPT_LIGHT_MAX_DEG: {   // 0: the autotuner's choice (128 until it has run)
            const uint32_t v = value ? (uint32_t)std::min<int64_t>(value, 256) : 128;
            g->light_max_deg_set = value != 0;
            if (v != g->light_max_deg) { g->light_max_deg = v; g->prepared = false; }
            g->tuned_kernel = 0;
            return GA_OK;
        }
    }
    return fail(GA_ERR_INVALID_ARGUMENT, "unknown option %d", (int)opt);
}

}  // extern "C"
