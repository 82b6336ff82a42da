// Batched and plain multi-source delta-stepping kernels with the fused APSP epilogue (sm_100a).
//
// Both kernels are persistent: one CTA per workspace slot, each CTA takes source tiles from a device work counter until
// none are left. A tile is either NGX_TILE sources (batched form: lane s of every warp owns source s of the tile) or
// one source (plain form: the lanes of a warp stride over one vertex's arcs).
//
// Per tile the CTA runs delta-stepping with a common bucket bound theta for all its sources:
//   near phase   vertices whose pending (vertex, source) pairs lie below theta are expanded; an improvement below
//                theta marks the pair pending for the next iteration, one at or above theta marks it "far"; after
//                the iteration the next queue is compacted from the pending masks (warp ballot + prefix);
//   bucket step  when no near work is left, theta becomes (floor(d_min / delta) + 1) * delta, where d_min, the smallest
//                pending distance, was gathered by the relaxations that set far marks; one pass over the marks then moves
//                the pairs below theta to the near queue and finds the smallest that stays.
// Relaxation is fl(d[u] + len) compared and stored with a 64-bit atomicMin on the bit pattern, which orders
// non-negative doubles like their values. The label-correcting fixed point is the same as the reference Dijkstra's
// (PriorityQueueVariant.h:47-93: d[v] = min over arcs of fl(d[u] + |w|)), so distances are bit-identical.
//
// Race-freedom of the pending marks: expansions of iteration k read and clear pend[k % 2]; improvements made during
// iteration k set pend[(k + 1) % 2] and the far marks; iterations are separated by (group) barriers. A pair improved
// while its vertex is being expanded is therefore always expanded again in the next iteration, with the new distance.
// All distance reads go through L2 (__ldcg), where the atomics are performed.
//
// Epilogue (after a tile's distances are final), per (vertex, source), replacing summarize_distances
// (types/SsspResult.h:42-64) and the aggregation of AllPairsShortestPath::compute_apsp_impl (:110-163): unreachable
// count, exact sums of d and of 1/d (order-independent integer accumulators, rounded once), maximum finite distance,
// traversed arcs, and the distance histogram (bin floor(d / (hist_max / bins)), clamped to the last bin, as
// FixedSizeHistogram::add_data_point, external/cpp-utility/data-structure/Histogram.hpp:166-180). The distances are
// reset to +inf in the same pass, so the N x N distances never leave the per-CTA workspace.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "brandes_kernels.cuh"
#include "ngx_common.cuh"
#include "ngx_group.cuh"

namespace ngx {

constexpr unsigned kFullMask = 0xFFFFFFFFu;

struct TileOutputs {
    unsigned long long* acc_sum;    // per graph: kAccDigits words of the exact sum of distances, then kAccDigits for 1/d
    unsigned long long* acc_inv;    // unused by the tile kernel (acc_sum + kAccDigits of each graph)
    unsigned long long* counters;   // per graph: kCounterCount words (see Counter)
    unsigned long long* hist;       // per graph: hist_bins words (or nullptr)
    int hist_bins;
    double hist_width;
    double hist_max;
    double* src_sum;                // per tile position (or nullptr)
    double* src_max;
    double* src_inv;
    unsigned long long* src_unreach;
    unsigned long long* src_arcs;
    double* rows;                   // num_sources x n distance rows (or nullptr)
};


struct SsspParams {
    DeviceCsr g;                   // concatenated CSR: row_ptr over all graphs' rows, arcs with graph-local targets; g.n = largest n
    const int32_t* sources;        // tile order (graph-local ids)
    int64_t num_sources;
    int64_t num_tiles;             // work items
    double delta;
    const GraphDesc* graphs;       // batch table (tile kernel)
    // distances from and to the landmarks, kTile rows of num_vertices each (nullptr: none), see landmark_bounds
    const double* landmark_from;
    const double* landmark_to;
    const WorkItem* items;         // work items in scheduling order, or nullptr: tile t of graph 0
    unsigned long long max_iterations;  // per tile
    unsigned long long* tile_counter;
    int* error;
    const volatile int* abort_flag;
    // workspace, carved per slot (blockIdx.x)
    unsigned long long* ws_dist;   // slots * n * width (width = kTile batched, 1 plain)
    uint32_t* ws_pend;             // slots * 3n: two pending masks (alternating by iteration parity) and the far marks
    int32_t* ws_queue;             // slots * 2n
    uint32_t* ws_stamp;            // slots * n; tile kernel: the distance phase's bound[], then the DAG passes' stamps
    // reach lists (graphs of several strongly connected components; nullptr otherwise): per vertex the tile's
    // sources that reached it, and the list of the vertices reached, so that per-tile passes visit only those
    uint32_t* ws_reach;            // slots * n
    int32_t* ws_touched;           // slots * n
    // groups: the CTAs blockIdx.x / group_size share slot (blockIdx.x / group_size) and its tiles
    int group_size;
    int64_t group_stride;          // words of group storage per slot (group_stride_words)
    unsigned long long* group_ws;  // slots * group_stride words, zero at launch
    TileOutputs out;
};

// Bytes of per-slot workspace for a graph with n vertices.
inline size_t sssp_slot_bytes(int64_t n, int width) {
    return static_cast<size_t>(n) * (static_cast<size_t>(width) * 8 + 4 * 2 + 4 + 4 * 2 + 4) + 256;
}


__device__ __forceinline__ double next_theta(double d_min, double delta) {
    const double theta = (floor(__ddiv_rn(d_min, delta)) + 1.0) * delta;
    return theta > d_min ? theta : INFINITY;
}

// Control block of the CTAs working on one tile: one per workspace slot in global memory, and a copy in each CTA's
// shared memory that every group barrier refreshes (ngx_group.cuh). Only atomics and barrier updates change it.
struct TileShared {
    long long tile;
    int qlen[2];
    int cur;
    int bucket_len;                 // bucket step: entries pushed so far (qlen[cur] is still being read as 0 by late warps)
    int stop;
    unsigned stamp;                 // id of the DAG pass about to run (dedup of its level lists)
    double theta;
    unsigned long long min_bits;    // a lower bound of the smallest pending far distance (+inf: none is pending)
    unsigned long long min_left;    // bucket step: smallest far distance that stays far
    unsigned long long iterations;
    unsigned long long overflow;    // histogram overflow of the tile (plain form)
    // Brandes / adjoint levels
    unsigned level;
    int lvl_start;
    int lvl_len;
    int next_len;
    unsigned long long active_pairs;  // reached (vertex, source) pairs other than the sources, counted by the DAG pass
    unsigned long long dag_arcs;      // DAG arcs of all the tile's sources, counted by the DAG pass
    int grab;                       // next queue entry handed to a warp in the current near iteration
    int touched_len;                // vertices the tile has reached so far (reach lists; see SsspParams::ws_touched)
    // the state of a CTA that left its group (ngx_group.cuh): no tile, nothing queued, pending or levelled
    __device__ void halt() {
        stop = 1;
        tile = 0x7FFFFFFFFFFFFFFFll;
        qlen[0] = 0;
        qlen[1] = 0;
        min_bits = kInfBits;
        level = 0u;
        lvl_start = 0;
        lvl_len = 0;
    }
};
static_assert(sizeof(TileShared) % 8 == 0, "TileShared is copied in 8-byte words");

// Per-slot group storage, in 8-byte words: the control block, the barrier, one scan partial per CTA, and (groups of
// several CTAs) the per-source epilogue sums: exact accumulators of d and 1/d, unreachable, arcs and maximum per source.
constexpr int kCtlWords = static_cast<int>(sizeof(TileShared) / 8);
constexpr int kGroupAccWords = 2 * kTile * kAccDigits + 3 * kTile;
inline int64_t group_stride_words(int group_size) {
    const int64_t words = kCtlWords + 1 + group_size + (group_size > 1 ? kGroupAccWords : 0);
    return (words + 31) / 32 * 32;  // 256-byte aligned slots
}

// This CTA's view of its tile group (see SsspParams::group_*). A group of one CTA keeps the control block in the CTA's
// shared memory (`local`), where its counters are shared-memory atomics; larger groups keep it in global memory.
template <typename Params>
__device__ __forceinline__ Group<TileShared> tile_group(const Params& p, TileShared* local) {
    unsigned long long* const gws = p.group_ws + (blockIdx.x / p.group_size) * p.group_stride;
    TileShared* const ctl = p.group_size == 1 ? local : reinterpret_cast<TileShared*>(gws);
    return Group<TileShared>{ ctl, reinterpret_cast<GroupBarrier*>(gws + kCtlWords), gws + kCtlWords + 1, p.group_size,
                              static_cast<int>(blockIdx.x % p.group_size), p.error };
}

// Smallest of the lanes' values, in every lane.
__device__ __forceinline__ unsigned long long warp_min(unsigned long long x) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const unsigned long long o = __shfl_xor_sync(kFullMask, x, off);
        x = o < x ? o : x;
    }
    return x;
}

// Queue entries a warp takes at a time (guided self-scheduling): the entries not yet handed out over twice the group's
// warps, clamped to 1..32, so a near iteration starts with large chunks (one round of loads serves many entries) and ends
// with single entries (an expansion can be work for a whole warp: a coarse last chunk would leave the other warps of
// the group waiting at the barrier that closes the iteration). Where entries are small (mean out-degree below
// kFilterDegree) packed_expand works several in the time of one, and a warp takes its whole share, up to 8, at once.
__device__ __forceinline__ int expand_chunk(int remaining, int group_warps, bool small_entries) {
    int c = remaining / (2 * group_warps);
    if (small_entries && c < 8) {
        const int share = remaining / group_warps;
        c = share < 8 ? share : 8;
    }
    return c < 1 ? 1 : (c > 32 ? 32 : c);
}

// The reach list of a tile: mask[v] has bit s set once source s reached v; a vertex is appended to list[] (length
// *len) by the relaxation that gives it its first finite distance of the tile. Disabled when mask is nullptr.
struct Reach {
    uint32_t* mask;
    int32_t* list;
    int* len;
    __device__ __forceinline__ void add(int v, uint32_t bit) const {
        if (atomicOr(&mask[v], bit) == 0u) {
            list[atomicAdd(len, 1)] = v;
        }
    }
};

// Arcs of one vertex that batched_expand filters together (four per lane).
constexpr int kArcBlock = 128;

// One queue entry a warp has taken: a vertex, its pending sources, its first arc and out-degree.
struct __align__(16) QueueEntry {
    int v;
    uint32_t mask;
    uint32_t beg;
    int deg;
};

// A warp's scratch in the distance phase. Keeping the chunk's entries here and the pointers in ExpandArgs leaves the
// registers to the reads in flight: with all of it in registers the compiler spilled the records just read, so that each
// read was waited for before the next was issued (measured on the 100,000-vertex connectome, 16 warps x 2 CTAs per SM:
// 3700 cycles for a vertex's four arc reads per lane, 1500 without spills).
struct WarpScratch {
    Arc kept[kArcBlock];     // arcs that passed the filter (batched_expand); id = position in the row
    QueueEntry entry[32];    // the chunk
    int rank[32];            // pending sources by rank (batched_expand), entry << 5 | source (packed_expand)
};

// A warp's share of the run's work counters.
struct WarpWork {
    unsigned long long expansions;
    unsigned long long lane_expansions;
};

// Near iterations between two looks at the abort flag: it lies in host memory, and the read (about a microsecond over
// PCIe) would be on the path of every iteration's barrier. A power of two.
constexpr unsigned long long kAbortPoll = 8;

constexpr int kMaxWarps = 16;
constexpr int kAccBytes = 2 * kTile * kAccDigits * 8;

// Per-tile arguments of the distance phase, in shared memory.
struct ExpandArgs {
    const Arc* arcs;
    const int64_t* row_ptr;
    const Arc* rarcs;             // in-arcs (DAG passes)
    const int64_t* rrow_ptr;
    unsigned long long* dist;
    uint32_t* marks;              // pending masks of even and odd iterations, far marks: three times n_slot words
    int32_t* queue;               // two queues of n_slot entries
    uint8_t* bound;
    int* grab;
    Reach reach;
    uint32_t n_slot;
    int nsrc;
    int bound_base;
    int group_warps;
    int n;
    int small_entries;
};

// Dynamic shared memory of the tile kernel, before the histogram. The warp scratch of the distance phase and of the DAG
// passes overlays the epilogue's accumulators (2 x kTile x kAccDigits words, which the epilogue zeroes first) and, after
// them, the scan partials of the DAG phase.
struct __align__(16) TileSmem {
    WarpScratch warp[kMaxWarps];
    WarpWork work[kMaxWarps];
    ExpandArgs args;
    TileShared ctl;
};
static_assert(sizeof(WarpScratch) * kMaxWarps >= kAccBytes + (512 + 3) * 8, "accumulators and scan partials fit in the warp scratch");
static_assert(sizeof(TileSmem) % 16 == 0, "the histogram follows");

// The relaxations of kUnroll arcs by this lane's source, their loads done: arc u relaxes d[x[u]][src] with nd[u] (cur[u] =
// the distance read before); an infinite nd[u] relaxes nothing. The atomic minima are issued back to back and not waited
// for, then the marks. dist_s points at the source's column. With reach lists (kReach) the old value is needed: the first
// finite distance of (x, s) appends x to the tile's reached vertices.
template <int kUnroll, bool kReach>
__device__ __forceinline__ void relax_lane(const int (&x)[kUnroll], int src, const double (&nd)[kUnroll], const unsigned long long (&cur)[kUnroll],
                                           unsigned long long* dist_s, const TileSmem& sh, unsigned long long& far_min) {
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
        const unsigned long long nb = static_cast<unsigned long long>(__double_as_longlong(nd[u]));
        if (nb < cur[u]) {
            atomicMin(&dist_s[static_cast<int64_t>(x[u]) * kTile], nb);
        }
    }
    const uint32_t bit = 1u << src;
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
        if (static_cast<unsigned long long>(__double_as_longlong(nd[u])) < cur[u]) {
            if (kReach && cur[u] == kInfBits) {
                sh.args.reach.add(x[u], bit);
            }
            uint32_t which = static_cast<uint32_t>(sh.ctl.cur ^ 1);
            if (!(nd[u] < sh.ctl.theta)) {
                which = 2u;
                const unsigned long long nb = static_cast<unsigned long long>(__double_as_longlong(nd[u]));
                far_min = nb < far_min ? nb : far_min;
            }
            atomicOr(&sh.args.marks[static_cast<size_t>(which) * sh.args.n_slot + static_cast<uint32_t>(x[u])], bit);
        }
    }
}

// ------------------------------------------------------------------------------------------ batched form
// A bound is one byte, so that the bounds of 100,000 vertices fit in a fair part of an SM's L1: the exponent and five
// mantissa bits of the row maximum (steps of 3 %), counted from a quarter of the bucket width (8 octaves: up to 64
// bucket widths). kNoBound stands for unknown and for anything larger. Truncation keeps the order of non-negative
// doubles, so key(a) > key(b) implies a > b.
constexpr int kNoBound = 255;
__device__ __forceinline__ int bound_key(uint32_t hi, int base) { return static_cast<int>(hi >> 15) - base; }
// Read through L1 (unlike the distances): the tile's group barriers order a reader after the reset of the tile before,
// and within a tile a stale bound is only weaker. volatile: not moved across a barrier.
__device__ __forceinline__ int ld_bound(const uint8_t* p) {
    uint32_t v;
    asm volatile("ld.global.L1::evict_last.u8 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return static_cast<int>(v);
}
// An arc record that this SM is not expected to read again soon: it does not displace the bounds from L1.
__device__ __forceinline__ Arc ldg_arc_once(const Arc* p) {
    int4 v;
    asm("ld.global.nc.L1::no_allocate.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return Arc{ v.x, v.y, __hiloint2double(v.w, v.z) };
}

// Vertices with fewer arcs are not filtered: at out-degree 6 (integer weights) 84 % of the arcs pass, at 20 and more
// (log-normal and integer weights) 36-60 % of the (arc, source) pairs remain.
constexpr int kFilterDegree = 16;

// Expands vertex v for the k sources pending on it, in two steps.
// 1. The arc filter. bound[x] is an upper bound of every d[x][s] of the tile: each expansion of x reads its whole
//    distance row (256 contiguous bytes) and stores the key of the row's maximum. Distances only decrease, so a bound
//    never becomes false and a stale one is only weaker. With d_min the smallest pending distance of v, an arc (v, x)
//    whose fl(d_min + len) has a larger key than bound[x] is longer than every final d[x][s]: its relaxations can
//    neither improve nor tie with any of them (fl is monotone), so the arc is dropped for a one-byte read instead of k
//    8-byte reads.
// 2. The pair loop. Each lane keeps one pending source for all its pairs (lane mod k' of them, k' = k rounded up to a
//    power of two) and takes every (32 / k')-th kept arc, so a pair costs one shared-memory read, an addition, a distance
//    read and a comparison; up to half of the lanes idle when k is just above a power of two, which is cheaper than
//    finding each pair's arc and source anew (three shuffles and a carry per pair).
// An improvement below theta sets the pair's bit in pend_nxt (the next iteration's queue is compacted from those
// masks after the iteration), one at or above theta its far mark. The kUnroll relaxations of a lane are issued back
// to back and waited for together.
// The atomic minimum is not waited for. An improvement is judged against the distance read before it, so
// a relaxation that lost a race to a smaller value may still set a pending bit or a far mark: the pair is then
// expanded once more with its (smaller) current distance, or its superseded far mark is cleared or moved by the next
// expansion or bucket step, which changes the work and never the fixed point.
// The caller has taken v's pending mask (entry.mask, non-zero) and cleared it and v's superseded far marks: see
// expand_queue. Lanes >= nsrc hold no source.
template <int kUnroll, bool kReach>
__device__ __forceinline__ void batched_expand(TileSmem& sh, WarpScratch& w, WarpWork& work, int j, int lane, unsigned long long& far_min) {
    const QueueEntry entry = w.entry[j];
    const uint32_t amask = entry.mask;
    unsigned long long* const dist = sh.args.dist;
    const Arc* const arcs = sh.args.arcs + entry.beg;
    const int64_t vrow = static_cast<int64_t>(entry.v) * kTile + lane;
    const unsigned long long row_bits = __ldcg(&dist[vrow]);
    const int old_bound = ld_bound(&sh.args.bound[entry.v]);
    const uint32_t row_hi = static_cast<uint32_t>(row_bits >> 32);
    const int bound_base = sh.args.bound_base;
    const uint32_t row_max = __reduce_max_sync(kFullMask, lane < sh.args.nsrc ? row_hi : 0u);
    const int max_key = bound_key(row_max, bound_base);
    if (lane == 0 && max_key < old_bound) {
        sh.args.bound[entry.v] = static_cast<uint8_t>(max_key > 0 ? max_key : 0);
    }
    const uint32_t min_hi = __reduce_min_sync(kFullMask, ((amask >> lane) & 1u) != 0u ? row_hi : 0xFFFFFFFFu);
    const double d_min = __hiloint2double(static_cast<int>(min_hi), 0);  // at most every pending distance
    const int k = __popc(amask);
    // this lane's source: the r-th pending one, r = lane mod k rounded up to a power of two (no source for r >= k), and
    // its distance to v
    if ((amask >> lane) & 1u) {
        w.rank[__popc(amask & lanemask_lt())] = lane;
    }
    if (lane == 0) {
        work.expansions += 1ull;
        work.lane_expansions += static_cast<unsigned long long>(k);
    }
    __syncwarp();
    const int log_k = 32 - __clz(k - 1);
    const int r = lane & ((1 << log_k) - 1);
    const int src = r < k ? w.rank[r] : 0;
    const double dvs = __longlong_as_double(static_cast<long long>(__shfl_sync(kFullMask, row_bits, src)));
    unsigned long long* const dist_s = dist + src;
    const int first_a = r < k ? lane >> log_k : kArcBlock;  // this lane's first kept arc of a block
    const int step_a = 32 >> log_k;
    const bool filter = entry.deg >= kFilterDegree;
    for (int a0 = 0; a0 < entry.deg; a0 += kArcBlock) {
        int kept = 0;
        {
            Arc arc[kArcBlock / 32];
            int ub[kArcBlock / 32];
            const uint8_t* const bound = sh.args.bound;
#pragma unroll
            for (int u = 0; u < kArcBlock / 32; ++u) {
                // a lane past the last arc reads the last one again and keeps nothing
                const int i = a0 + u * 32 + lane;
                arc[u] = ldg_arc_once(&arcs[i < entry.deg ? i : entry.deg - 1]);
            }
#pragma unroll
            for (int u = 0; u < kArcBlock / 32; ++u) {
                ub[u] = filter ? ld_bound(&bound[arc[u].col]) : kNoBound;
            }
#pragma unroll
            for (int u = 0; u < kArcBlock / 32; ++u) {
                const int i = a0 + u * 32 + lane;
                const int key = bound_key(static_cast<uint32_t>(__double2hiint(__dadd_rn(d_min, arc[u].len))), bound_base);
                const bool keep = i < entry.deg && (key <= ub[u] || ub[u] == kNoBound);
                const unsigned bal = __ballot_sync(kFullMask, keep);
                if (keep) {
                    w.kept[kept + __popc(bal & lanemask_lt())] = Arc{ arc[u].col, i, arc[u].len };
                }
                kept += __popc(bal);
            }
        }
        __syncwarp();
        int a = first_a;
        for (int a_warp = 0; a_warp < kept; a_warp += step_a * kUnroll) {
            int x[kUnroll];
            double nd[kUnroll];
            unsigned long long cur[kUnroll];
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) {
                // a lane without a pair reads the first kept arc's and relaxes nothing
                const Arc kept_arc = w.kept[a < kept ? a : 0];
                x[u] = kept_arc.col;
                nd[u] = a < kept ? __dadd_rn(dvs, kept_arc.len) : INFINITY;
                cur[u] = __ldcg(&dist_s[static_cast<int64_t>(x[u]) * kTile]);
                a += step_a;
            }
            relax_lane<kUnroll, kReach>(x, src, nd, cur, dist_s, sh, far_min);
        }
        __syncwarp();  // the next block of arcs (the next vertex) overwrites kept (and rank)
    }
}

// Queue entries with fewer (arc, pending source) pairs than this leave most of a warp idle in batched_expand (32 lanes,
// several arcs per lane in flight); consecutive ones are expanded together by packed_expand.
constexpr int kPackPairs = 64;

// Expands a group of m small queue entries together: w.rank[t], t < ktot <= 32, names the t-th (entry, pending source) of
// the group. Lane t takes it and walks its entry's arcs, kUnroll at a time: the lanes of an entry read the same arc
// records and neighbouring distances of the same rows, no lane needs to find its pairs, and the group takes as long as
// its entry with the most arcs. The relaxations and the counters are batched_expand's; the arcs are not filtered (a bound
// read per arc would cost as much as the few distance reads it saves).
template <int kUnroll, bool kReach>
__device__ __forceinline__ void packed_expand(TileSmem& sh, WarpScratch& w, WarpWork& work, int m, int ktot, int lane,
                                              unsigned long long& far_min) {
    const int code = w.rank[lane < ktot ? lane : 0];
    const int src = code & 31;
    const QueueEntry entry = w.entry[code >> 5];
    unsigned long long* const dist_s = sh.args.dist + src;
    const unsigned long long v_bits = __ldcg(&dist_s[static_cast<int64_t>(entry.v) * kTile]);
    if (lane == 0) {
        work.expansions += static_cast<unsigned long long>(m);
        work.lane_expansions += static_cast<unsigned long long>(ktot);
    }
    const int deg = lane < ktot ? entry.deg : 0;
    const int most = __reduce_max_sync(kFullMask, deg);
    const int with_arcs = __ffs(__ballot_sync(kFullMask, deg > 0)) - 1;
    const uint32_t some_beg = __shfl_sync(kFullMask, entry.beg, with_arcs < 0 ? 0 : with_arcs);
    const double dvs = __longlong_as_double(static_cast<long long>(v_bits));
    const Arc* const arcs = sh.args.arcs + (deg > 0 ? entry.beg : some_beg);
    for (int a0 = 0; a0 < most; a0 += kUnroll) {
        int x[kUnroll];
        double nd[kUnroll];
        unsigned long long cur[kUnroll];
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
            // a lane past its last arc reads its first one again (a lane without arcs: another lane's) and relaxes nothing
            const int a = a0 + u;
            const Arc arc = ldg_arc(&arcs[a < deg ? a : 0]);
            x[u] = arc.col;
            nd[u] = a < deg ? __dadd_rn(dvs, arc.len) : INFINITY;
            cur[u] = __ldcg(&dist_s[static_cast<int64_t>(x[u]) * kTile]);
        }
        relax_lane<kUnroll, kReach>(x, src, nd, cur, dist_s, sh, far_min);
    }
}

// One near iteration of a tile: the warps of the group take the queue in chunks (expand_chunk) from a shared counter;
// lane j fetches entry j's vertex, its pending mask, far marks and row offsets (one round of parallel loads), clears the
// mask and the superseded far marks, and the warp then expands the vertices one after another: one at a time when a
// vertex has a loop iteration's worth of (arc, source) pairs or more, else with its small neighbours in the chunk.
// Not inlined: the registers of the other phases are saved around the call instead of being spilled inside its loops.
template <int kUnroll, bool kReach>
__device__ __noinline__ void expand_queue(unsigned long long* min_bits) {
    extern __shared__ __align__(16) unsigned long long smem[];
    TileSmem& sh = *reinterpret_cast<TileSmem*>(smem);
    const int lane = threadIdx.x & 31;
    WarpScratch& w = sh.warp[threadIdx.x >> 5];
    WarpWork& work = sh.work[threadIdx.x >> 5];
    unsigned long long far_min = kInfBits;
    for (;;) {
        int base = 0;
        int chunk = 0;
        const int qlen = sh.ctl.qlen[sh.ctl.cur];
        if (lane == 0) {
            // the grab counter is in shared memory for single-CTA tiles and in global memory for groups: a volatile
            // generic load reads either (for global memory, from L2)
            int* const grab = sh.args.grab;
            chunk = expand_chunk(qlen - *reinterpret_cast<volatile int*>(grab), sh.args.group_warps, sh.args.small_entries != 0);
            base = atomicAdd(grab, chunk);
        }
        base = __shfl_sync(kFullMask, base, 0);
        chunk = __shfl_sync(kFullMask, chunk, 0);
        if (base >= qlen) {
            break;
        }
        const int count = qlen - base < chunk ? qlen - base : chunk;
        QueueEntry mine{ 0, 0u, 0u, 0 };
        if (lane < count) {
            const uint32_t n_slot = sh.args.n_slot;
            const int cur = sh.ctl.cur;
            uint32_t* const pend_cur = sh.args.marks + static_cast<size_t>(cur) * n_slot;
            uint32_t* const far = sh.args.marks + static_cast<size_t>(2) * n_slot;
            mine.v = __ldcg(&sh.args.queue[static_cast<size_t>(cur) * n_slot + static_cast<uint32_t>(base + lane)]);
            mine.mask = __ldcg(&pend_cur[mine.v]);
            const uint32_t fm = __ldcg(&far[mine.v]);
            const int64_t beg = __ldg(&sh.args.row_ptr[mine.v]);
            mine.beg = static_cast<uint32_t>(beg);  // arc indices are 32-bit, as in the reverse CSR
            mine.deg = static_cast<int>(__ldg(&sh.args.row_ptr[mine.v + 1]) - beg);
            if (mine.mask != 0u) {
                pend_cur[mine.v] = 0u;
                if (fm & mine.mask) {
                    atomicAnd(&far[mine.v], ~mine.mask);  // those far marks are superseded by the near values expanded now
                }
            }
        }
        w.entry[lane] = mine;
        __syncwarp();
        // entries with fewer pairs than one loop iteration holds go in groups (packed_expand), the others one by one
        const int kj = __popc(mine.mask);
        const unsigned any_mask = __ballot_sync(kFullMask, mine.mask != 0u);
        const unsigned small_mask = __ballot_sync(kFullMask, mine.mask != 0u && kj * mine.deg < kPackPairs);
        int j = 0;
        while (j < count) {
            const unsigned rest = any_mask & ~((1u << j) - 1u);
            if (rest == 0u) {
                break;
            }
            j = __ffs(rest) - 1;  // the next entry with pending sources
            if ((small_mask >> j) & 1u) {
                // the small entries from j up to the next large one, as many as hold 32 pending sources
                const unsigned large_after = any_mask & ~small_mask & ~((1u << j) - 1u);
                const int stop = large_after != 0u ? __ffs(large_after) - 1 : 32;
                const unsigned run = small_mask & ~((1u << j) - 1u) & (stop >= 32 ? kFullMask : ((1u << stop) - 1u));
                const bool in_run = (run >> lane) & 1u;
                const int kl = in_run ? __popc(w.entry[lane].mask) : 0;
                int kin = kl;
#pragma unroll
                for (int off = 1; off < 32; off <<= 1) {
                    const int ku = __shfl_up_sync(kFullMask, kin, off);
                    if (lane >= off) {
                        kin += ku;
                    }
                }
                const bool in_fit = in_run && kin <= 32;
                const unsigned fit = __ballot_sync(kFullMask, in_fit);
                const int m = __popc(fit);
                const int most = __reduce_max_sync(kFullMask, in_fit ? w.entry[lane].deg : 0);
                // lane by lane the group takes `most` steps, kUnroll at a time; one by one, each entry takes a round of
                // filter reads and one or two of distance reads
                if (m > 1 && most <= 4 * m) {
                    if (in_fit) {
                        int at = kin - kl;
                        for (uint32_t mask = w.entry[lane].mask; mask != 0u; mask &= mask - 1u) {
                            w.rank[at++] = lane << 5 | (__ffs(mask) - 1);
                        }
                    }
                    const int last_lane = 31 - __clz(fit);
                    const int ktot = __shfl_sync(kFullMask, kin, last_lane);
                    __syncwarp();
                    packed_expand<kUnroll, kReach>(sh, w, work, m, ktot, lane, far_min);
                    __syncwarp();  // the next group overwrites rank
                    j = last_lane + 1;
                    continue;
                }
            }
            batched_expand<kUnroll, kReach>(sh, w, work, j, lane, far_min);
            ++j;
        }
        __syncwarp();  // the next chunk overwrites the entries
    }
    far_min = warp_min(far_min);
    if (lane == 0 && far_min != kInfBits) {
        atomicMin(min_bits, far_min);
    }
}

// ------------------------------------------------------------------------------------------ shortest-path DAG
// low[v] = high word of the smallest d[v][s] of the tile (final distances): a lower bound of every one of them.
__device__ __forceinline__ void dag_low(const unsigned long long* dist, uint32_t* low, int64_t n, int nsrc, int lane, int gw, int gwarps) {
    constexpr int kRows = 4;
    for (int64_t v0 = gw; v0 < n; v0 += static_cast<int64_t>(kRows) * gwarps) {
        uint32_t hi[kRows];
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
            const int64_t v = v0 + static_cast<int64_t>(i) * gwarps;
            hi[i] = v < n && lane < nsrc ? static_cast<uint32_t>(__ldcg(&dist[v * kTile + lane]) >> 32) : 0xFFFFFFFFu;
        }
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
            const int64_t v = v0 + static_cast<int64_t>(i) * gwarps;
            const uint32_t least = __reduce_min_sync(kFullMask, hi[i]);
            if (v < n && lane == 0) {
                low[v] = least;
            }
        }
    }
}

// Calls visit(u, e) in every lane in `active` for each DAG in-arc u -> v of its source (fl(d[u][s] + len) == d[v][s], e =
// the arc's forward index), in reverse-CSR order. An arc can be on some source's DAG only if fl(low[u] + len) is at most
// the largest d[v][s] (fl is monotone), so 128 in-arcs at a time are filtered with one 4-byte read each, and only the
// rows of the rest (16 % at out-degree 100, 30-50 % at 40) are read, four rows in flight.
template <typename Visit>
__device__ __forceinline__ void scan_in_arcs(const TileSmem& sh, WarpScratch& w, const uint32_t* low, int v, unsigned long long dv, bool active,
                                             int lane, const Visit& visit) {
    const uint32_t dv_max = __reduce_max_sync(kFullMask, active ? static_cast<uint32_t>(dv >> 32) : 0u);
    const int64_t beg = __ldg(&sh.args.rrow_ptr[v]);
    const int deg = static_cast<int>(__ldg(&sh.args.rrow_ptr[v + 1]) - beg);
    const Arc* const arcs = sh.args.rarcs + beg;
    const unsigned long long* const dist_s = sh.args.dist + lane;
    for (int a0 = 0; a0 < deg; a0 += kArcBlock) {
        int kept = 0;
        {
            Arc arc[kArcBlock / 32];
            uint32_t lo[kArcBlock / 32];
#pragma unroll
            for (int u = 0; u < kArcBlock / 32; ++u) {
                const int i = a0 + u * 32 + lane;
                arc[u] = ldg_arc_once(&arcs[i < deg ? i : deg - 1]);
            }
#pragma unroll
            for (int u = 0; u < kArcBlock / 32; ++u) {
                lo[u] = __ldcg(&low[arc[u].col]);
            }
#pragma unroll
            for (int u = 0; u < kArcBlock / 32; ++u) {
                const int i = a0 + u * 32 + lane;
                const double least = __dadd_rn(__hiloint2double(static_cast<int>(lo[u]), 0), arc[u].len);
                const bool keep = i < deg && static_cast<uint32_t>(__double2hiint(least)) <= dv_max;
                const unsigned bal = __ballot_sync(kFullMask, keep);
                if (keep) {
                    w.kept[kept + __popc(bal & lanemask_lt())] = arc[u];
                }
                kept += __popc(bal);
            }
        }
        __syncwarp();
        constexpr int kRows = 4;
        for (int a = 0; a < kept; a += kRows) {
            unsigned long long du[kRows];
#pragma unroll
            for (int u = 0; u < kRows; ++u) {
                du[u] = __ldcg(&dist_s[static_cast<int64_t>(w.kept[a + u < kept ? a + u : a].col) * kTile]);
            }
#pragma unroll
            for (int u = 0; u < kRows; ++u) {
                const Arc arc = w.kept[a + u < kept ? a + u : a];
                if (a + u < kept && active && du[u] != kInfBits && on_dag(du[u], arc.len, dv)) {
                    visit(arc.col, static_cast<uint32_t>(arc.id));
                }
            }
        }
        __syncwarp();  // the next block of arcs overwrites kept
    }
}

// cnt[v][s] = DAG predecessors of (v, s), pred[v][s] = forward index of one of their arcs (the only one when cnt is 1),
// scnt[u][s] += 1 for each DAG arc u -> v, sigma = 0; warp per vertex, lane per source. keep[v][s] = that arc's
// source (kKeepArc: its forward index), for passes after pred's storage is reused. src_lane: this lane's source vertex (-1 without one).
template <bool kKeepArc>
__device__ __noinline__ void dag_count(const uint32_t* low, int src_lane, double* sigma, uint32_t* cnt, uint32_t* scnt, uint32_t* pred,
                                       uint32_t* keep, TileShared* ctl, int gw) {
    extern __shared__ __align__(16) unsigned long long smem[];
    TileSmem& sh = *reinterpret_cast<TileSmem*>(smem);
    const int lane = threadIdx.x & 31;
    WarpScratch& w = sh.warp[threadIdx.x >> 5];
    unsigned active_count = 0;
    unsigned arc_count = 0;
    for (int v = gw; v < sh.args.n; v += sh.args.group_warps) {
        const int64_t row = static_cast<int64_t>(v) * kTile + lane;
        const unsigned long long dv = __ldcg(&sh.args.dist[row]);
        const bool active = src_lane >= 0 && dv != kInfBits && v != src_lane;
        uint32_t c = 0;
        uint32_t first = 0;
        int from = 0;
        if (__ballot_sync(kFullMask, active) != 0u) {
            active_count += active ? 1u : 0u;
            scan_in_arcs(sh, w, low, v, dv, active, lane, [&](int u, uint32_t e) {
                first = c == 0 ? e : first;
                from = u;
                ++c;
                atomicAdd(&scnt[static_cast<int64_t>(u) * kTile + lane], 1u);
            });
        }
        sigma[row] = 0.0;
        cnt[row] = c;
        pred[row] = first;
        keep[row] = kKeepArc ? first : static_cast<uint32_t>(from);
        arc_count += c;
    }
    const unsigned pairs = __reduce_add_sync(kFullMask, active_count);
    const unsigned long long arcs = __reduce_add_sync(kFullMask, arc_count & 0xFFFFu) +
                                    (static_cast<unsigned long long>(__reduce_add_sync(kFullMask, arc_count >> 16)) << 16);
    if (lane == 0 && arcs != 0ull) {
        atomicAdd(&ctl->active_pairs, static_cast<unsigned long long>(pairs));
        atomicAdd(&ctl->dag_arcs, arcs);
    }
}

// Betweenness dependencies when every DAG of the tile is a tree (as many DAG arcs as reached non-source pairs, the rule
// for tie-free weights). Every path count is 1, so delta[v][s] is the number of descendants of v: an integer, exact in
// any order. acc[v][s] (zero before) gathers it from the leaves up in one atomic per pair: the low word sums
// 1 + delta of the children, the high word counts the children done, and whoever adds the last child goes on with v. So
// there are no lists, no levels and no barriers; the walks of a warp that go on wait in its scratch until 32 of them
// make a full step. parent and scnt are those of dag_count, s_src the tile's sources.
__device__ __noinline__ void dag_tree_walk(const uint32_t* cnt, const uint32_t* parent, const uint32_t* scnt, unsigned long long* acc,
                                           const int* s_src, int gw) {
    extern __shared__ __align__(16) unsigned long long smem[];
    TileSmem& sh = *reinterpret_cast<TileSmem*>(smem);
    const int lane = threadIdx.x & 31;
    uint2* const stack = reinterpret_cast<uint2*>(sh.warp[threadIdx.x >> 5].kept);  // (v << 5 | s, delta), 256 entries
    constexpr int kRows = 4;
    static_assert(sizeof(Arc) * kArcBlock / sizeof(uint2) >= 32 * (kRows + 1), "a round's pushes fit on top of a partial step");
    int waiting = 0;
    // one child of (up, s) is done with `size` descendants and itself; pushes (up, s) when it was the last
    const auto arrive = [&](bool on, uint32_t up, uint32_t s, uint32_t size) {
        bool go_on = false;
        uint32_t sum = 0;
        if (on) {
            const int64_t row = static_cast<int64_t>(up) * kTile + s;
            const uint32_t children = __ldcg(&scnt[row]);
            const unsigned long long old = atomicAdd(&acc[row], (1ull << 32) | (1ull + size));
            sum = static_cast<uint32_t>(old) + 1u + size;
            go_on = static_cast<uint32_t>(old >> 32) + 1u == children && static_cast<int>(up) != s_src[s];
        }
        const unsigned bal = __ballot_sync(kFullMask, go_on);
        if (go_on) {
            stack[waiting + __popc(bal & lanemask_lt())] = make_uint2(up << 5 | s, sum);
        }
        waiting += __popc(bal);
        __syncwarp();
    };
    const auto step = [&](int take) {
        waiting -= take;
        const uint2 e = stack[waiting + (lane < take ? lane : 0)];
        __syncwarp();
        const uint32_t s = e.x & 31u;
        const uint32_t up = lane < take ? __ldcg(&parent[static_cast<int64_t>(e.x >> 5) * kTile + s]) : 0u;
        arrive(lane < take, up, s, e.y);
    };
    for (int v0 = gw; v0 < sh.args.n; v0 += kRows * sh.args.group_warps) {
        bool leaf[kRows];
        uint32_t up[kRows];
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
            const int64_t v = v0 + static_cast<int64_t>(i) * sh.args.group_warps;
            const int64_t row = v * kTile + lane;
            leaf[i] = v < sh.args.n && __ldcg(&cnt[row]) != 0u && __ldcg(&scnt[row]) == 0u;
            up[i] = leaf[i] ? __ldcg(&parent[row]) : 0u;
        }
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
            arrive(leaf[i], up[i], static_cast<uint32_t>(lane), 0u);
        }
        while (waiting >= 32) {
            step(32);
        }
    }
    while (waiting > 0) {
        step(waiting < 32 ? waiting : 32);
    }
}

// Fills the successor lists: each DAG arc u -> v is appended to (u, s), as its target v (kTarget: betweenness needs
// nothing else) or as its forward-CSR index (the adjoint also needs the arc). A (v, s) with a single DAG predecessor
// takes it from pred[v][s]; only vertices with several for some source scan their in-arcs again.
template <bool kTarget>
__device__ __noinline__ void dag_fill(const int32_t* arc_src, const uint32_t* low, const uint32_t* cnt, const uint32_t* pred, const uint32_t* soff,
                                      uint32_t* sfill, uint32_t* succ, int gw) {
    extern __shared__ __align__(16) unsigned long long smem[];
    TileSmem& sh = *reinterpret_cast<TileSmem*>(smem);
    const int lane = threadIdx.x & 31;
    WarpScratch& w = sh.warp[threadIdx.x >> 5];
    constexpr int kRows = 2;  // single-predecessor lanes of two vertices, their reads side by side
    for (int v0 = gw; v0 < sh.args.n; v0 += kRows * sh.args.group_warps) {
        uint32_t c[kRows], e[kRows], pos[kRows], off[kRows];
        int64_t urow[kRows];
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
            const int64_t v = v0 + static_cast<int64_t>(i) * sh.args.group_warps;
            c[i] = v < sh.args.n ? __ldcg(&cnt[v * kTile + lane]) : 0u;
            e[i] = c[i] == 1u ? __ldcg(&pred[v * kTile + lane]) : 0u;
        }
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
            urow[i] = c[i] == 1u ? static_cast<int64_t>(__ldg(&arc_src[e[i]])) * kTile + lane : 0;
        }
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
            pos[i] = c[i] == 1u ? atomicAdd(&sfill[urow[i]], 1u) : 0u;
            off[i] = c[i] == 1u ? __ldcg(&soff[urow[i]]) : 0u;
        }
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
            if (c[i] == 1u) {
                const int64_t v = v0 + static_cast<int64_t>(i) * sh.args.group_warps;
                succ[off[i] + pos[i]] = kTarget ? static_cast<uint32_t>(v) : e[i];
            }
        }
#pragma unroll 1
        for (int i = 0; i < kRows; ++i) {
            const int v = v0 + i * sh.args.group_warps;
            const bool active = c[i] >= 2u;
            if (v < sh.args.n && __ballot_sync(kFullMask, active) != 0u) {
                const unsigned long long dv = __ldcg(&sh.args.dist[static_cast<int64_t>(v) * kTile + lane]);
                scan_in_arcs(sh, w, low, v, dv, active, lane, [&](int u, uint32_t fwd) {
                    const int64_t to = static_cast<int64_t>(u) * kTile + lane;
                    const uint32_t at = atomicAdd(&sfill[to], 1u);
                    succ[__ldcg(&soff[to]) + at] = kTarget ? static_cast<uint32_t>(v) : fwd;
                });
            }
        }
    }
}

// The next iteration's queue: the group's warps scan the pending masks `pend` (over the tile's reached vertices when
// it keeps a reach list: no other vertex can be pending) and append every vertex with a pending source to `q`, 32 at
// a time with one ballot and one atomic per warp.
template <bool kReach>
__device__ __forceinline__ void compact_queue(const uint32_t* pend, int32_t* q, int* qlen, int64_t span, const Reach& reach, int lane, int gw,
                                              int gwarps) {
    for (int64_t vb = static_cast<int64_t>(gw) * 32; vb < span; vb += static_cast<int64_t>(gwarps) * 32) {
        const int64_t i = vb + lane;
        const int64_t v = i < span ? (kReach ? static_cast<int64_t>(__ldcg(&reach.list[i])) : i) : 0;
        const uint32_t m = i < span ? __ldcg(&pend[v]) : 0u;
        const unsigned bal = __ballot_sync(kFullMask, m != 0u);
        if (bal != 0u) {
            int qb = 0;
            if (lane == 0) {
                qb = atomicAdd(qlen, __popc(bal));
            }
            qb = __shfl_sync(kFullMask, qb, 0);
            if (m != 0u) {
                q[qb + __popc(bal & lanemask_lt())] = static_cast<int32_t>(v);
            }
        }
    }
}

// The tile's first bounds, from kTile landmarks: d[x][s] <= d(s, l) + d(l, x) for every landmark l, so the smallest over l of
// max_s d(s, l) + d(l, x) bounds the row of x before any of its sources has reached it. Rounded sums over at most 2^31
// arcs differ from the exact path length by less than 2^-21 of it each way; the factor covers all of them. reach is
// shared memory. The caller separates this from the expansions by a group barrier.
__device__ __forceinline__ void landmark_bounds(const SsspParams& p, int64_t n, const int* s_src, int nsrc, unsigned long long* reach, uint8_t* bound,
                                                int bound_base, int64_t first, int64_t stride) {
    if (threadIdx.x < kTile) {
        reach[threadIdx.x] = 0ull;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kTile * nsrc; i += blockDim.x) {
        const int l = i & (kTile - 1);
        atomicMax(&reach[l], static_cast<unsigned long long>(__double_as_longlong(__ldg(&p.landmark_to[l * n + s_src[i / kTile]]))));
    }
    __syncthreads();
    for (int64_t x = first; x < n; x += stride) {
        double least = INFINITY;
#pragma unroll 8
        for (int l = 0; l < kTile; ++l) {
            least = fmin(least, __longlong_as_double(static_cast<long long>(reach[l])) + __ldg(&p.landmark_from[l * n + x]));
        }
        const int key = bound_key(static_cast<uint32_t>(__double2hiint(least * (1.0 + 0x1p-20))), bound_base);
        bound[x] = static_cast<uint8_t>(key < 0 ? 0 : (key < kNoBound ? key : kNoBound));
    }
}

// kMulti: the launch may put several CTAs on a tile (p.group_size > 1, cooperative launch); without it the group is
// the CTA itself, whose control block lives in shared memory. kReach: the tiles keep reach lists.
template <int kMode, int kUnroll, int kBlock, int kMinBlocks, bool kMulti = false, bool kReach = false>
__global__ void __launch_bounds__(kBlock, kMinBlocks) tile_kernel(const __grid_constant__ SsspParams p, const __grid_constant__ BrandesParams b) {
    extern __shared__ __align__(16) unsigned long long smem[];
    unsigned long long* s_acc_sum = smem;                                // kTile * kAccDigits
    unsigned long long* s_acc_inv = smem + kTile * kAccDigits;          // kTile * kAccDigits
    static_assert(kBlock <= 32 * kMaxWarps, "one warp scratch per warp");
    TileSmem& sh = *reinterpret_cast<TileSmem*>(smem);
    unsigned int* s_hist = reinterpret_cast<unsigned int*>(&sh + 1);
    unsigned long long* s_part = smem + 2 * kTile * kAccDigits;  // kBlock + 3 words
    TileShared& s = sh.ctl;
    __shared__ unsigned s_bar;
    __shared__ int s_src[kTile];
    __shared__ unsigned long long s_unreach[kTile];
    __shared__ unsigned long long s_arcs[kTile];
    __shared__ unsigned long long s_max[kTile];

    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;
    const int64_t n_slot = p.g.n;  // every slot holds the largest graph of the batch
    // The CTAs blockIdx.x / group_size share workspace slot `slot` and work on its tiles together. The group's
    // pointers and indices are recomputed from the launch parameters where they are used (fewer live registers).
    const int64_t slot = blockIdx.x / p.group_size;
    const auto grp = [&]() { return tile_group(p, &s); };
    const auto ctl = [&]() {
        return kMulti ? reinterpret_cast<TileShared*>(p.group_ws + (blockIdx.x / p.group_size) * p.group_stride) : &s;
    };
    // a group barrier whose last arrival applies `update` to the control block (a block barrier without kMulti)
    const auto sync = [&](auto&& update) {
        if constexpr (kMulti) {
            grp().sync(s, s_bar, update);
        } else {
            __syncthreads();
            if (threadIdx.x == 0) {
                update(s);
            }
            __syncthreads();
        }
    };
    const auto sync0 = [&]() { sync([](volatile TileShared&) {}); };
    // A CTA that gave up at a barrier (Group::sync) has no work and no complete state of the others': parents, counts and lists
    // may be words nobody wrote. The distance phase finds it halted; the DAG phase leaves the tile loop, and with it the kernel,
    // after the barrier at which it gave up. Always false for single-CTA tiles. (The epilogue's one barrier is followed by
    // sums at fixed places only, which a run that ends with NGX_TIMEOUT does not return; a way out there cost the distance
    // kernel 2 %: 0.376 and 0.384 ms on 300 vertices.)
    const auto left = [&]() { return kMulti && s.stop != 0; };
    // this thread's (warp's) index among the group's threads (warps), and their counts
#define NGX_GT (kMulti ? static_cast<int64_t>(blockIdx.x % p.group_size) * blockDim.x + threadIdx.x : static_cast<int64_t>(threadIdx.x))
#define NGX_GTHREADS (kMulti ? static_cast<int64_t>(p.group_size) * blockDim.x : static_cast<int64_t>(blockDim.x))
#define NGX_GW (kMulti ? static_cast<int>(blockIdx.x % p.group_size) * static_cast<int>(blockDim.x >> 5) + static_cast<int>(threadIdx.x >> 5) \
                       : static_cast<int>(threadIdx.x >> 5))
#define NGX_GWARPS (kMulti ? p.group_size * static_cast<int>(blockDim.x >> 5) : static_cast<int>(blockDim.x >> 5))
    if (lane == 0) {
        sh.work[warp] = WarpWork{ 0ull, 0ull };
    }

    unsigned long long* dist = p.ws_dist + slot * n_slot * kTile;
    uint32_t* pend0 = p.ws_pend + slot * 3 * n_slot;
    uint32_t* pend1 = pend0 + n_slot;
    uint32_t* far = pend1 + n_slot;
    int32_t* q0 = p.ws_queue + slot * 2 * n_slot;
    int32_t* q1 = q0 + n_slot;
    uint32_t* stamp = p.ws_stamp + slot * n_slot;
    uint8_t* const bound = reinterpret_cast<uint8_t*>(stamp);
    // reach lists: compiled in only for the kernels that keep them (kReach), so the others carry no extra registers
    const Reach reach{ kReach ? p.ws_reach + slot * n_slot : nullptr, kReach ? p.ws_touched + slot * n_slot : nullptr,
                       kReach ? &ctl()->touched_len : nullptr };
    const int64_t nt_slot = n_slot * kTile;
    double* sigma = nullptr;
    double* delta = nullptr;
    double* delta_g = nullptr;
    uint32_t* cnt = nullptr;
    uint32_t* lvl = nullptr;
    int32_t* list = nullptr;
    int32_t* loff = nullptr;
    uint32_t* scnt = nullptr;
    uint32_t* soff = nullptr;
    uint32_t* succ = nullptr;
    if constexpr (kMode != kModeApsp) {
        scnt = b.ws_scnt + slot * nt_slot;
        soff = b.ws_soff + slot * (nt_slot + 1);
        succ = b.ws_succ + slot * b.succ_capacity;
        sigma = b.ws_sigma + slot * nt_slot;
        delta = b.ws_delta + slot * nt_slot;
        delta_g = kMode == kModeGrad ? b.ws_delta_g + slot * nt_slot : nullptr;
        cnt = b.ws_cnt + slot * nt_slot;
        lvl = b.ws_lvl + slot * nt_slot;
        list = b.ws_list + slot * nt_slot;
        loff = b.ws_loff + slot * (n_slot + 2);
        for (int64_t i = NGX_GT; i < nt_slot; i += NGX_GTHREADS) {
            scnt[i] = 0u;
        }
    }

    for (int64_t i = NGX_GT; i < nt_slot; i += NGX_GTHREADS) {
        dist[i] = kInfBits;
    }
    for (int64_t i = NGX_GT; i < n_slot; i += NGX_GTHREADS) {
        pend0[i] = 0u;
        pend1[i] = 0u;
        far[i] = 0u;
        bound[i] = kNoBound;
        if (kReach) {
            reach.mask[i] = 0u;
        }
    }
    for (int i = tid; i < p.out.hist_bins; i += blockDim.x) {
        s_hist[i] = 0u;
    }
    if (tid == 0) {
        s_bar = 0u;
    }
    bool first_tile = true;

    for (;;) {
        // ---- the next work item, taken for the whole group; the slot's stamp counts on across tiles
        sync([&](volatile TileShared& c) {
            if (first_tile) {
                c.stamp = 1u;
            }
            c.tile = static_cast<long long>(atomicAdd(p.tile_counter, 1ull));
            c.stop = *reinterpret_cast<volatile int*>(p.error) != 0 ? 1 : 0;
            if (*p.abort_flag != 0) {
                atomicCAS(p.error, kDevOk, kDevAborted);
                c.stop = 1;
            }
            c.qlen[0] = 0;
            c.qlen[1] = 0;
            c.cur = 0;
            c.bucket_len = 0;
            c.iterations = 0;
            c.min_bits = kInfBits;
            c.min_left = kInfBits;
            c.active_pairs = 0;
            c.dag_arcs = 0;
            c.grab = 0;
            c.touched_len = 0;
            if (c.tile < p.num_tiles) {
                const WorkItem it = p.items != nullptr ? p.items[c.tile] : WorkItem{ 0, static_cast<int32_t>(c.tile) };
                c.theta = p.graphs[it.graph].delta;
            }
        });
        first_tile = false;
        if (s.stop != 0 || s.tile >= p.num_tiles) {
            break;
        }
        // ---- the work item: tile `item.tile` of graph `item.graph`
        const WorkItem item = p.items != nullptr ? p.items[s.tile] : WorkItem{ 0, static_cast<int32_t>(s.tile) };
        const GraphDesc gd = p.graphs[item.graph];
        const int64_t n = gd.n;
        const int64_t nt = n * kTile;
        const DeviceCsr g{ gd.n, gd.m, p.g.row_ptr + gd.row_off, p.g.arcs };
        const DeviceCsr rg{ gd.n, gd.m, b.rg.row_ptr + gd.row_off, b.rg.arcs };
        unsigned long long* const cnts = p.out.counters + static_cast<int64_t>(item.graph) * kCounterCount;
        unsigned long long* const acc_sum_g = p.out.acc_sum + static_cast<int64_t>(item.graph) * 2 * kAccDigits;
        unsigned long long* const acc_inv_g = acc_sum_g + kAccDigits;
        unsigned long long* const hist_g = p.out.hist != nullptr ? p.out.hist + static_cast<int64_t>(item.graph) * p.out.hist_bins : nullptr;
        unsigned long long* const bc_g = b.bc != nullptr ? b.bc + 2 * gd.bc_off : nullptr;
        const int64_t tile_first = static_cast<int64_t>(item.tile) * kTile;
        const int64_t base = gd.src_off + tile_first;
        const int nsrc = static_cast<int>(gd.num_sources - tile_first < kTile ? gd.num_sources - tile_first : kTile);
        if (tid < kTile) {
            s_src[tid] = tid < nsrc ? p.sources[base + tid] : -1;
            s_unreach[tid] = 0ull;
            s_arcs[tid] = 0ull;
            s_max[tid] = 0ull;
        }
        if (tid == 0) {
            sh.args = ExpandArgs{ g.arcs, g.row_ptr, rg.arcs, rg.row_ptr, dist, pend0, q0, bound, &ctl()->grab, reach,
                                  static_cast<uint32_t>(n_slot), nsrc, static_cast<int>(static_cast<uint32_t>(__double2hiint(0.25 * gd.delta)) >> 15),
                                  NGX_GWARPS, static_cast<int>(n), gd.m < kFilterDegree * gd.n ? 1 : 0 };
        }
        __syncthreads();
        if (!kReach && p.landmark_from != nullptr) {
            landmark_bounds(p, n, s_src, nsrc, s_max, bound, sh.args.bound_base, NGX_GT, NGX_GTHREADS);
            __syncthreads();
            if (tid < kTile) {
                s_max[tid] = 0ull;
            }
        }
        if ((!kMulti || grp().rank == 0) && warp == 0) {
            const int v = s_src[lane];
            if (v >= 0) {
                dist[static_cast<int64_t>(v) * kTile + lane] = 0ull;
                // pend0 is all zero between tiles: the first lane of a source repeated in the tile queues it
                if (atomicOr(&pend0[v], 1u << lane) == 0u) {
                    q0[atomicAdd(&ctl()->qlen[0], 1)] = v;
                }
                if (kReach) {
                    reach.add(v, 1u << lane);
                }
            }
        }
        sync0();

        // ------------------------------------------------------------ delta-stepping over the tile
        long long t_phase = clock64();
        for (;;) {
            for (;;) {
                const int cur = s.cur;
                const int qlen = s.qlen[cur];
                if (qlen == 0) {
                    break;
                }
                uint32_t* pend_nxt = cur ? pend0 : pend1;
                int32_t* q_nxt = cur ? q0 : q1;
                expand_queue<kUnroll, kReach>(&ctl()->min_bits);
                sync([&](volatile TileShared& c) {
                    c.qlen[cur] = 0;
                    c.grab = 0;
                    c.iterations = c.iterations + 1;
                    if (c.iterations > p.max_iterations) {
                        atomicCAS(p.error, kDevOk, kDevTimeout);
                        c.stop = 1;
                    } else if ((c.iterations & (kAbortPoll - 1)) == 0 && *p.abort_flag != 0) {
                        atomicCAS(p.error, kDevOk, kDevAborted);
                        c.stop = 1;
                    }
                });
                if (s.stop != 0) {
                    break;
                }
                // the next iteration's queue, from its pending masks (reach list: touched_len is final here)
                compact_queue<kReach>(pend_nxt, q_nxt, &ctl()->qlen[cur ^ 1], kReach ? static_cast<int64_t>(s.touched_len) : n, reach, lane,
                                      NGX_GW, NGX_GWARPS);
                sync([&](volatile TileShared& c) { c.cur = cur ^ 1; });
            }
            if (s.stop != 0) {
                break;
            }
            // bucket step: no near work is left. Every far mark set since the last step offered its distance to min_bits, and
            // that step left the smallest distance it kept far there, so the next bound needs no pass of its own. (A mark
            // that has been superseded may make it too low: the step then moves nothing and leaves the true minimum.)
            if (s.min_bits == kInfBits) {
                break;  // nothing pending: the tile's distances are final
            }
            const double theta = next_theta(__longlong_as_double(static_cast<long long>(s.min_bits)), gd.delta);
            // one pass over the far marks (of the tile's reached vertices when it keeps a reach list: no other vertex has
            // any) moves the pairs below the new bound into the near queue of the next iteration
            const int64_t span = kReach ? static_cast<int64_t>(s.touched_len) : n;
            const int cur = s.cur;
            uint32_t* pend_cur = cur ? pend1 : pend0;
            int32_t* q_cur = cur ? q1 : q0;
            unsigned long long left = kInfBits;
            for (int64_t vb = static_cast<int64_t>(NGX_GW) * 32; vb < span; vb += static_cast<int64_t>(NGX_GWARPS) * 32) {
                const int64_t i = vb + lane;
                const int64_t v = i < span ? (kReach ? static_cast<int64_t>(__ldcg(&reach.list[i])) : i) : 0;
                const uint32_t fm = i < span ? __ldcg(&far[v]) : 0u;
                unsigned any = __ballot_sync(kFullMask, fm != 0u);
                uint32_t moved = 0u;  // this lane's vertex: sources that move
                while (any != 0u) {
                    // two marked vertices at a time, their rows read side by side
                    const int l0 = __ffs(any) - 1;
                    any &= any - 1u;
                    const int l1 = any != 0u ? __ffs(any) - 1 : l0;
                    any &= any - 1u;
                    const uint32_t f0 = __shfl_sync(kFullMask, fm, l0);
                    const uint32_t f1 = __shfl_sync(kFullMask, fm, l1);
                    const int64_t v0 = __shfl_sync(kFullMask, v, l0);
                    const int64_t v1 = __shfl_sync(kFullMask, v, l1);
                    const unsigned long long d0 = (f0 >> lane) & 1u ? __ldcg(&dist[v0 * kTile + lane]) : kInfBits;
                    const unsigned long long d1 = (f1 >> lane) & 1u ? __ldcg(&dist[v1 * kTile + lane]) : kInfBits;
                    const bool near0 = __longlong_as_double(static_cast<long long>(d0)) < theta;
                    const bool near1 = __longlong_as_double(static_cast<long long>(d1)) < theta;
                    left = !near0 && d0 < left ? d0 : left;
                    left = !near1 && d1 < left ? d1 : left;
                    const unsigned n0 = __ballot_sync(kFullMask, near0);
                    const unsigned n1 = __ballot_sync(kFullMask, near1);
                    moved = lane == l0 ? n0 : (lane == l1 ? n1 : moved);
                }
                const unsigned bal = __ballot_sync(kFullMask, moved != 0u);
                if (bal != 0u) {
                    int qb = 0;
                    if (lane == 0) {
                        qb = atomicAdd(&ctl()->bucket_len, __popc(bal));
                    }
                    qb = __shfl_sync(kFullMask, qb, 0);
                    if (moved != 0u) {
                        far[v] = fm & ~moved;
                        pend_cur[v] = moved;
                        q_cur[qb + __popc(bal & lanemask_lt())] = static_cast<int32_t>(v);
                    }
                }
            }
            left = warp_min(left);
            if (lane == 0 && left != kInfBits) {
                atomicMin(&ctl()->min_left, left);
            }
            sync([&](volatile TileShared& c) {
                c.qlen[cur] = c.bucket_len;
                c.bucket_len = 0;
                c.theta = theta;
                c.min_bits = c.min_left;
                c.min_left = kInfBits;
            });
        }
        if (s.stop != 0) {
            break;
        }
        if (tid == 0) {
            const long long now = clock64();
            atomicAdd(&cnts[kCyclesSssp], static_cast<unsigned long long>(now - t_phase));
            t_phase = now;
        }
        bool tree = false;
        if constexpr (kMode != kModeApsp) {
            // ------------------------------------------------------------ shortest-path DAG: counts, sigma, delta
            // the level lists are built only after the successor lists: their storage holds pred[][] until then
            uint32_t* const pred = reinterpret_cast<uint32_t*>(list);
            uint32_t* const low = stamp;  // its words held the distance phase's bounds until here
            dag_low(dist, low, n, nsrc, lane, NGX_GW, NGX_GWARPS);
            sync0();
            if (left()) {
                break;
            }
            dag_count<kMode == kModeGrad>(low, lane < nsrc ? s_src[lane] : -1, sigma, cnt, scnt, pred, lvl, ctl(), NGX_GW);
            sync0();
            if (left()) {
                break;
            }
            // when every reached pair has exactly one DAG predecessor (as many DAG arcs as reached non-source pairs) the
            // DAGs are trees
            tree = s.dag_arcs == s.active_pairs && b.succ_capacity > 0;
            const bool tree_walk = kMode == kModeBrandes && tree;
          if (tree_walk) {
            if (tid == 0) {
                const long long now = clock64();
                atomicAdd(&cnts[kCyclesCount], static_cast<unsigned long long>(now - t_phase));
                t_phase = now;
            }
            dag_tree_walk(cnt, lvl, scnt, reinterpret_cast<unsigned long long*>(sigma), s_src, NGX_GW);
            sync0();
            if (left()) {
                break;
            }
            if (tid == 0) {
                if (!kMulti || grp().rank == 0) {
                    atomicAdd(&cnts[kDagEntries], s.active_pairs + static_cast<unsigned long long>(nsrc));
                }
                const long long now = clock64();
                atomicAdd(&cnts[kCyclesDelta], static_cast<unsigned long long>(now - t_phase));
                t_phase = now;
            }
          } else {
            const unsigned long long dag_arcs = group_exclusive_scan(grp(), s, s_bar, scnt, soff, nt, s_part);
            if (left()) {
                break;
            }
            const bool use_lists = dag_arcs <= static_cast<unsigned long long>(b.succ_capacity);
            for (int64_t i = NGX_GT; i < nt; i += NGX_GTHREADS) {
                scnt[i] = 0u;
            }
            sync0();
            if (left()) {
                break;
            }
            if (use_lists) {
                if (kMode == kModeBrandes || tree) {  // (targets only)
                    dag_fill<true>(b.arc_src, low, cnt, pred, soff, scnt, succ, NGX_GW);
                } else {
                    dag_fill<false>(b.arc_src, low, cnt, pred, soff, scnt, succ, NGX_GW);
                }
                sync0();
                if (left()) {
                    break;
                }
                dag_sort(soff, succ, nt, NGX_GT, NGX_GTHREADS);
            }
            if (!use_lists) {
                for (int64_t i = NGX_GT; i < n; i += NGX_GTHREADS) {
                    stamp[i] = 0u;
                }
                for (int64_t i = NGX_GT; i < nt; i += NGX_GTHREADS) {
                    lvl[i] = kNoLevel;
                    delta[i] = 0.0;  // pairs that no level releases keep it (see below)
                    if constexpr (kMode == kModeGrad) {
                        delta_g[i] = 0.0;
                    }
                }
            }
            sync([&](volatile TileShared& c) {
                if (!use_lists) {
                    c.stamp = c.stamp + 1u;
                }
                c.level = 0u;
                c.lvl_start = 0;
                c.lvl_len = 0;
                c.next_len = 0;
                loff[0] = 0;
            });
            if (left()) {
                break;
            }
            if (tid == 0) {
                const long long now = clock64();
                atomicAdd(&cnts[kCyclesCount], static_cast<unsigned long long>(now - t_phase));
                t_phase = now;
                if (!use_lists && (!kMulti || grp().rank == 0)) {
                    atomicAdd(&cnts[kDagScanTiles], 1ull);
                }
            }
            // the sources form level 0
            if ((!kMulti || grp().rank == 0) && warp == 0) {
                const int v = s_src[lane];
                if (v >= 0) {
                    const int64_t row = static_cast<int64_t>(v) * kTile + lane;
                    sigma[row] = 1.0;
                    if (!use_lists) {
                        lvl[row] = 0u;
                    }
                    if (use_lists) {
                        list[atomicAdd(&ctl()->lvl_len, 1)] = static_cast<int32_t>((static_cast<uint32_t>(v) << 5) | static_cast<uint32_t>(lane));
                    } else if (atomicExch(&stamp[v], s.stamp) != s.stamp) {
                        list[atomicAdd(&ctl()->lvl_len, 1)] = v;
                    }
                }
            }
            sync0();
            if (left()) {
                break;
            }
          if (use_lists) {
            // --- sigma and delta over the successor lists. In a tree every sigma is 1 and every child is released by its
            // only parent, so the sigma levels need neither sums nor counts.
            for (;;) {
                const int start = s.lvl_start;
                const int len = s.lvl_len;
                if (len == 0) {
                    break;
                }
                const unsigned level = s.level;
                // (tree tiles of betweenness took the walk above)
                if (kMode == kModeGrad && tree) {
                    dag_tree_level(list + start, len, sigma, soff, succ, list + start + len, &ctl()->next_len, lane, NGX_GW, NGX_GWARPS);
                } else {
                    dag_sigma_level<kMode == kModeBrandes>(g, list + start, len, sigma, cnt, soff, succ, list + start + len, &ctl()->next_len,
                                                           b.sigma_inexact, lane, NGX_GW, NGX_GWARPS);
                }
                sync([&](volatile TileShared& c) {
                    c.lvl_start = start + len;
                    c.lvl_len = c.next_len;
                    c.next_len = 0;
                    c.level = level + 1u;
                    loff[level + 1u] = start + len;
                });
                if (left()) {
                    break;
                }
            }
            if (left()) {
                break;
            }
            // Arcs that vanish against their distances (fl(d + len) == d) close cycles, whose pairs, and those behind them,
            // no level releases: they have no path count and their dependency is 0. No level writes it, so it is stored here;
            // a tile without such pairs (all listed) pays for one comparison.
            if (!tree && static_cast<unsigned long long>(s.lvl_start) < s.active_pairs + static_cast<unsigned long long>(nsrc)) {
                for (int64_t i = NGX_GT; i < nt; i += NGX_GTHREADS) {
                    if (__ldcg(&cnt[i]) != 0u) {
                        delta[i] = 0.0;
                        if constexpr (kMode == kModeGrad) {
                            delta_g[i] = 0.0;
                        }
                    }
                }
                sync0();
                if (left()) {
                    break;
                }
            }
            if (tid == 0) {
                const long long now = clock64();
                atomicAdd(&cnts[kCyclesSigma], static_cast<unsigned long long>(now - t_phase));
                t_phase = now;
            }
            const int levels = static_cast<int>(s.level);
            const int lowest = kMode == kModeGrad && !tree ? 0 : 1;  // the sources' own arcs get their terms from level 0, in a tree in the epilogue
            for (int level = levels - 1; level >= lowest; --level) {
                const int start = __ldcg(&loff[level]);
                const int end = __ldcg(&loff[level + 1]);
                if (kMode == kModeGrad && tree) {
                    dag_delta_level<kModeGrad, true>(g, list + start, end - start, dist, sigma, delta, delta_g, soff, succ, b.grad_cpl, b.grad_eff,
                                                 reinterpret_cast<double*>(s_acc_sum), lane, warp, NGX_GW, NGX_GWARPS);
                } else {
                    dag_delta_level<kMode, false>(g, list + start, end - start, dist, sigma, delta, delta_g, soff, succ, b.grad_cpl, b.grad_eff,
                                                  reinterpret_cast<double*>(s_acc_sum), lane, warp, NGX_GW, NGX_GWARPS);
                }
                sync0();
                if (left()) {
                    break;
                }
            }
            if (left()) {
                break;
            }
            if (tid == 0) {
                if ((!kMulti || grp().rank == 0)) {
                    atomicAdd(&cnts[kDagLevels], static_cast<unsigned long long>(levels));
                    atomicAdd(&cnts[kDagEntries], static_cast<unsigned long long>(__ldcg(&loff[levels])));
                }
                const long long now = clock64();
                atomicAdd(&cnts[kCyclesDelta], static_cast<unsigned long long>(now - t_phase));
                t_phase = now;
            }
          } else {
            // --- too many DAG arcs for the lists (many ties): the arc-scanning passes, one vertex per warp
            for (;;) {
                const int start = s.lvl_start;
                const int len = s.lvl_len;
                if (len == 0) {
                    break;
                }
                const unsigned level = s.level;
                const unsigned level_stamp = s.stamp + 1u;
                if (b.sigma_pull != 0) {
                    for (int i = NGX_GW; i < len; i += NGX_GWARPS) {
                        brandes_sigma_vertex<true, 2>(g, rg, __ldcg(&list[start + i]), level, nsrc, lane, dist, sigma, cnt, lvl, stamp, level_stamp,
                                                      list + start + len, &ctl()->next_len, b.sigma_inexact);
                    }
                } else {
                    for (int i = NGX_GW; i < len; i += NGX_GWARPS) {
                        brandes_sigma_vertex<false, 2>(g, rg, __ldcg(&list[start + i]), level, nsrc, lane, dist, sigma, cnt, lvl, stamp, level_stamp,
                                                       list + start + len, &ctl()->next_len, b.sigma_inexact);
                    }
                }
                sync([&](volatile TileShared& c) {
                    c.lvl_start = start + len;
                    c.lvl_len = c.next_len;
                    c.next_len = 0;
                    c.stamp = level_stamp;
                    c.level = level + 1u;
                    loff[level + 1u] = start + len;
                });
                if (left()) {
                    break;
                }
            }
            if (left()) {
                break;
            }
            if (tid == 0) {
                const long long now = clock64();
                atomicAdd(&cnts[kCyclesSigma], static_cast<unsigned long long>(now - t_phase));
                t_phase = now;
            }
            // s.level is one past the last non-empty level; loff[s.level] is the end of the lists
            const int levels = static_cast<int>(s.level);
            const int lowest = kMode == kModeGrad ? 0 : 1;
            for (int level = levels - 1; level >= lowest; --level) {
                const int start = __ldcg(&loff[level]);
                const int end = __ldcg(&loff[level + 1]);
                for (int i = start + NGX_GW; i < end; i += NGX_GWARPS) {
                    brandes_delta_vertex<kMode, 2>(g, __ldcg(&list[i]), static_cast<unsigned>(level), nsrc, lane, dist, sigma, delta, delta_g, lvl,
                                                   b.grad_cpl, b.grad_eff);
                }
                sync0();
                if (left()) {
                    break;
                }
            }
            if (left()) {
                break;
            }
            if (tid == 0) {
                if ((!kMulti || grp().rank == 0)) {
                    atomicAdd(&cnts[kDagLevels], static_cast<unsigned long long>(levels));
                    atomicAdd(&cnts[kDagEntries], static_cast<unsigned long long>(__ldcg(&loff[levels])));
                }
                const long long now = clock64();
                atomicAdd(&cnts[kCyclesDelta], static_cast<unsigned long long>(now - t_phase));
                t_phase = now;
            }
          }
          }
        }

        // ------------------------------------------------------------ epilogue: fused APSP summaries, reset
        // the passes before borrowed the accumulators, which must start at zero (each ended with a barrier)
        for (int i = tid; i < 2 * kTile * kAccDigits; i += blockDim.x) {
            smem[i] = 0ull;
        }
        __syncthreads();
        const int my_src = s_src[lane];
        const bool valid = lane < nsrc;
        unsigned long long unreach = 0, arcs = 0, mx = 0, overflow = 0;
        // APSP with a reach list visits the reached vertices only: every other vertex is unreached by every source and
        // its state was never touched; the DAG passes have written every vertex's rows, and distance rows need every
        // vertex, so those visit all of them
        const bool by_list = kReach && kMode == kModeApsp && p.out.rows == nullptr;
        const int64_t span = by_list ? static_cast<int64_t>(s.touched_len) : n;
        if (by_list && valid && (!kMulti || grp().rank == 0) && warp == 0) {
            unreach = static_cast<unsigned long long>(n - span);
        }
        for (int64_t i = NGX_GW; i < span; i += NGX_GWARPS) {
            const int64_t v = by_list ? static_cast<int64_t>(__ldcg(&reach.list[i])) : i;
            if (lane == 0) {
                if constexpr (kMode == kModeApsp) {
                    bound[v] = kNoBound;
                } else {
                    stamp[v] = 0xFFFFFFFFu;  // whole words: stamps reach past the graph's n bounds, into a larger graph's
                }
                if (kReach) {
                    reach.mask[v] = 0u;
                }
            }
            unsigned long long* slot_ptr = &dist[v * kTile + lane];
            const unsigned long long bits = __ldcg(slot_ptr);
            *slot_ptr = kInfBits;
            if constexpr (kMode != kModeApsp) {
                const int64_t row = v * kTile + lane;
                if constexpr (kMode == kModeBrandes) {
                    // BrandesVariant.h:156: every settled vertex but the source gains its dependency
                    const bool gains = valid && v != my_src && bits != kInfBits;
                    if (tree) {
                        // integers (descendant counts): exact in double and in fixed point alike
                        const unsigned long long dep = gains ? __ldcg(reinterpret_cast<unsigned long long*>(&sigma[row])) & 0xFFFFFFFFull : 0ull;
                        const unsigned long long sum = __reduce_add_sync(kFullMask, static_cast<unsigned>(dep & 0xFFFFull)) +
                                                       (static_cast<unsigned long long>(__reduce_add_sync(kFullMask, static_cast<unsigned>(dep >> 16))) << 16);
                        if (lane == 0 && sum != 0ull) {
                            atomicAdd(&bc_g[2 * v + 1], sum);
                        }
                    } else {
                        const double dep = gains ? __ldcg(&delta[row]) : 0.0;
                        // summed over the tile's sources in fixed point, exactly: betweenness does not depend on how
                        // the sources are grouped into tiles
                        unsigned long long lo, hi;
                        fixed_parts(dep, lo, hi);
                        fixed_warp_sum(lo, hi);
                        if (lane == 0 && (lo | hi) != 0ull) {
                            fixed_add_parts(&bc_g[2 * v], lo, hi);
                        }
                    }
                } else if (tree) {
                    const bool on = valid && v != my_src && bits != kInfBits;
                    const double inv = on ? 1.0 / __longlong_as_double(static_cast<long long>(bits)) : 0.0;
                    add_arc_terms(g.arcs, on, on ? __ldcg(&lvl[row]) : 0u, on ? 1.0 + __ldcg(&delta[row]) : 0.0,
                                  on ? inv * inv + __ldcg(&delta_g[row]) : 0.0, lane, b.grad_cpl, b.grad_eff);
                }
                scnt[row] = 0u;
            }
            if (!valid) {
                continue;
            }
            const double d = __longlong_as_double(static_cast<long long>(bits));
            if (p.out.rows != nullptr) {
                p.out.rows[(base + lane) * n + v] = d;
            }
            if (bits == kInfBits) {
                ++unreach;
                continue;
            }
            arcs += static_cast<unsigned long long>(__ldg(&g.row_ptr[v + 1]) - __ldg(&g.row_ptr[v]));
            mx = bits > mx ? bits : mx;
            acc_add_shared(&s_acc_sum[lane * kAccDigits], d);
            if (bits != 0ull) {
                acc_add_shared(&s_acc_inv[lane * kAccDigits], __ddiv_rn(1.0, d));
            }
            if (p.out.hist_bins > 0 && v != my_src) {
                if (d >= p.out.hist_max) {
                    ++overflow;
                } else {
                    unsigned long long bin = static_cast<unsigned long long>(__ddiv_rn(d, p.out.hist_width));
                    if (bin >= static_cast<unsigned long long>(p.out.hist_bins)) {
                        bin = static_cast<unsigned long long>(p.out.hist_bins) - 1ull;
                    }
                    atomicAdd(&s_hist[bin], 1u);
                }
            }
        }
        if (valid) {
            atomicAdd(&s_unreach[lane], unreach);
            atomicAdd(&s_arcs[lane], arcs);
            atomicMax(&s_max[lane], mx);
        }
        if (overflow != 0) {
            atomicAdd(&cnts[kHistOverflow], overflow);
        }
        __syncthreads();
        if (kMulti && p.group_size > 1) {
            // the group's CTAs add their per-source sums into the group's (exact integer adds), and the first CTA
            // finishes the tile's per-source outputs from them
            unsigned long long* const g_acc = p.group_ws + slot * p.group_stride + kCtlWords + 1 + p.group_size;  // kGroupAccWords
            for (int i = tid; i < 2 * kTile * kAccDigits; i += blockDim.x) {
                if (smem[i] != 0ull) {
                    atomicAdd(&g_acc[i], smem[i]);
                }
            }
            if (tid < kTile) {
                atomicAdd(&g_acc[2 * kTile * kAccDigits + tid], s_unreach[tid]);
                atomicAdd(&g_acc[2 * kTile * kAccDigits + kTile + tid], s_arcs[tid]);
                atomicMax(&g_acc[2 * kTile * kAccDigits + 2 * kTile + tid], s_max[tid]);
            }
            sync0();
            if ((!kMulti || grp().rank == 0)) {
                for (int i = tid; i < 2 * kTile * kAccDigits; i += blockDim.x) {
                    smem[i] = __ldcg(&g_acc[i]);
                    g_acc[i] = 0ull;
                }
                if (tid < kTile) {
                    unsigned long long* const per = g_acc + 2 * kTile * kAccDigits;
                    s_unreach[tid] = __ldcg(&per[tid]);
                    s_arcs[tid] = __ldcg(&per[kTile + tid]);
                    s_max[tid] = __ldcg(&per[2 * kTile + tid]);
                    per[tid] = 0ull;
                    per[kTile + tid] = 0ull;
                    per[2 * kTile + tid] = 0ull;
                }
            }
            __syncthreads();
        }
        if ((!kMulti || grp().rank == 0)) {
            if (tid < nsrc) {
                unsigned long long* a_sum = &s_acc_sum[tid * kAccDigits];
                unsigned long long* a_inv = &s_acc_inv[tid * kAccDigits];
                acc_normalize(a_sum);
                acc_normalize(a_inv);
                const int64_t pos = base + tid;
                if (p.out.src_sum != nullptr) p.out.src_sum[pos] = acc_round_normalized(a_sum);
                if (p.out.src_inv != nullptr) p.out.src_inv[pos] = acc_round_normalized(a_inv);
                if (p.out.src_max != nullptr) p.out.src_max[pos] = __longlong_as_double(static_cast<long long>(s_max[tid]));
                if (p.out.src_unreach != nullptr) p.out.src_unreach[pos] = s_unreach[tid];
                if (p.out.src_arcs != nullptr) p.out.src_arcs[pos] = s_arcs[tid];
                const unsigned long long reached = static_cast<unsigned long long>(n) - s_unreach[tid];
                atomicAdd(&cnts[kUnreachable], s_unreach[tid]);
                atomicAdd(&cnts[kReachedPairs], reached - 1ull);
                atomicAdd(&cnts[kTraversedArcs], s_arcs[tid]);
                atomicMax(&cnts[kDiameterBits], s_max[tid]);
            }
            __syncthreads();
            for (int i = tid; i < kAccDigits; i += blockDim.x) {
                unsigned long long t_sum = 0, t_inv = 0;
                for (int k = 0; k < nsrc; ++k) {
                    t_sum += s_acc_sum[k * kAccDigits + i];
                    t_inv += s_acc_inv[k * kAccDigits + i];
                }
                if (t_sum != 0) atomicAdd(&acc_sum_g[i], t_sum);
                if (t_inv != 0) atomicAdd(&acc_inv_g[i], t_inv);
            }
            if (tid == 0) {
                atomicAdd(&cnts[kIterations], s.iterations);
            }
        }
        for (int i = tid; i < p.out.hist_bins; i += blockDim.x) {
            if (s_hist[i] != 0u) {
                atomicAdd(&hist_g[i], static_cast<unsigned long long>(s_hist[i]));
                s_hist[i] = 0u;
            }
        }
        __syncthreads();
        if (tid == 0) {
            atomicAdd(&cnts[kCyclesEpilogue], static_cast<unsigned long long>(clock64() - t_phase));
        }
    }
    if (lane == 0 && sh.work[warp].expansions != 0) {
        // whole-launch totals, kept in the first graph's counters
        atomicAdd(&p.out.counters[kExpansions], sh.work[warp].expansions);
        atomicAdd(&p.out.counters[kLaneExpansions], sh.work[warp].lane_expansions);
    }
#undef NGX_GT
#undef NGX_GTHREADS
#undef NGX_GW
#undef NGX_GWARPS
}

// ------------------------------------------------------------------------------------------ plain form
__device__ __forceinline__ void plain_push(bool push, int x, int lane, int32_t* q, int* qlen) {
    const unsigned mask = __ballot_sync(kFullMask, push);
    if (mask == 0u) {
        return;
    }
    int base = 0;
    if (lane == __ffs(mask) - 1) {
        base = atomicAdd(qlen, __popc(mask));
    }
    base = __shfl_sync(kFullMask, base, __ffs(mask) - 1);
    if (push) {
        q[base + __popc(mask & lanemask_lt())] = x;
    }
}

// Brandes for the one source of a plain tile (BrandesVariant.h:79-159), by one CTA with warp-per-vertex passes over
// the final distances: DAG predecessor counts from each vertex's in-arcs; Kahn levels over the out-arcs (the last
// predecessor of x to be done appends x to the next level); sigma of each new level pulled over its in-arcs (integer
// sums, exact in FP64 below 2^53); dependencies pulled over the out-arcs, level by level from the last,
// delta[u] = sum over DAG arcs u -> x of sigma[u] * ((1 + delta[x]) / sigma[x]), each lane's terms in arc order and
// the lanes combined by a fixed shuffle tree; every vertex but the source adds delta[u] to its 128-bit fixed-point
// betweenness. The arrays are per CTA: sigma, delta, cnt, list (n each) and loff (n + 2).
__device__ __forceinline__ double warp_sum_fixed_order(double x) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        x += __shfl_xor_sync(kFullMask, x, off);
    }
    return x;
}

__device__ void plain_brandes(const DeviceCsr& g, const DeviceCsr& rg, int64_t n, int src, const unsigned long long* dist, double* sigma,
                              double* delta, uint32_t* cnt, int32_t* list, int32_t* loff, unsigned long long* bc, TileShared& s, int tid,
                              int lane, int warp, int nwarps) {
    // DAG predecessors of every reached vertex
    for (int64_t v = warp; v < n; v += nwarps) {
        const unsigned long long dv = __ldcg(&dist[v]);
        unsigned c = 0;
        if (dv != kInfBits && v != src) {
            const int64_t beg = __ldg(&rg.row_ptr[v]);
            const int64_t end = __ldg(&rg.row_ptr[v + 1]);
            for (int64_t e = beg + lane; e < end; e += 32) {
                const Arc a = ldg_arc(&rg.arcs[e]);
                c += on_dag(__ldcg(&dist[a.col]), a.len, dv) ? 1u : 0u;
            }
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            c += __shfl_xor_sync(kFullMask, c, off);
        }
        if (lane == 0) {
            cnt[v] = c;
            sigma[v] = v == src ? 1.0 : 0.0;
            delta[v] = 0.0;
        }
    }
    if (tid == 0) {
        list[0] = src;
        loff[0] = 0;
        loff[1] = 1;
        s.level = 0u;
        s.next_len = 0;
    }
    __syncthreads();
    // Kahn levels, and sigma of each new level
    for (;;) {
        const unsigned level = s.level;
        const int start = loff[level];
        const int len = loff[level + 1] - start;
        if (len == 0) {
            break;
        }
        for (int i = warp; i < len; i += nwarps) {
            const int u = list[start + i];
            const unsigned long long du = __ldcg(&dist[u]);
            const int64_t beg = __ldg(&g.row_ptr[u]);
            const int64_t end = __ldg(&g.row_ptr[u + 1]);
            for (int64_t e0 = beg; e0 < end; e0 += 32) {
                const int64_t e = e0 + lane;
                bool ready = false;
                int x = 0;
                if (e < end) {
                    const Arc a = ldg_arc(&g.arcs[e]);
                    x = a.col;
                    ready = on_dag(du, a.len, __ldcg(&dist[x])) && atomicSub(&cnt[x], 1u) == 1u;
                }
                plain_push(ready, x, lane, list + start + len, &s.next_len);
            }
        }
        __syncthreads();
        const int next = start + len;
        const int next_len = s.next_len;
        for (int i = warp; i < next_len; i += nwarps) {
            const int x = __ldcg(&list[next + i]);
            const unsigned long long dx = __ldcg(&dist[x]);
            const int64_t beg = __ldg(&rg.row_ptr[x]);
            const int64_t end = __ldg(&rg.row_ptr[x + 1]);
            double acc = 0.0;
            for (int64_t e = beg + lane; e < end; e += 32) {
                const Arc a = ldg_arc(&rg.arcs[e]);
                if (on_dag(__ldcg(&dist[a.col]), a.len, dx)) {
                    acc += __ldcg(&sigma[a.col]);
                }
            }
            acc = warp_sum_fixed_order(acc);
            if (lane == 0) {
                sigma[x] = acc;
            }
        }
        __syncthreads();
        if (tid == 0) {
            loff[level + 2] = next + next_len;
            s.level = level + 1u;
            s.next_len = 0;
        }
        __syncthreads();
    }
    // dependencies, from the last level to the source's
    for (int level = static_cast<int>(s.level) - 1; level >= 0; --level) {
        const int start = loff[level];
        const int len = loff[level + 1] - start;
        for (int i = warp; i < len; i += nwarps) {
            const int u = __ldcg(&list[start + i]);
            const unsigned long long du = __ldcg(&dist[u]);
            const double su = __ldcg(&sigma[u]);
            const int64_t beg = __ldg(&g.row_ptr[u]);
            const int64_t end = __ldg(&g.row_ptr[u + 1]);
            double acc = 0.0;
            for (int64_t e = beg + lane; e < end; e += 32) {
                const Arc a = ldg_arc(&g.arcs[e]);
                if (on_dag(du, a.len, __ldcg(&dist[a.col]))) {
                    acc += su * ((1.0 + __ldcg(&delta[a.col])) / __ldcg(&sigma[a.col]));
                }
            }
            acc = warp_sum_fixed_order(acc);
            if (lane == 0) {
                delta[u] = acc;
                if (u != src && acc != 0.0) {
                    unsigned long long lo, hi;
                    fixed_parts(acc, lo, hi);
                    fixed_add_parts(&bc[2 * static_cast<int64_t>(u)], lo, hi);
                }
            }
        }
        __syncthreads();
    }
}

template <bool kBrandes>
__global__ void __launch_bounds__(512, 2) sssp_plain_kernel(const SsspParams p, const BrandesParams b) {
    extern __shared__ __align__(16) unsigned long long smem[];
    const int nwarps_max = 16;
    unsigned long long* s_acc_sum = smem;                             // nwarps_max * kAccDigits (one per warp)
    unsigned long long* s_acc_inv = smem + nwarps_max * kAccDigits;
    unsigned int* s_hist = reinterpret_cast<unsigned int*>(smem + 2 * nwarps_max * kAccDigits);
    __shared__ TileShared s;
    __shared__ unsigned long long s_unreach, s_arcs, s_max;

    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;
    const int nwarps = blockDim.x >> 5;
    const int64_t n = p.g.n;
    const int64_t slot = blockIdx.x;
    unsigned long long expansions = 0;

    unsigned long long* dist = p.ws_dist + slot * n;
    uint32_t* pend0 = p.ws_pend + slot * 3 * n;
    uint32_t* pend1 = pend0 + n;
    uint32_t* far = pend1 + n;
    int32_t* q0 = p.ws_queue + slot * 2 * n;
    int32_t* q1 = q0 + n;
    uint32_t* stamp = p.ws_stamp + slot * n;

    for (int64_t i = tid; i < n; i += blockDim.x) {
        dist[i] = kInfBits;
        pend0[i] = 0u;
        pend1[i] = 0u;
        far[i] = 0u;
        stamp[i] = 0u;
    }
    for (int i = tid; i < 2 * nwarps_max * kAccDigits; i += blockDim.x) {
        smem[i] = 0ull;
    }
    for (int i = tid; i < p.out.hist_bins; i += blockDim.x) {
        s_hist[i] = 0u;
    }
    if (tid == 0) {
        s.stamp = 1u;
    }
    __syncthreads();

    for (;;) {
        if (tid == 0) {
            s.tile = static_cast<long long>(atomicAdd(p.tile_counter, 1ull));
            s.stop = (*reinterpret_cast<volatile int*>(p.error) != 0) ? 1 : 0;
            s.qlen[0] = 0;
            s.qlen[1] = 0;
            s.cur = 0;
            s.theta = p.delta;
            s.iterations = 0;
            s.overflow = 0;
            s_unreach = 0;
            s_arcs = 0;
            s_max = 0;
        }
        __syncthreads();
        if (s.stop != 0 || s.tile >= p.num_tiles) {
            break;
        }
        const int64_t pos = s.tile;
        const int src = p.sources[pos];
        if (tid == 0) {
            dist[src] = 0ull;
            pend0[src] = 1u;
            stamp[src] = s.stamp;
            q0[0] = src;
            s.qlen[0] = 1;
        }
        __syncthreads();

        for (;;) {
            for (;;) {
                const int cur = s.cur;
                const int qlen = s.qlen[cur];
                if (qlen == 0) {
                    break;
                }
                uint32_t* pend_cur = cur ? pend1 : pend0;
                uint32_t* pend_nxt = cur ? pend0 : pend1;
                const int32_t* q_cur = cur ? q1 : q0;
                int32_t* q_nxt = cur ? q0 : q1;
                const unsigned next_stamp = s.stamp + 1u;
                const double theta = s.theta;
                for (int i = warp; i < qlen; i += nwarps) {
                    const int v = __ldcg(&q_cur[i]);
                    if (__ldcg(&pend_cur[v]) == 0u) {
                        continue;
                    }
                    const double dv = __longlong_as_double(static_cast<long long>(__ldcg(&dist[v])));
                    expansions += 1;
                    if (lane == 0) {
                        pend_cur[v] = 0u;
                        far[v] = 0u;  // a near value supersedes any far mark; no far mark can be set while d[v] < theta
                    }
                    const int64_t beg = __ldg(&p.g.row_ptr[v]);
                    const int64_t end = __ldg(&p.g.row_ptr[v + 1]);
                    for (int64_t e0 = beg; e0 < end; e0 += 32) {
                        const int64_t e = e0 + lane;
                        bool push = false;
                        int x = 0;
                        if (e < end) {
                            const Arc a = ldg_arc(&p.g.arcs[e]);
                            x = a.col;
                            const double nd = __dadd_rn(dv, a.len);
                            const unsigned long long nb = static_cast<unsigned long long>(__double_as_longlong(nd));
                            if (nb < __ldcg(&dist[x])) {
                                const unsigned long long old = atomicMin(&dist[x], nb);
                                if (nb < old) {
                                    if (nd < theta) {
                                        pend_nxt[x] = 1u;
                                        push = atomicExch(&stamp[x], next_stamp) != next_stamp;
                                    } else {
                                        far[x] = 1u;
                                    }
                                }
                            }
                        }
                        plain_push(push, x, lane, q_nxt, &s.qlen[cur ^ 1]);
                    }
                }
                __syncthreads();
                if (tid == 0) {
                    s.qlen[cur] = 0;
                    s.cur = cur ^ 1;
                    s.stamp = next_stamp;
                    s.iterations += 1;
                    if (s.iterations > p.max_iterations) {
                        atomicCAS(p.error, kDevOk, kDevTimeout);
                        s.stop = 1;
                    } else if (*p.abort_flag != 0) {
                        atomicCAS(p.error, kDevOk, kDevAborted);
                        s.stop = 1;
                    }
                }
                __syncthreads();
                if (s.stop != 0) {
                    break;
                }
            }
            if (s.stop != 0) {
                break;
            }
            if (tid == 0) {
                s.min_bits = kInfBits;
            }
            __syncthreads();
            unsigned long long local_min = kInfBits;
            for (int64_t v = tid; v < n; v += blockDim.x) {
                if (__ldcg(&far[v]) != 0u) {
                    const unsigned long long d = __ldcg(&dist[v]);
                    local_min = d < local_min ? d : local_min;
                }
            }
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) {
                const unsigned long long o = __shfl_xor_sync(kFullMask, local_min, off);
                local_min = o < local_min ? o : local_min;
            }
            if (lane == 0 && local_min != kInfBits) {
                atomicMin(&s.min_bits, local_min);
            }
            __syncthreads();
            if (s.min_bits == kInfBits) {
                break;
            }
            const double theta = next_theta(__longlong_as_double(static_cast<long long>(s.min_bits)), p.delta);
            const int cur = s.cur;
            uint32_t* pend_cur = cur ? pend1 : pend0;
            int32_t* q_cur = cur ? q1 : q0;
            for (int64_t vb = 0; vb < n; vb += blockDim.x) {
                const int64_t v = vb + tid;
                bool push = false;
                if (v < n && __ldcg(&far[v]) != 0u) {
                    if (__longlong_as_double(static_cast<long long>(__ldcg(&dist[v]))) < theta) {
                        far[v] = 0u;
                        pend_cur[v] = 1u;
                        push = true;
                    }
                }
                plain_push(push, static_cast<int>(v), lane, q_cur, &s.qlen[cur]);
            }
            __syncthreads();
            if (tid == 0) {
                s.theta = theta;
            }
            __syncthreads();
        }
        if (s.stop != 0) {
            break;
        }
        if constexpr (kBrandes) {
            plain_brandes(p.g, b.rg, n, src, dist, b.ws_sigma + slot * n, b.ws_delta + slot * n, b.ws_cnt + slot * n, b.ws_list + slot * n,
                          b.ws_loff + slot * (n + 2), b.bc, s, tid, lane, warp, nwarps);
        }

        // epilogue: one accumulator pair per warp, combined exactly
        unsigned long long* a_sum = &s_acc_sum[warp * kAccDigits];
        unsigned long long* a_inv = &s_acc_inv[warp * kAccDigits];
        unsigned long long unreach = 0, arcs = 0, mx = 0, overflow = 0;
        for (int64_t v = tid; v < n; v += blockDim.x) {
            const unsigned long long bits = __ldcg(&dist[v]);
            dist[v] = kInfBits;
            const double d = __longlong_as_double(static_cast<long long>(bits));
            if (p.out.rows != nullptr) {
                p.out.rows[pos * n + v] = d;
            }
            if (bits == kInfBits) {
                ++unreach;
                continue;
            }
            arcs += static_cast<unsigned long long>(__ldg(&p.g.row_ptr[v + 1]) - __ldg(&p.g.row_ptr[v]));
            mx = bits > mx ? bits : mx;
            acc_add_shared(a_sum, d);
            if (bits != 0ull) {
                acc_add_shared(a_inv, __ddiv_rn(1.0, d));
            }
            if (p.out.hist_bins > 0 && v != src) {
                if (d >= p.out.hist_max) {
                    ++overflow;
                } else {
                    unsigned long long bin = static_cast<unsigned long long>(__ddiv_rn(d, p.out.hist_width));
                    if (bin >= static_cast<unsigned long long>(p.out.hist_bins)) {
                        bin = static_cast<unsigned long long>(p.out.hist_bins) - 1ull;
                    }
                    atomicAdd(&s_hist[bin], 1u);
                }
            }
        }
        atomicAdd(&s_unreach, unreach);
        atomicAdd(&s_arcs, arcs);
        atomicMax(&s_max, mx);
        if (overflow != 0) {
            atomicAdd(&s.overflow, overflow);
        }
        __syncthreads();
        // fold the per-warp accumulators into warp 0's, digit-wise (each digit < 2^33 * adds, far below 2^64)
        for (int i = tid; i < kAccDigits; i += blockDim.x) {
            for (int w = 1; w < nwarps; ++w) {
                s_acc_sum[i] += s_acc_sum[w * kAccDigits + i];
                s_acc_inv[i] += s_acc_inv[w * kAccDigits + i];
                s_acc_sum[w * kAccDigits + i] = 0ull;
                s_acc_inv[w * kAccDigits + i] = 0ull;
            }
        }
        __syncthreads();
        if (tid == 0) {
            acc_normalize(s_acc_sum);
            acc_normalize(s_acc_inv);
            if (p.out.src_sum != nullptr) p.out.src_sum[pos] = acc_round_normalized(s_acc_sum);
            if (p.out.src_inv != nullptr) p.out.src_inv[pos] = acc_round_normalized(s_acc_inv);
            if (p.out.src_max != nullptr) p.out.src_max[pos] = __longlong_as_double(static_cast<long long>(s_max));
            if (p.out.src_unreach != nullptr) p.out.src_unreach[pos] = s_unreach;
            if (p.out.src_arcs != nullptr) p.out.src_arcs[pos] = s_arcs;
            atomicAdd(&p.out.counters[kUnreachable], s_unreach);
            atomicAdd(&p.out.counters[kReachedPairs], static_cast<unsigned long long>(n) - s_unreach - 1ull);
            atomicAdd(&p.out.counters[kTraversedArcs], s_arcs);
            atomicMax(&p.out.counters[kDiameterBits], s_max);
            if (s.overflow != 0) atomicAdd(&p.out.counters[kHistOverflow], s.overflow);
            atomicAdd(&p.out.counters[kIterations], s.iterations);
        }
        __syncthreads();
        for (int i = tid; i < kAccDigits; i += blockDim.x) {
            if (s_acc_sum[i] != 0) atomicAdd(&p.out.acc_sum[i], s_acc_sum[i]);
            if (s_acc_inv[i] != 0) atomicAdd(&p.out.acc_inv[i], s_acc_inv[i]);
        }
        for (int i = tid; i < p.out.hist_bins; i += blockDim.x) {
            if (s_hist[i] != 0u) {
                atomicAdd(&p.out.hist[i], static_cast<unsigned long long>(s_hist[i]));
                s_hist[i] = 0u;
            }
        }
        __syncthreads();
        for (int i = tid; i < kAccDigits; i += blockDim.x) {
            s_acc_sum[i] = 0ull;
            s_acc_inv[i] = 0ull;
        }
        __syncthreads();
    }
    if (lane == 0 && expansions != 0) {
        atomicAdd(&p.out.counters[kExpansions], expansions);
        atomicAdd(&p.out.counters[kLaneExpansions], expansions);
    }
}

}  // namespace ngx
