// Host side of the tile runs: source tiling, workspace sizing, launch, result reduction.
//
// Replaces AllPairsShortestPath::compute_apsp_impl's per-source loop (source/metrics/paths/AllPairsShortestPath.h:110-163)
// and compute_apsp_impl_delta_stepping (:197-247) with one persistent launch over all source tiles, of one graph or of
// a batch of graphs.

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <utility>
#include <vector>

#include "ngx_common.cuh"
#include "ngx_graph.h"
#include "ngx_run.h"
#include "sssp_kernels.cuh"

namespace ngx {

namespace {
#ifndef NGX_BATCHED_UNROLL
#define NGX_BATCHED_UNROLL 4  // (arc, source) pairs in flight per lane in the distance phase
#endif
constexpr int kBatchedUnroll = NGX_BATCHED_UNROLL;
constexpr int kPlainWarpsMax = 16;
constexpr int kBatchedDefaultBlock = 512;
constexpr int kMaxGroupSize = 512;  // CTAs sharing one tile at most (above any SM count x resident CTAs per SM used here)

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }
}  // namespace

int prepare_sources(const ngx_graph* g, const ngx_apsp_opts* opts, std::vector<int32_t>& sources) {
    if (opts->sources == nullptr) {
        sources.resize(static_cast<size_t>(g->n));
        for (int64_t i = 0; i < g->n; ++i) {
            sources[static_cast<size_t>(i)] = static_cast<int32_t>(i);
        }
        return NGX_OK;
    }
    if (opts->num_sources < 0) {
        return fail(NGX_INVALID_ARGUMENT, "num_sources is negative");
    }
    sources.resize(static_cast<size_t>(opts->num_sources));
    for (int64_t i = 0; i < opts->num_sources; ++i) {
        const int64_t s = opts->sources[i];
        if (s < 0 || s >= g->n) {
            return fail(NGX_INVALID_ARGUMENT, "source " + std::to_string(s) + " is out of range");
        }
        sources[static_cast<size_t>(i)] = static_cast<int32_t>(s);
    }
    return NGX_OK;
}

double degree_delta_scale(int64_t n, int64_t m) {
    const double degree = n > 0 ? static_cast<double>(m) / static_cast<double>(n) : 1.0;
    const double scale = 2.0 / std::sqrt(degree > 1.0 ? degree : 1.0);
    return scale < 0.125 ? 0.125 : (scale > 2.0 ? 2.0 : scale);
}

double default_delta_scale(const GraphPart& part) {
    const double spread = part.mean_len_regular * part.mean_len_inverse;  // the same for both metrics
    const bool wide = part.m_stored < 28 * part.n || spread < 2.0;
    return (wide ? 2.0 : 1.0) * degree_delta_scale(part.n, part.m_stored);
}

double pick_delta(double mean_len, double requested, double scale) {
    if (requested > 0.0 && std::isfinite(requested)) {
        return requested;
    }
    const double base = mean_len > 0.0 && std::isfinite(mean_len) ? mean_len : 1.0;
    return base * (scale > 0.0 ? scale : 1.0);
}

int check_opts(const ngx_graph* g, const ngx_apsp_opts* opts) {
    if (g == nullptr || opts == nullptr) {
        return fail(NGX_INVALID_ARGUMENT, "graph or opts is NULL");
    }
    if (opts->metric != NGX_METRIC_REGULAR && opts->metric != NGX_METRIC_INVERSE) {
        return fail(NGX_INVALID_ARGUMENT, "unknown metric");
    }
    if (opts->mode != NGX_MODE_BATCHED && opts->mode != NGX_MODE_PLAIN) {
        return fail(NGX_INVALID_ARGUMENT, "unknown mode");
    }
    if (opts->hist_bins < 0 || opts->hist_bins > kMaxHistBins) {
        return fail(NGX_INVALID_ARGUMENT, "hist_bins must be in [0, " + std::to_string(kMaxHistBins) + "]");
    }
    if (opts->tile_ctas < 0 || opts->tile_ctas > kMaxGroupSize) {
        return fail(NGX_INVALID_ARGUMENT, "tile_ctas must be in [0, " + std::to_string(kMaxGroupSize) + "]");
    }
    if (opts->block_threads != 0 && (opts->block_threads < 64 || opts->block_threads > 512 || opts->block_threads % 32 != 0)) {
        return fail(NGX_INVALID_ARGUMENT, "block_threads must be a multiple of 32 in [64, 512]");
    }
    return NGX_OK;
}

int alloc_outputs(ngx_graph* g, int64_t num_graphs, int64_t num_sources, int64_t hist_bins, bool want_rows, RunOutputs& o, bool persistent) {
    const size_t s = static_cast<size_t>(num_sources);
    const size_t gcount = static_cast<size_t>(num_graphs);
    size_t off = 0;
    const auto take = [&](size_t bytes) {
        const size_t at = off;
        off += align256(bytes);
        return at;
    };
    const size_t a_acc = take(gcount * 2 * kAccDigits * 8);
    const size_t a_cnt = take(gcount * kCounterCount * 8);
    const size_t a_err = take(8);
    const size_t a_tile = take(8);
    const size_t a_hist = take(gcount * static_cast<size_t>(std::max<int64_t>(hist_bins, 1)) * 8);
    const size_t zeroed = off;  // everything above starts at zero
    const size_t a_graphs = take(gcount * sizeof(GraphDesc));
    const size_t a_sources = take(std::max<size_t>(s, 1) * 4);
    const size_t a_f64 = take(3 * s * 8);
    const size_t a_u64 = take(2 * s * 8);
    const size_t a_rows = want_rows ? take(s * static_cast<size_t>(g->n) * 8) : 0;
    if (persistent) {
        if (off > g->persistent_bytes) {
            NGX_CUDA_TRY(cudaStreamSynchronize(g->stream));
            cudaFree(g->d_persistent);
            g->d_persistent = nullptr;
            g->persistent_bytes = 0;
            NGX_CUDA_TRY(cudaMalloc(&g->d_persistent, off));
            g->persistent_bytes = off;
        }
        o.block = g->d_persistent;
        o.owned = false;
    } else {
        if (const int rc = grow_buffer(g, &g->d_call_out, &g->call_out_bytes, off); rc != NGX_OK) {
            return rc;
        }
        o.block = g->d_call_out;
        o.owned = false;
    }
    o.bytes = off;
    o.zeroed_bytes = zeroed;
    char* b = static_cast<char*>(o.block);
    o.acc = reinterpret_cast<unsigned long long*>(b + a_acc);
    o.counters = reinterpret_cast<unsigned long long*>(b + a_cnt);
    o.error = reinterpret_cast<int*>(b + a_err);
    o.tile_counter = reinterpret_cast<unsigned long long*>(b + a_tile);
    o.hist = reinterpret_cast<unsigned long long*>(b + a_hist);
    o.graphs = reinterpret_cast<GraphDesc*>(b + a_graphs);
    o.sources = reinterpret_cast<int32_t*>(b + a_sources);
    o.src_f64 = reinterpret_cast<double*>(b + a_f64);
    o.src_u64 = reinterpret_cast<unsigned long long*>(b + a_u64);
    o.rows = want_rows ? reinterpret_cast<double*>(b + a_rows) : nullptr;
    o.num_graphs = num_graphs;
    o.num_sources = num_sources;
    return NGX_OK;
}

void free_outputs(ngx_graph* g, RunOutputs& o) {
    if (o.block != nullptr && o.owned) {
        cudaFreeAsync(o.block, g->stream);
    }
    o.block = nullptr;
}

int device_error_status(int code) {
    switch (code) {
    case kDevOk: return NGX_OK;
    case kDevTimeout: return fail(NGX_TIMEOUT, "a source tile exceeded max_iterations delta-stepping phases");
    case kDevAborted: return fail(NGX_ABORTED, "run aborted by ngx_graph_request_abort");
    default: return fail(NGX_CUDA_ERROR, "unknown device error code " + std::to_string(code));
    }
}

// The instantiation for a block size; 256 threads with ctas_per_sm >= 4 selects the 4-CTA (64-register) build. Tile
// groups of several CTAs (multi) and reach lists (reach) are built for the default shape only (512 threads x 2 CTAs per
// SM); nullptr for other combinations.
template <int kMode>
const void* tile_kernel_for_block(int block, int ctas_per_sm, bool reach, bool multi) {
    if (reach || multi) {
        if (block != kBatchedDefaultBlock) {
            return nullptr;
        }
        if (multi && reach) return reinterpret_cast<const void*>(&tile_kernel<kMode, kBatchedUnroll, 512, 2, true, true>);
        if (multi) return reinterpret_cast<const void*>(&tile_kernel<kMode, kBatchedUnroll, 512, 2, true, false>);
        return reinterpret_cast<const void*>(&tile_kernel<kMode, kBatchedUnroll, 512, 2, false, true>);
    }
    switch (block) {
    case 256:
        return ctas_per_sm >= 4 ? reinterpret_cast<const void*>(&tile_kernel<kMode, kBatchedUnroll, 256, 4>)
                                : reinterpret_cast<const void*>(&tile_kernel<kMode, kBatchedUnroll, 256, 3>);
    case 384: return reinterpret_cast<const void*>(&tile_kernel<kMode, kBatchedUnroll, 384, 2>);
    case 512: return reinterpret_cast<const void*>(&tile_kernel<kMode, kBatchedUnroll, 512, 2>);
    default: return nullptr;
    }
}

// CTAs per tile group: the caller's choice, else the size with the least modelled time.
//  * Work per phase. A tile's phases (near iterations, bucket steps, DAG passes) end with a barrier of its group, and the
//    entries of a phase grow with n while their number grows slowly, so larger graphs feed more CTAs. Measured kernel
//    times over many tiles (Brandes unless noted, CTAs per tile: ms): n = 1e4, degree 40: 3: 79, 7: 62, 10-14: 58, 24: 66;
//    n = 2e4, degree 6: 1: 267, 4: 217, 14: 197; n = 3e4, degree 40: 7: 183, 21: 152, 42: 156; n = 5e4 (gradient): 9: 73,
//    18-37: 67, 49: 69; n = 1e5, degree 100 (APSP): 37-49: 176, 74: 179, 148: 234; n = 3e5, degree 40: 4: 337, 37-74: 264,
//    100: 325; n = 1e6: 18: 309, 74: 279; batches of mixed graphs, mean n 800: 1: 19.3, 2: 16.4, 8: 29; 3200: 1: 138, 6: 127,
//    11: 156; 13,400: 1: 637, 11: 522, 24: 581. Those follow (1 + b + l) / g for a tile's time: b = 250 g / n (1 + g / 100)
//    for the barriers, more by the cube root of the degree below 40 (less work per phase), and l = 0.2 for each doubling of
//    the distance-phase bytes in flight (280 per vertex and slot) beyond 65 MB, where the rate of random sector reads from
//    L2 starts to fall (microbenchmark: half at 100 MB).
//  * Waves. The tiles run in waves of resident / g, counted whole when there are few: 63 tiles of n = 2000 (gradient) want
//    4 CTAs and one wave (2.2 ms; 3: 2.6, 5 and two waves: 3.1, 9: 2.7). Few tiles take the CTAs that would idle, up to
//    0.6 sqrt(n) (n = 2e4, 2 tiles: 37: 1.22, 74: 0.94, 148: 1.05 ms; n = 300, 10 tiles: 4: 0.49, 8-29: 0.45). At least
//    four tiles stay in flight.
//  * Sparse graphs (mean out-degree below 4) have long shortest paths, so many phases with few entries each: one CTA per
//    tile while there are two tiles for every resident CTA, more in proportion when there are fewer. Right at n = 2e4 and
//    degree 2 (626 tiles, APSP: 1: 65, 2: 66, 4: 71, 16: 109 ms) and with few tiles (n = 1e5, degree 3, 94 tiles, the rule's 6:
//    46, 8-16: 47, 1: 86); larger graphs and degrees near 4 with many tiles would be faster with 4 to 16: n = 2e4, degree 3.9: 1:
//    85, 4: 76; n = 6e4, degree 2: 1: 561, 4: 552; n = 1e5, degree 3, 500 tiles: 1: 320, the rule's 323, 8: 251; n = 3e5, degree
//    3.9, 313 tiles: the rule's 715, 16: 465 (four tiles in L2, the rule before this one: 112, 1391, 601 and 878 ms).
//  * Memory: when the device affords fewer workspace slots than that, each slot gets enough CTAs to use every SM.
int choose_group_size(int requested, int64_t resident, int64_t num_tiles, int64_t affordable_slots, double typical_n, double mean_degree) {
    if (requested > 0) {
        return static_cast<int>(std::min<int64_t>({ static_cast<int64_t>(requested), resident, static_cast<int64_t>(kMaxGroupSize) }));
    }
    const int64_t tiles = std::max<int64_t>(1, num_tiles);
    const double n = std::max(typical_n, 1.0);
    const double sparse = std::cbrt(std::max(1.0, 40.0 / std::max(mean_degree, 1.0)));
    int64_t most = std::min(std::max(resident / 4, resident / tiles), static_cast<int64_t>(0.6 * std::sqrt(n)));
    if (mean_degree < 4.0) {
        most = std::min(most, std::max<int64_t>(1, 2 * resident / tiles));
    }
    most = std::max<int64_t>(1, std::min({ most, resident, static_cast<int64_t>(kMaxGroupSize) }));
    int64_t group = 1;
    double least = INFINITY;
    for (int64_t g = 1; g <= most; ++g) {
        const int64_t slots = resident / g;
        const double waves = tiles > 8 * slots ? static_cast<double>(tiles) / static_cast<double>(slots)
                                               : static_cast<double>((tiles + slots - 1) / slots);
        const double size = static_cast<double>(g);
        const double in_flight = 280.0 * n * static_cast<double>(std::min(slots, tiles));
        const double barriers = 250.0 * sparse * size / n * (1.0 + size / 100.0);
        const double time = waves * (1.0 + barriers + 0.2 * std::max(0.0, std::log2(in_flight / 65e6))) / size;
        if (time < least) {
            least = time;
            group = g;
        }
    }
    if (affordable_slots < std::min(resident, num_tiles)) {
        // enough CTAs per slot that the affordable slots hold every resident CTA (rounded up: the slot count then
        // follows from the group size, and no CTA is left without a slot)
        const int64_t slots = std::max<int64_t>(1, affordable_slots);
        group = std::max<int64_t>(group, (resident + slots - 1) / slots);
    }
    return static_cast<int>(std::max<int64_t>(1, std::min<int64_t>({ group, resident, static_cast<int64_t>(kMaxGroupSize) })));
}

// Launches the tile kernel: cooperative when several CTAs share a tile (they wait for one another at group barriers,
// so all of them must be resident at once).
cudaError_t launch_tile_kernel(const void* kernel, int64_t grid, int block, size_t smem, cudaStream_t stream, int group_size, void** args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(grid));
    cfg.blockDim = dim3(static_cast<unsigned>(block));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = group_size > 1 ? 1 : 0;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelExC(&cfg, kernel, args);
}

int launch_tiles(ngx_graph* g, const ngx_apsp_opts* opts, int tile_mode, const TileJob& job, int64_t hist_bins, double hist_max, RunOutputs& o,
                 DagOutputs* extra, float* kernel_ms, bool synchronous) {
    // the plain (one source per CTA) form runs APSP and Brandes; the adjoint is batched only
    const bool batched = opts->mode == NGX_MODE_BATCHED || tile_mode == kModeGrad;
    const int width = batched ? kTile : 1;
    const int64_t num_tiles = batched ? job.num_items : job.num_sources;
    const int block = opts->block_threads > 0 ? opts->block_threads : (batched ? kBatchedDefaultBlock : 512);
    const size_t fixed_smem = batched ? sizeof(TileSmem) : static_cast<size_t>(2) * kPlainWarpsMax * kAccDigits * 8;
    const size_t smem = fixed_smem + static_cast<size_t>(hist_bins) * 4;
    if (!batched && job.num_graphs != 1) {
        return fail(NGX_UNSUPPORTED, "the plain form runs one graph at a time");
    }
    if (num_tiles == 0) {
        return NGX_OK;
    }

    const void* kernel = tile_mode == kModeBrandes ? reinterpret_cast<const void*>(&sssp_plain_kernel<true>)
                                                   : reinterpret_cast<const void*>(&sssp_plain_kernel<false>);
    // reach lists (several strongly connected components) and tile groups run with the default block shape only
    const bool default_shape = block == kBatchedDefaultBlock && (opts->ctas_per_sm == 0 || opts->ctas_per_sm >= 2);
    if (batched && opts->tile_ctas > 1 && !default_shape) {
        return fail(NGX_INVALID_ARGUMENT, "tile groups (tile_ctas > 1) run with the default block shape (512 threads, 2 CTAs per SM)");
    }
    const bool track = batched && job.track_reach && default_shape;
    const auto pick = [&](bool reach, bool multi) -> const void* {
        return tile_mode == kModeBrandes ? tile_kernel_for_block<kModeBrandes>(block, opts->ctas_per_sm, reach, multi)
               : tile_mode == kModeGrad  ? tile_kernel_for_block<kModeGrad>(block, opts->ctas_per_sm, reach, multi)
                                         : tile_kernel_for_block<kModeApsp>(block, opts->ctas_per_sm, reach, multi);
    };
    if (batched) {
        kernel = pick(track, false);
        if (kernel == nullptr) {
            return fail(NGX_INVALID_ARGUMENT, "batched mode supports block_threads 256, 384 or 512");
        }
    }
    NGX_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    int per_sm = 0;
    NGX_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, smem));
    if (per_sm <= 0) {
        return fail(NGX_UNSUPPORTED, "kernel does not fit on an SM with this block size and histogram");
    }
    if (opts->ctas_per_sm > 0) {
        per_sm = std::min(per_sm, opts->ctas_per_sm);
    }
    const int64_t n = job.n_max;
    const int64_t resident = static_cast<int64_t>(g->sm_count) * per_sm;
    const size_t reach_bytes = track ? static_cast<size_t>(n) * 8 + 512 : 0;  // reach mask + reached list
    const size_t dag_bytes = tile_mode == kModeApsp ? 0 : batched ? brandes_slot_bytes(n, tile_mode == kModeGrad) : plain_brandes_slot_bytes(n);
    const size_t data_bytes = sssp_slot_bytes(n, width) + dag_bytes + reach_bytes;
    // the sizes the group rule goes by: the graph's, or the mean over a batch's graphs
    const double typical_n = job.num_graphs > 1 ? static_cast<double>(g->n_total) / static_cast<double>(job.num_graphs) : static_cast<double>(n);
    const double mean_degree = static_cast<double>(job.num_arcs) / std::max(1.0, typical_n * static_cast<double>(job.num_graphs));
    const auto group_bytes_of = [](int ctas) { return static_cast<size_t>(group_stride_words(ctas)) * 8; };
    const auto slots_of = [&](int ctas) { return std::min<int64_t>(num_tiles, resident / ctas); };
    // a workspace kept from an earlier run that holds what an unlimited device would get needs no look at the free memory
    // (a driver call of tens of microseconds)
    int group = batched && default_shape ? choose_group_size(opts->tile_ctas, resident, num_tiles, resident, typical_n, mean_degree) : 1;
    size_t slot_bytes = data_bytes + group_bytes_of(group);
    int64_t slots = slots_of(group);
    if (static_cast<size_t>(slots) * slot_bytes > std::min(g->workspace_bytes, workspace_cap(g))) {
        const size_t budget = workspace_budget(g);
        // the group size decides the group storage per slot, which the slot count must leave room for
        const int64_t affordable = static_cast<int64_t>(budget / (data_bytes + group_bytes_of(kMaxGroupSize)));
        group = batched && default_shape ? choose_group_size(opts->tile_ctas, resident, num_tiles, affordable, typical_n, mean_degree) : 1;
        slot_bytes = data_bytes + group_bytes_of(group);
        slots = std::min<int64_t>(slots_of(group), static_cast<int64_t>(budget / slot_bytes));
    }
    if (group > 1) {
        kernel = pick(track, true);  // the same shape and occupancy, built for groups
        NGX_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    }
    const size_t group_bytes = group_bytes_of(group);
    if (slots <= 0) {
        return fail(NGX_OUT_OF_MEMORY, "not enough device memory for one workspace slot (" + std::to_string(slot_bytes) + " bytes)");
    }
    if (const int rc = ensure_workspace(g, static_cast<size_t>(slots) * slot_bytes); rc != NGX_OK) {
        return rc;
    }
    char* ws = static_cast<char*>(g->d_workspace);
    // group storage first (256-byte aligned slots), then the slot arrays
    unsigned long long* group_ws = reinterpret_cast<unsigned long long*>(ws);
    ws += static_cast<size_t>(slots) * group_bytes;
    SsspParams p{};
    p.g = job.reverse ? g->reverse_csr() : g->csr(opts->metric);
    p.g.n = n;
    p.landmark_from = job.landmark_from;
    p.landmark_to = job.landmark_to;
    p.sources = o.sources;
    p.num_sources = job.num_sources;
    p.num_tiles = num_tiles;
    p.delta = job.plain_delta;
    p.graphs = o.graphs;
    p.items = job.d_items;
    p.max_iterations = opts->max_iterations > 0 ? opts->max_iterations : static_cast<unsigned long long>(4 * n + 64);
    p.tile_counter = o.tile_counter;
    p.error = o.error;
    p.abort_flag = g->d_abort;
    p.ws_dist = reinterpret_cast<unsigned long long*>(ws);
    ws += static_cast<size_t>(slots) * n * width * 8;
    p.ws_pend = reinterpret_cast<uint32_t*>(ws);
    ws += static_cast<size_t>(slots) * 3 * n * 4;
    p.ws_queue = reinterpret_cast<int32_t*>(ws);
    ws += static_cast<size_t>(slots) * 2 * n * 4;
    p.ws_stamp = reinterpret_cast<uint32_t*>(ws);
    ws += static_cast<size_t>(slots) * n * 4;
    p.group_size = group;
    p.group_stride = group_stride_words(group);
    p.group_ws = group_ws;
    if (track) {
        ws = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(ws) + 255) & ~uintptr_t(255));
        p.ws_reach = reinterpret_cast<uint32_t*>(ws);
        ws += static_cast<size_t>(slots) * n * 4;
        p.ws_touched = reinterpret_cast<int32_t*>(ws);
        ws += static_cast<size_t>(slots) * n * 4;
    }
    BrandesParams bp{};
    if (tile_mode == kModeBrandes && !batched) {
        // plain form: sigma, delta, predecessor counts and the level list per vertex, the level offsets
        ws = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(ws) + 255) & ~uintptr_t(255));
        bp.rg = g->reverse_csr();
        bp.ws_sigma = reinterpret_cast<double*>(ws);
        ws += static_cast<size_t>(slots) * n * 8;
        bp.ws_delta = reinterpret_cast<double*>(ws);
        ws += static_cast<size_t>(slots) * n * 8;
        bp.ws_cnt = reinterpret_cast<uint32_t*>(ws);
        ws += static_cast<size_t>(slots) * n * 4;
        bp.ws_list = reinterpret_cast<int32_t*>(ws);
        ws += static_cast<size_t>(slots) * n * 4;
        bp.ws_loff = reinterpret_cast<int32_t*>(ws);
        if (extra != nullptr) {
            bp.bc = extra->bc;
        }
    } else if (tile_mode != kModeApsp) {
        const size_t nt = static_cast<size_t>(n) * kTile;
        ws = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(ws) + 255) & ~uintptr_t(255));
        bp.rg = g->reverse_csr();
        bp.arc_src = g->d_arc_src;
        bp.ws_sigma = reinterpret_cast<double*>(ws);
        ws += static_cast<size_t>(slots) * nt * 8;
        bp.ws_delta = reinterpret_cast<double*>(ws);
        ws += static_cast<size_t>(slots) * nt * 8;
        if (tile_mode == kModeGrad) {
            bp.ws_delta_g = reinterpret_cast<double*>(ws);
            ws += static_cast<size_t>(slots) * nt * 8;
        }
        bp.ws_cnt = reinterpret_cast<uint32_t*>(ws);
        ws += static_cast<size_t>(slots) * nt * 4;
        bp.ws_lvl = reinterpret_cast<uint32_t*>(ws);
        ws += static_cast<size_t>(slots) * nt * 4;
        bp.ws_list = reinterpret_cast<int32_t*>(ws);
        ws += static_cast<size_t>(slots) * nt * 4;
        bp.ws_loff = reinterpret_cast<int32_t*>(ws);
        ws += static_cast<size_t>(slots) * static_cast<size_t>(n + 2) * 4;
        bp.ws_scnt = reinterpret_cast<uint32_t*>(ws);
        ws += static_cast<size_t>(slots) * nt * 4;
        bp.ws_soff = reinterpret_cast<uint32_t*>(ws);
        ws += static_cast<size_t>(slots) * (nt + 1) * 4;
        // list entries pack (vertex << 5 | source) into 32 bits; larger graphs use the arc-scanning passes
        bp.succ_capacity = n < (int64_t(1) << 26) ? static_cast<int64_t>(nt) * kSuccPerPair : 0;
        bp.ws_succ = reinterpret_cast<uint32_t*>(ws);
        if (extra != nullptr) {
            bp.bc = extra->bc;
            bp.grad_cpl = extra->grad_cpl;
            bp.grad_eff = extra->grad_eff;
            bp.sigma_inexact = extra->sigma_inexact;
            bp.sigma_pull = extra->sigma_pull;
        }
    }
    p.out.acc_sum = o.acc;
    p.out.acc_inv = o.acc + kAccDigits;
    p.out.counters = o.counters;
    p.out.hist = hist_bins > 0 ? o.hist : nullptr;
    p.out.hist_bins = static_cast<int>(hist_bins);
    p.out.hist_max = hist_max;
    p.out.hist_width = hist_bins > 0 ? hist_max / static_cast<double>(hist_bins) : 0.0;
    p.out.src_sum = o.src_f64;
    p.out.src_max = o.src_f64 + job.num_sources;
    p.out.src_inv = o.src_f64 + 2 * job.num_sources;
    p.out.src_unreach = o.src_u64;
    p.out.src_arcs = o.src_u64 + job.num_sources;
    p.out.rows = job.rows != nullptr ? job.rows : o.rows;

    if (synchronous) {
        if (g->run_start == nullptr) {
            NGX_CUDA_TRY(cudaEventCreate(&g->run_start));
        }
        if (g->run_stop == nullptr) {
            NGX_CUDA_TRY(cudaEventCreate(&g->run_stop));
        }
        cudaEventRecord(g->run_start, g->stream);
    }
    cudaError_t err = cudaSuccess;
    if (batched) {
        void* args[] = { &p, &bp };
        err = cudaMemsetAsync(group_ws, 0, static_cast<size_t>(slots) * group_bytes, g->stream);
        if (err == cudaSuccess) {
            err = launch_tile_kernel(kernel, slots * group, block, smem, g->stream, group, args);
        }
    } else {
        if (tile_mode == kModeBrandes) {
            sssp_plain_kernel<true><<<static_cast<unsigned>(slots), block, smem, g->stream>>>(p, bp);
        } else {
            sssp_plain_kernel<false><<<static_cast<unsigned>(slots), block, smem, g->stream>>>(p, bp);
        }
        err = cudaGetLastError();
    }
    if (!synchronous) {
        return err == cudaSuccess ? NGX_OK : cuda_fail(err, "tile kernel launch");
    }
    cudaEventRecord(g->run_stop, g->stream);
    int code = 0;
    if (err == cudaSuccess) {
        err = cudaMemcpyAsync(&code, o.error, sizeof(int), cudaMemcpyDeviceToHost, g->stream);
    }
    const cudaError_t done = cudaStreamSynchronize(g->stream);
    err = err == cudaSuccess ? done : err;
    float ms = 0.0f;
    if (err == cudaSuccess) {
        err = cudaEventElapsedTime(&ms, g->run_start, g->run_stop);
    }
    if (err != cudaSuccess) {
        return cuda_fail(err, "tile kernel");
    }
    if (kernel_ms != nullptr) {
        *kernel_ms += ms;
    }
    return device_error_status(code);
}

// Launches the batched APSP tile kernel on the graph's stream with its workspace carved from `ws` (`ws_bytes` bytes,
// 256-byte aligned) instead of the handle's workspace: nothing is allocated. Per-source outputs are written only where
// `o` has them. Returns after the launch; the caller synchronizes.
int launch_apsp_in_workspace(ngx_graph* g, const ngx_apsp_opts* opts, const TileJob& job, int64_t hist_bins, double hist_max, RunOutputs& o, void* ws,
                             size_t ws_bytes) {
    const int block = opts->block_threads > 0 ? opts->block_threads : kBatchedDefaultBlock;
    const void* kernel = tile_kernel_for_block<kModeApsp>(block, opts->ctas_per_sm, false, false);
    if (kernel == nullptr) {
        return fail(NGX_INVALID_ARGUMENT, "batched mode supports block_threads 256, 384 or 512");
    }
    if (job.num_items == 0) {
        return NGX_OK;
    }
    const size_t smem = sizeof(TileSmem) + static_cast<size_t>(hist_bins) * 4;
    NGX_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    int per_sm = 0;
    NGX_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, smem));
    if (per_sm <= 0) {
        return fail(NGX_UNSUPPORTED, "kernel does not fit on an SM with this block size and histogram");
    }
    if (opts->ctas_per_sm > 0) {
        per_sm = std::min(per_sm, opts->ctas_per_sm);
    }
    const int64_t n = job.n_max;
    const size_t group_bytes = static_cast<size_t>(group_stride_words(1)) * 8;  // one CTA per tile
    const size_t slot_bytes = sssp_slot_bytes(n, kTile) + group_bytes;
    int64_t slots = std::min<int64_t>(job.num_items, static_cast<int64_t>(g->sm_count) * per_sm);
    slots = std::min<int64_t>(slots, static_cast<int64_t>(ws_bytes / slot_bytes));
    if (slots <= 0) {
        return fail(NGX_OUT_OF_MEMORY, "the workspace holds no slot of " + std::to_string(slot_bytes) + " bytes");
    }
    char* w = static_cast<char*>(ws);
    unsigned long long* group_ws = reinterpret_cast<unsigned long long*>(w);
    w += static_cast<size_t>(slots) * group_bytes;
    SsspParams p{};
    p.g = g->csr(opts->metric);
    p.g.n = n;
    p.sources = o.sources;
    p.num_sources = job.num_sources;
    p.num_tiles = job.num_items;
    p.delta = job.plain_delta;
    p.graphs = o.graphs;
    p.items = job.d_items;
    p.max_iterations = opts->max_iterations > 0 ? opts->max_iterations : static_cast<unsigned long long>(4 * n + 64);
    p.tile_counter = o.tile_counter;
    p.error = o.error;
    p.abort_flag = g->d_abort;
    p.ws_dist = reinterpret_cast<unsigned long long*>(w);
    w += static_cast<size_t>(slots) * n * kTile * 8;
    p.ws_pend = reinterpret_cast<uint32_t*>(w);
    w += static_cast<size_t>(slots) * 3 * n * 4;
    p.ws_queue = reinterpret_cast<int32_t*>(w);
    w += static_cast<size_t>(slots) * 2 * n * 4;
    p.ws_stamp = reinterpret_cast<uint32_t*>(w);
    p.group_size = 1;
    p.group_stride = group_stride_words(1);
    p.group_ws = group_ws;
    BrandesParams bp{};
    p.out.acc_sum = o.acc;
    p.out.acc_inv = o.acc + kAccDigits;
    p.out.counters = o.counters;
    p.out.hist = hist_bins > 0 ? o.hist : nullptr;
    p.out.hist_bins = static_cast<int>(hist_bins);
    p.out.hist_max = hist_max;
    p.out.hist_width = hist_bins > 0 ? hist_max / static_cast<double>(hist_bins) : 0.0;
    if (o.src_f64 != nullptr) {
        p.out.src_sum = o.src_f64;
        p.out.src_max = o.src_f64 + job.num_sources;
        p.out.src_inv = o.src_f64 + 2 * job.num_sources;
    }
    if (o.src_u64 != nullptr) {
        p.out.src_unreach = o.src_u64;
        p.out.src_arcs = o.src_u64 + job.num_sources;
    }
    void* args[] = { &p, &bp };
    cudaError_t err = cudaMemsetAsync(group_ws, 0, static_cast<size_t>(slots) * group_bytes, g->stream);
    if (err == cudaSuccess) {
        err = cudaLaunchKernel(kernel, dim3(static_cast<unsigned>(slots)), dim3(block), args, smem, g->stream);
    }
    return err == cudaSuccess ? NGX_OK : cuda_fail(err, "tile kernel launch");
}

void clear_result_totals(ngx_apsp_result* r) {
    r->sum_distances = r->sum_inverse = r->diameter = 0.0;
    r->unreachable = r->reached_pairs = r->traversed_arcs = r->hist_overflow = 0;
    r->hist_max = 0.0;
    r->cpl = r->efficiency = 0.0;
    r->kernel_ms = 0.0;
    r->phases = r->expansions = r->lane_expansions = r->dag_levels = r->dag_entries = r->dag_scan_tiles = 0;
    for (int i = 0; i < 5; ++i) {
        r->phase_cycles[i] = 0;
    }
}

// Reduces graph `gi`'s accumulators and counters (host copies) into a result; copies its optional device outputs.
int collect_graph(ngx_graph* g, const RunOutputs& o, const unsigned long long* acc_all, const unsigned long long* counters_all, int64_t gi,
                  int64_t src_off, int64_t num_sources, int64_t hist_bins, double hist_max, ngx_apsp_result* r, const int32_t* scatter) {
    unsigned long long acc[2 * kAccDigits];
    std::memcpy(acc, acc_all + gi * 2 * kAccDigits, sizeof(acc));
    const unsigned long long* counters = counters_all + gi * kCounterCount;
    acc_normalize(acc);
    acc_normalize(acc + kAccDigits);
    r->sum_distances = acc_round_normalized(acc);
    r->sum_inverse = acc_round_normalized(acc + kAccDigits);
    if (r->acc_digits != nullptr) {
        std::memcpy(r->acc_digits, acc, sizeof(acc));
    }
    std::memcpy(&r->diameter, &counters[kDiameterBits], sizeof(double));
    r->unreachable = counters[kUnreachable];
    r->reached_pairs = counters[kReachedPairs];
    r->traversed_arcs = counters[kTraversedArcs];
    r->hist_overflow = counters[kHistOverflow];
    r->hist_max = hist_max;
    r->phases = counters[kIterations];
    r->expansions = counters[kExpansions];
    r->lane_expansions = counters[kLaneExpansions];
    r->dag_levels = counters[kDagLevels];
    r->dag_entries = counters[kDagEntries];
    r->dag_scan_tiles = counters[kDagScanTiles];
    for (int i = 0; i < 5; ++i) {
        r->phase_cycles[i] = counters[kCyclesSssp + i];
    }
    // AllPairsShortestPath.h:154-158: both averages are over the R reached ordered pairs (0 / 0 gives NaN, as there)
    r->cpl = r->sum_distances / static_cast<double>(r->reached_pairs);
    r->efficiency = r->sum_inverse / static_cast<double>(r->reached_pairs);
    const size_t s = static_cast<size_t>(num_sources);
    const size_t total = static_cast<size_t>(o.num_sources);
    const size_t at = static_cast<size_t>(src_off);
    if (r->hist != nullptr && hist_bins > 0) {
        NGX_CUDA_TRY(cudaMemcpyAsync(r->hist, o.hist + gi * hist_bins, static_cast<size_t>(hist_bins) * 8, cudaMemcpyDeviceToHost, g->stream));
    }
    if (s > 0 && scatter != nullptr) {
        // the run took the sources in the graph's locality order: entry i belongs to vertex scatter[i]
        // (all the wanted arrays come back with one wait)
        const std::pair<void*, const void*> wanted[] = { { r->src_sum, o.src_f64 + at },
                                                         { r->src_max, o.src_f64 + total + at },
                                                         { r->src_sum_inverse, o.src_f64 + 2 * total + at },
                                                         { r->src_unreachable, o.src_u64 + at },
                                                         { r->src_arcs, o.src_u64 + total + at } };
        std::vector<unsigned long long> tmp(5 * s);
        for (size_t k = 0; k < 5; ++k) {
            if (wanted[k].first != nullptr) {
                NGX_CUDA_TRY(cudaMemcpyAsync(tmp.data() + k * s, wanted[k].second, s * 8, cudaMemcpyDeviceToHost, g->stream));
            }
        }
        NGX_CUDA_TRY(cudaStreamSynchronize(g->stream));
        for (size_t k = 0; k < 5; ++k) {
            if (auto* out = static_cast<unsigned long long*>(wanted[k].first); out != nullptr) {
                for (size_t i = 0; i < s; ++i) {
                    out[scatter[i]] = tmp[k * s + i];
                }
            }
        }
        return NGX_OK;
    }
    if (s > 0) {
        if (r->src_sum != nullptr) NGX_CUDA_TRY(cudaMemcpyAsync(r->src_sum, o.src_f64 + at, s * 8, cudaMemcpyDeviceToHost, g->stream));
        if (r->src_max != nullptr) NGX_CUDA_TRY(cudaMemcpyAsync(r->src_max, o.src_f64 + total + at, s * 8, cudaMemcpyDeviceToHost, g->stream));
        if (r->src_sum_inverse != nullptr) {
            NGX_CUDA_TRY(cudaMemcpyAsync(r->src_sum_inverse, o.src_f64 + 2 * total + at, s * 8, cudaMemcpyDeviceToHost, g->stream));
        }
        if (r->src_unreachable != nullptr) NGX_CUDA_TRY(cudaMemcpyAsync(r->src_unreachable, o.src_u64 + at, s * 8, cudaMemcpyDeviceToHost, g->stream));
        if (r->src_arcs != nullptr) NGX_CUDA_TRY(cudaMemcpyAsync(r->src_arcs, o.src_u64 + total + at, s * 8, cudaMemcpyDeviceToHost, g->stream));
    }
    return NGX_OK;
}

int read_totals(ngx_graph* g, const RunOutputs& o, std::vector<unsigned long long>& acc, std::vector<unsigned long long>& counters) {
    acc.resize(static_cast<size_t>(o.num_graphs) * 2 * kAccDigits);
    counters.resize(static_cast<size_t>(o.num_graphs) * kCounterCount);
    NGX_CUDA_TRY(cudaMemcpyAsync(acc.data(), o.acc, acc.size() * 8, cudaMemcpyDeviceToHost, g->stream));
    NGX_CUDA_TRY(cudaMemcpyAsync(counters.data(), o.counters, counters.size() * 8, cudaMemcpyDeviceToHost, g->stream));
    NGX_CUDA_TRY(cudaStreamSynchronize(g->stream));
    return NGX_OK;
}

// One single-graph run of `sources` (graph 0 of the handle).
int run_sources(ngx_graph* g, const ngx_apsp_opts* opts, int tile_mode, const std::vector<int32_t>& sources, int64_t hist_bins, double hist_max,
                bool want_rows, DagOutputs* extra, RunOutputs& o, float* ms, const TileJob* with = nullptr) {
    const int64_t num_sources = static_cast<int64_t>(sources.size());
    if (const int rc = alloc_outputs(g, 1, num_sources, hist_bins, want_rows, o, false); rc != NGX_OK) {
        return rc;
    }
    const GraphPart& part = g->parts[0];
    const bool batched = opts->mode == NGX_MODE_BATCHED || tile_mode == kModeGrad;
    const double delta = pick_delta(opts->metric == NGX_METRIC_INVERSE ? part.mean_len_inverse : part.mean_len_regular, opts->delta,
                                    batched ? default_delta_scale(part) : degree_delta_scale(part.n, part.m_stored));
    const GraphDesc desc{ part.n, part.m_stored, part.row_off, 0, num_sources, part.vertex_off, delta };
    NGX_CUDA_TRY(cudaMemsetAsync(o.block, 0, o.zeroed_bytes, g->stream));
    NGX_CUDA_TRY(cudaMemcpyAsync(o.graphs, &desc, sizeof(desc), cudaMemcpyHostToDevice, g->stream));
    NGX_CUDA_TRY(cudaMemcpyAsync(o.sources, sources.data(), sizeof(int32_t) * sources.size(), cudaMemcpyHostToDevice, g->stream));
    TileJob job = with != nullptr ? *with : TileJob{};  // (its landmark fields)
    job.num_graphs = 1;
    job.num_items = (num_sources + kTile - 1) / kTile;
    job.d_items = nullptr;
    job.num_sources = num_sources;
    job.n_max = part.n;
    job.num_arcs = part.m_stored;
    job.plain_delta = delta;
    job.track_reach = g->scc_components > 1;
    return launch_tiles(g, opts, tile_mode, job, hist_bins, hist_max, o, extra, ms, true);
}

// Bytes of the landmarks' distance rows, from and to.
size_t landmark_bytes(const ngx_graph* g) { return 2 * static_cast<size_t>(kTile) * static_cast<size_t>(g->n) * sizeof(double); }

// Whether a run of `tiles` source tiles pays for landmark bounds: two more tiles, each run by itself, and memory for
// 2 x kTile rows.
//  * Twelve waves or more of the library's own group size. Kernel times without and with at that line, log-normal lengths of
//    sigma 1 (APSP; Brandes; gradient, ms): 14,000 vertices at degree 40, 252 tiles: 30.7, 29.6; 39.1, 38.0; 58.0, 57.1; 20,000
//    at 60, 252: 47.5, 43.7; 58.5, 55.3; 88.7, 85.6; 30,000 at 40, 168: 45.1, 42.9; 55.5, 54.5; 86.8, 85.2; 50,000 at 40, 96: 44.6,
//    43.8; 55.0, 55.5; 85.2, 84.9; 100,000 at 40, 60: 57.2, 58.8; 71.4, 72.0; 113.5, 114.1 (the one graph that would have the line
//    higher, at 75 tiles); 100,000 at 100, 60: 69.9, 64.4; 84.6, 81.4; 128.8, 125.2; 200,000 at 40, 48: 93.9, 93.0; 118.7, 118.6;
//    194.7, 194.0; 1,000,000 at 40, 48: 527, 500; 661, 644; 1127, 1108.
//  * 128 tiles or more where the caller sets the group size, since waves of any size say little about a tile's work: with 74
//    CTAs (12 waves are 48 tiles) APSP without and with, 30,000 at 40: 48 tiles 17.5, 18.2; 64: 23.4, 23.7; 96: 34.8, 34.7; 128:
//    46.7, 45.7; 8000 at 40: 48: 9.2, 9.9; 96: 18.2, 18.6; 128: 24.3, 24.4; 160: 30.7, 29.9.
//  * Lengths that spread: mean(len) x mean(1 / len) is 1 for equal lengths, 1.3 and 2.7 for log-normal weights of sigma 0.5
//    and 1, 1.6 for integers up to 10. Measured kernel times without and with: sigma 1, APSP of 148 tiles on 100,000
//    vertices 181 and 158 ms, Brandes of 74 tiles 108 and 102 ms, APSP of 938 tiles on 30,000 vertices 267 and 240 ms;
//    sigma 0.5, gradient of 128 tiles 115 and 118 ms; integers 60.5 and 60.2; unit weights 125.4 and 126.4.
//  * A strongly connected graph (tiles with reach lists start without bounds) of filtered vertices, the regular metric
//    (the reverse arcs have no other lengths), and an eighth of the workspace memory.
bool landmarks_pay(const ngx_graph* g, const ngx_apsp_opts* opts, int64_t tiles) {
    const GraphPart& part = g->parts[0];
    if (opts->mode != NGX_MODE_BATCHED || opts->metric != NGX_METRIC_REGULAR || opts->max_iterations != 0 || g->scc_components != 1 ||
        g->m_stored < kFilterDegree * g->n || part.mean_len_regular * part.mean_len_inverse < 2.0) {
        return false;
    }
    const int64_t resident = 2 * static_cast<int64_t>(g->sm_count);  // the default launch shape
    const int group = choose_group_size(opts->tile_ctas, resident, tiles, resident, static_cast<double>(g->n),
                                        static_cast<double>(g->m_stored) / static_cast<double>(g->n));
    return tiles >= 12 * (resident / group) && (opts->tile_ctas == 0 || tiles >= 128) && landmark_bytes(g) <= (workspace_budget(g) + g->landmarks_bytes) / 8;
}

// Distances from and to kTile landmarks spread over the vertex ids, for the tiles' first bounds (landmark_bounds): one tile
// over the forward arcs and one over the reverse arcs.
int compute_landmarks(ngx_graph* g, const ngx_apsp_opts* opts, TileJob* with, float* ms) {
    const size_t rows = static_cast<size_t>(kTile) * static_cast<size_t>(g->n);
    const size_t bytes = landmark_bytes(g);
    if (g->memory_budget != 0 && g->workspace_bytes + bytes > g->memory_budget) {
        // the budget holds both only with a smaller workspace, which the runs below allocate
        if (const int rc = release_workspace(g); rc != NGX_OK) {
            return rc;
        }
    }
    if (g->d_landmarks == nullptr) {
        NGX_CUDA_TRY(cudaMalloc(&g->d_landmarks, bytes));
        g->landmarks_bytes = bytes;
    }
    std::vector<int32_t> landmarks(kTile);
    for (int64_t l = 0; l < kTile; ++l) {
        landmarks[static_cast<size_t>(l)] = static_cast<int32_t>((2 * l + 1) * g->n / (2 * kTile));
    }
    ngx_apsp_opts plain = *opts;
    plain.tile_ctas = 0;
    for (int to = 0; to < 2; ++to) {
        TileJob job;
        job.rows = static_cast<double*>(g->d_landmarks) + (to != 0 ? rows : 0);
        job.reverse = to != 0;
        RunOutputs o;
        const int rc = run_sources(g, &plain, kModeApsp, landmarks, 0, 0.0, false, nullptr, o, ms, &job);
        free_outputs(g, o);
        if (rc != NGX_OK) {
            return rc;
        }
    }
    with->landmark_from = static_cast<const double*>(g->d_landmarks);
    with->landmark_to = with->landmark_from + rows;
    return NGX_OK;
}

// Histogram bound when the caller gives none: 1.5 x the largest eccentricity of up to one tile of sources spread
// over the requested list (plus the overflow count for anything beyond it).
int auto_hist_max(ngx_graph* g, const ngx_apsp_opts* opts, const std::vector<int32_t>& sources, double* out) {
    const int64_t k = std::min<int64_t>(kTile, static_cast<int64_t>(sources.size()));
    std::vector<int32_t> sample(static_cast<size_t>(k));
    for (int64_t i = 0; i < k; ++i) {
        sample[static_cast<size_t>(i)] = sources[static_cast<size_t>(i * static_cast<int64_t>(sources.size()) / k)];
    }
    ngx_apsp_opts sample_opts = *opts;
    sample_opts.mode = NGX_MODE_BATCHED;
    RunOutputs o;
    int rc = run_sources(g, &sample_opts, kModeApsp, sample, 0, 0.0, false, nullptr, o, nullptr);
    unsigned long long bits = 0;
    if (rc == NGX_OK) {
        std::vector<unsigned long long> acc, counters;
        rc = read_totals(g, o, acc, counters);
        if (rc == NGX_OK) {
            bits = counters[kDiameterBits];
        }
    }
    free_outputs(g, o);
    double ecc = 0.0;
    std::memcpy(&ecc, &bits, sizeof(double));
    *out = ecc > 0.0 ? 1.5 * ecc : 1.0;
    return rc;
}

int run_apsp(ngx_graph* g, const ngx_apsp_opts* caller_opts, ngx_apsp_result* result, double* rows, int tile_mode, DagOutputs* extra) {
    if (const int rc = check_opts(g, caller_opts); rc != NGX_OK) {
        return rc;
    }
    // options left at 0 take the handle's tuned values for this task (ngx_graph_autotune), if any
    ngx_apsp_opts tuned_opts = *caller_opts;
    const ngx_tuning& t = g->tuned[tile_mode];
    if (t.block_threads > 0 && tuned_opts.mode == NGX_MODE_BATCHED) {
        if (tuned_opts.block_threads == 0 && tuned_opts.ctas_per_sm == 0) {
            tuned_opts.block_threads = t.block_threads;
            tuned_opts.ctas_per_sm = t.ctas_per_sm;
        }
        if (tuned_opts.tile_ctas == 0) {
            tuned_opts.tile_ctas = t.tile_ctas;
        }
        if (!(tuned_opts.delta > 0.0) && g->parts.size() == 1) {
            const GraphPart& part = g->parts[0];
            tuned_opts.delta = pick_delta(tuned_opts.metric == NGX_METRIC_INVERSE ? part.mean_len_inverse : part.mean_len_regular, 0.0, t.delta_scale);
        }
    }
    const ngx_apsp_opts* opts = &tuned_opts;
    if (g->parts.size() != 1) {
        return fail(NGX_INVALID_ARGUMENT, "this handle holds a batch of graphs: use ngx_batch_run");
    }
    NGX_CUDA_TRY(cudaSetDevice(g->device));
    *g->h_abort = 0;
    // the strongly connected components decide whether tiles keep reach lists (several components)
    if (const int rc = ensure_components(g); rc != NGX_OK) {
        return rc;
    }
    std::vector<int32_t> sources;
    if (const int rc = prepare_sources(g, opts, sources); rc != NGX_OK) {
        return rc;
    }
    // all sources: in the graph's locality order (tiles of nearby sources), results scattered back by vertex;
    // distance rows keep vertex order
    const int32_t* scatter = nullptr;
    if (opts->sources == nullptr && rows == nullptr) {
        if (const int rc = ensure_source_order(g); rc != NGX_OK) {
            return rc;
        }
    }
    if (opts->sources == nullptr && rows == nullptr && g->source_order.size() == sources.size()) {
        sources.assign(g->source_order.begin(), g->source_order.end());
        scatter = g->source_order.data();
    }
    ngx_apsp_result scratch{};
    ngx_apsp_result* r = result != nullptr ? result : &scratch;
    clear_result_totals(r);
    const int64_t num_sources = static_cast<int64_t>(sources.size());
    if (num_sources == 0 || g->n == 0) {
        r->cpl = r->efficiency = NAN;  // no reached pairs, as 0 / 0 in AllPairsShortestPath.h:157-158
        return NGX_OK;
    }
    const bool landmarks = landmarks_pay(g, opts, (num_sources + kTile - 1) / kTile);
    if (!landmarks) {
        drop_landmarks(g);
    }
    const int64_t hist_bins = opts->hist_bins;
    double hist_max = opts->hist_max;
    if (hist_bins > 0 && !(hist_max > 0.0)) {
        if (const int rc = auto_hist_max(g, opts, sources, &hist_max); rc != NGX_OK) {
            return rc;
        }
    }
    RunOutputs o;
    float ms = 0.0f;
    TileJob with;
    if (landmarks) {
        const int rc_l = compute_landmarks(g, opts, &with, &ms);
        if (rc_l == NGX_OUT_OF_MEMORY || rc_l == NGX_TIMEOUT) {
            cudaGetLastError();  // the run does without
            set_last_error("");
            with = TileJob{};
            drop_landmarks(g);
        } else if (rc_l != NGX_OK) {
            return rc_l;
        }
    }
    int rc = run_sources(g, opts, tile_mode, sources, hist_bins, hist_max, rows != nullptr, extra, o, &ms, &with);
    if (rc == NGX_OK) {
        std::vector<unsigned long long> acc, counters;
        rc = read_totals(g, o, acc, counters);
        if (rc == NGX_OK) {
            rc = collect_graph(g, o, acc.data(), counters.data(), 0, 0, num_sources, hist_bins, hist_max, r, scatter);
        }
        r->kernel_ms = ms;
    }
    if (rc == NGX_OK && rows != nullptr) {
        const cudaError_t err = cudaMemcpyAsync(rows, o.rows, static_cast<size_t>(num_sources) * static_cast<size_t>(g->n) * 8, cudaMemcpyDeviceToHost,
                                                g->stream);
        if (err != cudaSuccess) {
            rc = cuda_fail(err, "copying distance rows");
        }
    }
    cudaStreamSynchronize(g->stream);
    free_outputs(g, o);
    return rc;
}

}  // namespace ngx

using namespace ngx;

extern "C" {

int ngx_apsp(ngx_graph* graph, const ngx_apsp_opts* opts, ngx_apsp_result* result) {
    return guard_host("ngx_apsp", [&]() -> int { return run_apsp(graph, opts, result, nullptr, kModeApsp, nullptr); });
}

int ngx_sssp_rows(ngx_graph* graph, const ngx_apsp_opts* opts, double* rows) {
    return guard_host("ngx_sssp_rows", [&]() -> int {
        if (rows == nullptr || opts == nullptr) {
            return fail(NGX_INVALID_ARGUMENT, "ngx_sssp_rows: opts or rows is NULL");
        }
        ngx_apsp_opts o = *opts;
        o.hist_bins = 0;
        return run_apsp(graph, &o, nullptr, rows, kModeApsp, nullptr);
    });
}

}  // extern "C"
