// Host-side helpers shared by the APSP, Brandes and gradient runs (private to the library).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "ngx_common.cuh"
#include "ngx_graph.h"

namespace ngx {

constexpr int64_t kMaxHistBins = 16384;

// Device buffers of one run's reduced outputs, carved from one allocation.
struct RunOutputs {
    unsigned long long* acc = nullptr;       // per graph 2 * kAccDigits: exact sums of d and of 1/d
    unsigned long long* counters = nullptr;  // per graph kCounterCount
    unsigned long long* hist = nullptr;      // per graph hist_bins
    GraphDesc* graphs = nullptr;             // the run's graph table
    int32_t* sources = nullptr;              // all graphs' sources, graph after graph
    double* src_f64 = nullptr;               // 3 * S: per-source sum, max, inverse sum
    unsigned long long* src_u64 = nullptr;   // 2 * S: per-source unreachable, traversed arcs
    double* rows = nullptr;                  // S * n distance rows, when requested
    int* error = nullptr;
    unsigned long long* tile_counter = nullptr;
    void* block = nullptr;
    bool owned = true;                       // false: the graph's persistent buffer (CUDA graph replays)
    size_t bytes = 0;
    size_t zeroed_bytes = 0;                 // leading bytes (accumulators, counters, flags) reset before each run
    int64_t num_graphs = 0;
    int64_t num_sources = 0;
};

// What one launch covers: a graph table and sources already in the outputs block, and the work items.
struct TileJob {
    int64_t num_graphs = 1;
    int64_t num_items = 0;             // (graph, tile) work items
    const WorkItem* d_items = nullptr; // nullptr: tile t of graph 0
    int64_t num_sources = 0;
    int64_t n_max = 0;                 // largest graph (workspace slot size)
    int64_t num_arcs = 0;              // stored arcs of the job's graphs
    double plain_delta = 1.0;          // bucket width of the plain form (single graph)
    // single-graph runs with landmark bounds; a landmark run writes its distance rows to `rows`, over the reverse arcs
    // when `reverse`
    const double* landmark_from = nullptr;
    const double* landmark_to = nullptr;
    double* rows = nullptr;
    bool reverse = false;
    bool track_reach = false;          // keep per-tile reach lists (a graph of several strongly connected components)
};

// Device buffers of the DAG passes: per-vertex betweenness and per-arc gradients in 128-bit fixed point.
struct DagOutputs {
    unsigned long long* bc = nullptr;        // 2 * n
    unsigned long long* grad_cpl = nullptr;  // 2 * m_user
    unsigned long long* grad_eff = nullptr;  // 2 * m_user
    int* sigma_inexact = nullptr;            // device flag: a pushed sigma sum reached 2^53
    int sigma_pull = 0;                      // run the sigma pass in pull form
};

int check_opts(const ngx_graph* g, const ngx_apsp_opts* opts);
int run_apsp(ngx_graph* g, const ngx_apsp_opts* opts, ngx_apsp_result* result, double* rows, int tile_mode, DagOutputs* extra);
int prepare_sources(const ngx_graph* g, const ngx_apsp_opts* opts, std::vector<int32_t>& sources);
// A bucket width by density, as a multiple of the mean arc length: 2 / sqrt(mean out-degree), clamped to 0.125-2. Dense
// graphs want narrow buckets (many arcs relax into each bucket: a wide one re-relaxes more pairs), sparse ones wide buckets
// (few arcs per bucket: a narrow one runs many nearly empty phases).
double degree_delta_scale(int64_t n, int64_t m);
// Bucket width of the batched form when the caller gives none: twice that where wide buckets re-relax little, which is on
// sparse graphs (mean out-degree below 28) and where few arcs are much shorter than the mean (mean(len) x mean(1 / len)
// below 2: 1 for equal lengths, 1.3 and 2.7 for log-normal weights of sigma 0.5 and 1, 1.6 for integers up to 10). Kernel
// times in ms at 1 x and 2 x the width by density:
//   sigma 0.5: APSP of 2048 sources, n = 5e4, degree 40: 27.0, 25.8; gradient of the same 57.7, 56.2; Brandes, 3e4, 25: 39.1, 36.6;
//   integers: Brandes, n = 5000, degree 6: 13.2, 12.7; 1e4, 40: 59.5, 59.2; APSP, 3000, 50: 2.03, 2.04; unit weights equal;
//   sigma 1, sparse: APSP, n = 300, degree 8: 0.45, 0.37; 2e4, 2: 33.1, 29.8; 5e4, 6: 25.1, 24.1; Brandes, 3e4, 12: 42.3, 39.8;
//   the line, sigma 1, Brandes at degrees 20, 24, 28 and 31: n = 8000: 20.5, 20.6; 21.4, 21.4; 21.1, 21.6; 21.5, 21.7;
//   3e4: 40.2, 39.0; 39.6, 39.4; 39.9, 40.0; 40.8, 40.7; 2e5: 39.4, 38.2; 36.9, 35.6; 37.1, 36.4; 37.8, 37.1 (larger graphs
//   would have it higher); above it: APSP, 3e4, 60: 37.5, 37.8; 1e4, 90: 32.1, 32.7.
double default_delta_scale(const GraphPart& part);
double pick_delta(double mean_len, double requested, double scale);
int alloc_outputs(ngx_graph* g, int64_t num_graphs, int64_t num_sources, int64_t hist_bins, bool want_rows, RunOutputs& o, bool persistent);
void free_outputs(ngx_graph* g, RunOutputs& o);
int device_error_status(int code);
int launch_tiles(ngx_graph* g, const ngx_apsp_opts* opts, int tile_mode, const TileJob& job, int64_t hist_bins, double hist_max, RunOutputs& o,
                 DagOutputs* extra, float* kernel_ms, bool synchronous);
int launch_apsp_in_workspace(ngx_graph* g, const ngx_apsp_opts* opts, const TileJob& job, int64_t hist_bins, double hist_max, RunOutputs& o, void* ws,
                             size_t ws_bytes);
int read_totals(ngx_graph* g, const RunOutputs& o, std::vector<unsigned long long>& acc, std::vector<unsigned long long>& counters);
int collect_graph(ngx_graph* g, const RunOutputs& o, const unsigned long long* acc_all, const unsigned long long* counters_all, int64_t gi,
                  int64_t src_off, int64_t num_sources, int64_t hist_bins, double hist_max, ngx_apsp_result* r,
                  const int32_t* scatter = nullptr);
void clear_result_totals(ngx_apsp_result* r);

}  // namespace ngx
