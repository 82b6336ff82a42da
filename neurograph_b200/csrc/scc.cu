// Strongly connected components on the GPU: ngx_scc.
//
// Replaces StronglyConnectedComponents::compute_strongly_connected_components (source/metrics/connectivity/
// StronglyConnectedComponents.h:17-36): the number of components, the largest size and the size histogram, which
// every one of the reference's algorithms returns identically. Self arcs and weights are ignored; a vertex without
// arcs is a component of its own.
//
// Method (trimming + colouring, all passes over the device CSR and reverse CSR with a warp, or four lanes, per vertex):
//   trim     an unassigned vertex without an unassigned in- or out-neighbour (other than itself) is a component;
//   colour   every unassigned vertex starts with its own id and takes the largest colour among its unassigned
//            in-neighbours until nothing changes: colour(v) = the largest id that reaches v;
//   peel     each vertex whose colour is its own id is a root (the largest vertex of its component, which names the
//            component); the vertices of its colour that reach it are its component, found backwards: a vertex joins
//            when one of its out-neighbours of the same colour has joined.
// Trim, colour and peel repeat until every vertex has a component. Every pass is a kernel launch; the host
// reads the change flags after one or a few, so nothing waits on the device beyond one launch.

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <string>
#include <vector>

#include "ngx_common.cuh"
#include "ngx_graph.h"

namespace ngx {
namespace {

constexpr int kSccBlock = 256;

// The passes give each vertex a group of kLanes lanes of a warp: 32, or 4 at mean out-degrees below 8, where a whole warp
// would leave most lanes without an arc (300,000 vertices of out-degree 4: 4.2 -> 2.1 ms per call with the rest of the
// call's changes).
constexpr int kSparseLanes = 4;
template <int kLanes>
__device__ __forceinline__ int64_t first_vertex() {
    return (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) / kLanes;
}
template <int kLanes>
__device__ __forceinline__ int64_t vertex_stride() {
    return static_cast<int64_t>(gridDim.x) * blockDim.x / kLanes;
}
// The lanes of this lane's group, as a warp mask.
template <int kLanes>
__device__ __forceinline__ unsigned group_mask() {
    return kLanes == 32 ? 0xFFFFFFFFu : ((1u << (kLanes & 31)) - 1u) << (threadIdx.x & 31u & ~static_cast<unsigned>(kLanes - 1));
}

// Assigns every unassigned vertex that has no unassigned in- or out-neighbour besides itself.
template <int kLanes>
__global__ void scc_trim_kernel(int64_t n, const int64_t* row_ptr, const Arc* arcs, const int64_t* rrow_ptr, const Arc* rarcs, int32_t* comp,
                                int* changed) {
    const int lane = threadIdx.x & (kLanes - 1);
    const unsigned group = group_mask<kLanes>();
    for (int64_t v = first_vertex<kLanes>(); v < n; v += vertex_stride<kLanes>()) {
        if (comp[v] >= 0) {
            continue;  // uniform in the group
        }
        bool has_out = false, has_in = false;
        for (int64_t e = row_ptr[v] + lane; e < row_ptr[v + 1] && !has_out; e += kLanes) {
            const int32_t x = arcs[e].col;
            has_out = x != v && __ldcg(&comp[x]) < 0;
        }
        for (int64_t e = rrow_ptr[v] + lane; e < rrow_ptr[v + 1] && !has_in; e += kLanes) {
            const int32_t x = rarcs[e].col;
            has_in = x != v && __ldcg(&comp[x]) < 0;
        }
        const bool out_any = __any_sync(group, has_out);
        const bool in_any = __any_sync(group, has_in);
        if (lane == 0 && (!out_any || !in_any)) {
            comp[v] = static_cast<int32_t>(v);
            *changed = 1;
        }
    }
}

__global__ void scc_color_init_kernel(int64_t n, const int32_t* comp, int32_t* color, uint8_t* visited) {
    for (int64_t v = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; v < n; v += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        color[v] = comp[v] < 0 ? static_cast<int32_t>(v) : -1;
        visited[v] = 0;
    }
}

// colour(v) = max(colour(v), colour(u)) over unassigned in-neighbours u (pulled, so each vertex writes only itself).
template <int kLanes>
__global__ void scc_color_kernel(int64_t n, const int64_t* rrow_ptr, const Arc* rarcs, const int32_t* comp, int32_t* color, int* changed) {
    const int lane = threadIdx.x & (kLanes - 1);
    const unsigned group = group_mask<kLanes>();
    for (int64_t v = first_vertex<kLanes>(); v < n; v += vertex_stride<kLanes>()) {
        if (comp[v] >= 0) {
            continue;
        }
        int32_t best = -1;
        for (int64_t e = rrow_ptr[v] + lane; e < rrow_ptr[v + 1]; e += kLanes) {
            const int32_t u = rarcs[e].col;
            if (__ldcg(&comp[u]) < 0) {
                best = max(best, __ldcg(&color[u]));
            }
        }
#pragma unroll
        for (int off = kLanes / 2; off > 0; off >>= 1) {
            best = max(best, __shfl_xor_sync(group, best, off));
        }
        if (lane == 0 && best > __ldcg(&color[v])) {
            atomicMax(&color[v], best);
            *changed = 1;
        }
    }
}

__global__ void scc_roots_kernel(int64_t n, const int32_t* comp, const int32_t* color, uint8_t* visited) {
    for (int64_t v = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; v < n; v += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        if (comp[v] < 0 && color[v] == static_cast<int32_t>(v)) {
            visited[v] = 1;
        }
    }
}

// A vertex joins its colour's root when one of its out-neighbours of the same colour already has.
template <int kLanes>
__global__ void scc_backward_kernel(int64_t n, const int64_t* row_ptr, const Arc* arcs, const int32_t* comp, const int32_t* color, uint8_t* visited,
                                    int* changed) {
    const int lane = threadIdx.x & (kLanes - 1);
    const unsigned group = group_mask<kLanes>();
    for (int64_t v = first_vertex<kLanes>(); v < n; v += vertex_stride<kLanes>()) {
        if (comp[v] >= 0 || __ldcg(&visited[v]) != 0) {
            continue;
        }
        const int32_t cv = color[v];
        bool hit = false;
        for (int64_t e = row_ptr[v] + lane; e < row_ptr[v + 1] && !hit; e += kLanes) {
            const int32_t x = arcs[e].col;
            hit = __ldcg(&visited[x]) != 0 && __ldcg(&color[x]) == cv && __ldcg(&comp[x]) < 0;
        }
        if (__any_sync(group, hit) && lane == 0) {
            visited[v] = 1;
            *changed = 1;
        }
    }
}

__global__ void scc_assign_kernel(int64_t n, int32_t* comp, const int32_t* color, const uint8_t* visited, int* remaining) {
    for (int64_t v = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; v < n; v += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        if (comp[v] < 0) {
            if (visited[v] != 0) {
                comp[v] = color[v];
            } else {
                atomicAdd(remaining, 1);
            }
        }
    }
}

// table[key] += 1 for every active lane, the lanes of one key with one atomic: most vertices share the giant component
// and most components the size 1, and 270,000 atomics on one word take half a millisecond.
__device__ __forceinline__ void count_key(unsigned long long* table, long long key, bool on) {
    const unsigned act = __ballot_sync(0xFFFFFFFFu, on);
    if (on) {
        const unsigned peers = __match_any_sync(act, key);
        if (__ffs(peers) - 1 == static_cast<int>(threadIdx.x & 31)) {
            atomicAdd(&table[key], static_cast<unsigned long long>(__popc(peers)));
        }
    }
}

__global__ void scc_count_kernel(int64_t n, const int32_t* comp, unsigned long long* sizes) {
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t v0 = blockIdx.x * static_cast<int64_t>(blockDim.x); v0 < n; v0 += stride) {
        const int64_t v = v0 + threadIdx.x;
        count_key(sizes, v < n ? comp[v] : 0, v < n);
    }
}

// totals[0] = components, totals[1] = the largest one's size; hist[s] (unless nullptr) = components of size s.
__global__ void scc_summary_kernel(int64_t n, const unsigned long long* sizes, unsigned long long* totals, unsigned long long* hist) {
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    unsigned count = 0;
    unsigned long long largest = 0;
    for (int64_t v0 = blockIdx.x * static_cast<int64_t>(blockDim.x); v0 < n; v0 += stride) {
        const int64_t v = v0 + threadIdx.x;
        const unsigned long long size = v < n ? sizes[v] : 0ull;
        count += size != 0ull ? 1u : 0u;
        largest = size > largest ? size : largest;
        if (hist != nullptr) {
            count_key(hist, static_cast<long long>(size), size != 0ull);
        }
    }
    count = __reduce_add_sync(0xFFFFFFFFu, count);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const unsigned long long o = __shfl_xor_sync(0xFFFFFFFFu, largest, off);
        largest = o > largest ? o : largest;
    }
    if ((threadIdx.x & 31) == 0 && count != 0u) {
        atomicAdd(&totals[0], static_cast<unsigned long long>(count));
        atomicMax(&totals[1], largest);
    }
}

// The non-zero entries of the size histogram as (size, components) pairs, in any order; totals[2] counts them. There are
// at most about sqrt(2 n) different sizes, so far less comes back to the host than the histogram's n + 1 words.
__global__ void scc_pairs_kernel(int64_t n, const unsigned long long* hist, unsigned long long* totals, unsigned long long* pairs) {
    for (int64_t size = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; size <= n; size += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const unsigned long long count = hist[size];
        if (count != 0ull) {
            const unsigned long long at = atomicAdd(&totals[2], 1ull);
            pairs[2 * at] = static_cast<unsigned long long>(size);
            pairs[2 * at + 1] = count;
        }
    }
}

// Runs `launch(flag)` (which may set *flag) until a pass leaves its flag clear. Every pass that sets it makes progress on a
// finite quantity (an assignment, a larger colour, a new member), so n + 1 passes always suffice. Passes after the last
// change do nothing, so several are launched for each look at their flags where a pass costs less than the round trip
// to the host: up to 4e6 arcs, about 15 us either way. The pre-pass's cap counts the passes up to the first clear flag,
// as many as one look per pass would take.
constexpr int kPassesPerLook = 4;
template <typename Launch>
int until_stable(ngx_graph* g, int* d_flags, int64_t max_passes, Launch launch) {
    const int per_look = g->m_stored <= 4000000 ? kPassesPerLook : 1;
    int flags[kPassesPerLook] = {};
    for (int64_t pass = 0; pass <= max_passes; pass += per_look) {
        NGX_CUDA_TRY(cudaMemsetAsync(d_flags, 0, per_look * sizeof(int), g->stream));
        for (int i = 0; i < per_look; ++i) {
            launch(d_flags + i);
        }
        NGX_CUDA_TRY(cudaGetLastError());
        NGX_CUDA_TRY(cudaMemcpyAsync(flags, d_flags, per_look * sizeof(int), cudaMemcpyDeviceToHost, g->stream));
        NGX_CUDA_TRY(cudaStreamSynchronize(g->stream));
        int changing = 0;
        while (changing < per_look && flags[changing] != 0) {
            ++changing;
        }
        const bool stable = changing < per_look;
        if (g->scc_pass_cap > 0 && (g->scc_passes += changing + (stable ? 1 : 0)) > g->scc_pass_cap) {
            return fail(NGX_TIMEOUT, "ngx_scc: more passes than the pre-pass allows");
        }
        if (stable) {
            return NGX_OK;
        }
    }
    return fail(NGX_TIMEOUT, "ngx_scc: a pass did not converge");
}

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

}  // namespace
}  // namespace ngx

using namespace ngx;

extern "C" {

int ngx_scc(ngx_graph* g, int32_t* component, uint64_t* number_components, uint64_t* largest_component, uint64_t* size_histogram) {
    return guard_host("ngx_scc", [&]() -> int {
        if (g == nullptr || number_components == nullptr || largest_component == nullptr) {
            return fail(NGX_INVALID_ARGUMENT, "ngx_scc: graph or outputs are NULL");
        }
        if (g->parts.size() != 1) {
            return fail(NGX_INVALID_ARGUMENT, "ngx_scc: this handle holds a batch of graphs");
        }
        const int64_t n = g->n;
        *number_components = 0;
        *largest_component = 0;
        if (size_histogram != nullptr) {
            std::fill(size_histogram, size_histogram + n + 1, uint64_t(0));
        }
        if (n == 0) {
            return NGX_OK;
        }
        NGX_CUDA_TRY(cudaSetDevice(g->device));
        const size_t words = static_cast<size_t>(n);
        // device layout: comp i32[n] | color i32[n] | sizes u64[n] | visited u8[n] | flags i32[kPassesPerLook + 1], totals u64[3] |
        // (size, components) pairs | size histogram u64[n + 1], each 256-byte aligned
        const size_t off_color = align256(words * 4);
        const size_t off_sizes = off_color + align256(words * 4);
        const size_t off_visited = off_sizes + align256(words * 8);
        const size_t off_flags = off_visited + align256(words);
        const size_t off_pairs = off_flags + 256;
        // distinct component sizes: 1 + 2 + ... + k <= n
        const size_t most_pairs = static_cast<size_t>(std::sqrt(2.0 * static_cast<double>(n))) + 2;
        const size_t off_hist = off_pairs + align256(most_pairs * 16);
        const size_t bytes = off_hist + (size_histogram != nullptr ? align256((words + 1) * 8) : 0);
        if (const int rc = grow_buffer(g, &g->d_call_out, &g->call_out_bytes, bytes); rc != NGX_OK) {
            return rc;
        }
        char* base = static_cast<char*>(g->d_call_out);
        auto* comp = reinterpret_cast<int32_t*>(base);
        auto* color = reinterpret_cast<int32_t*>(base + off_color);
        auto* sizes = reinterpret_cast<unsigned long long*>(base + off_sizes);
        auto* visited = reinterpret_cast<uint8_t*>(base + off_visited);
        auto* flags = reinterpret_cast<int*>(base + off_flags);
        NGX_CUDA_TRY(cudaMemsetAsync(comp, 0xFF, words * 4, g->stream));  // -1: no component yet
        const int vgrid = static_cast<int>(std::min<int64_t>((n + kSccBlock - 1) / kSccBlock, 8 * int64_t(g->sm_count)));
        const bool few_arcs = g->m_stored < 8 * n;
        const int64_t lanes = few_arcs ? kSparseLanes : 32;
        const int wgrid = static_cast<int>(std::min<int64_t>((n * lanes + kSccBlock - 1) / kSccBlock, 32 * int64_t(g->sm_count)));
        const int64_t* row_ptr = g->d_row_ptr;
        const Arc* arcs = g->d_arcs_regular;
        const int64_t* rrow_ptr = g->d_rrow_ptr;
        const Arc* rarcs = g->d_rarcs;
        // every round assigns at least the largest unassigned vertex (its own colour's root)
        bool done = false;
        for (int64_t round = 0; round <= n && !done; ++round) {
            int rc = until_stable(g, flags, n, [&](int* flag) {
                const auto kernel = few_arcs ? scc_trim_kernel<kSparseLanes> : scc_trim_kernel<32>;
                kernel<<<wgrid, kSccBlock, 0, g->stream>>>(n, row_ptr, arcs, rrow_ptr, rarcs, comp, flag);
            });
            if (rc != NGX_OK) {
                return rc;
            }
            scc_color_init_kernel<<<vgrid, kSccBlock, 0, g->stream>>>(n, comp, color, visited);
            NGX_CUDA_TRY(cudaGetLastError());
            rc = until_stable(g, flags, n, [&](int* flag) {
                const auto kernel = few_arcs ? scc_color_kernel<kSparseLanes> : scc_color_kernel<32>;
                kernel<<<wgrid, kSccBlock, 0, g->stream>>>(n, rrow_ptr, rarcs, comp, color, flag);
            });
            if (rc != NGX_OK) {
                return rc;
            }
            scc_roots_kernel<<<vgrid, kSccBlock, 0, g->stream>>>(n, comp, color, visited);
            NGX_CUDA_TRY(cudaGetLastError());
            rc = until_stable(g, flags, n, [&](int* flag) {
                const auto kernel = few_arcs ? scc_backward_kernel<kSparseLanes> : scc_backward_kernel<32>;
                kernel<<<wgrid, kSccBlock, 0, g->stream>>>(n, row_ptr, arcs, comp, color, visited, flag);
            });
            if (rc != NGX_OK) {
                return rc;
            }
            int* const left = flags + kPassesPerLook;  // vertices without a component remain
            NGX_CUDA_TRY(cudaMemsetAsync(left, 0, sizeof(int), g->stream));
            scc_assign_kernel<<<vgrid, kSccBlock, 0, g->stream>>>(n, comp, color, visited, left);
            NGX_CUDA_TRY(cudaGetLastError());
            int remaining = 0;
            NGX_CUDA_TRY(cudaMemcpyAsync(&remaining, left, sizeof(int), cudaMemcpyDeviceToHost, g->stream));
            NGX_CUDA_TRY(cudaStreamSynchronize(g->stream));
            done = remaining == 0;
        }
        if (!done) {
            return fail(NGX_TIMEOUT, "ngx_scc: components did not converge");
        }
        // component sizes: a component is named by its largest vertex, so sizes[] is indexed by vertex
        NGX_CUDA_TRY(cudaMemsetAsync(sizes, 0, words * 8, g->stream));
        scc_count_kernel<<<vgrid, kSccBlock, 0, g->stream>>>(n, comp, sizes);
        NGX_CUDA_TRY(cudaGetLastError());
        auto* totals = reinterpret_cast<unsigned long long*>(base + off_flags + 64);
        auto* pairs = reinterpret_cast<unsigned long long*>(base + off_pairs);
        auto* hist = size_histogram != nullptr ? reinterpret_cast<unsigned long long*>(base + off_hist) : nullptr;
        NGX_CUDA_TRY(cudaMemsetAsync(totals, 0, 3 * sizeof(unsigned long long), g->stream));
        if (hist != nullptr) {
            NGX_CUDA_TRY(cudaMemsetAsync(hist, 0, (words + 1) * 8, g->stream));
        }
        scc_summary_kernel<<<vgrid, kSccBlock, 0, g->stream>>>(n, sizes, totals, hist);
        NGX_CUDA_TRY(cudaGetLastError());
        if (hist != nullptr) {
            scc_pairs_kernel<<<vgrid, kSccBlock, 0, g->stream>>>(n, hist, totals, pairs);
            NGX_CUDA_TRY(cudaGetLastError());
        }
        // totals and pairs are neighbours: one copy
        std::vector<unsigned long long> host((off_pairs - off_flags) / 8 + (hist != nullptr ? 2 * most_pairs : 0));
        NGX_CUDA_TRY(cudaMemcpyAsync(host.data(), base + off_flags, host.size() * 8, cudaMemcpyDeviceToHost, g->stream));
        if (component != nullptr) {
            NGX_CUDA_TRY(cudaMemcpyAsync(component, comp, words * 4, cudaMemcpyDeviceToHost, g->stream));
        }
        NGX_CUDA_TRY(cudaStreamSynchronize(g->stream));
        *number_components = host[8];
        *largest_component = host[9];
        if (size_histogram != nullptr) {
            const unsigned long long* const found = host.data() + (off_pairs - off_flags) / 8;
            for (unsigned long long k = 0; k < host[10]; ++k) {
                size_histogram[found[2 * k]] = found[2 * k + 1];
            }
        }
        return NGX_OK;
    });
}

}  // extern "C"
