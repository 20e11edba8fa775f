// Building the hot-table pull engine's layout (gbx_pull.cuh).
//
// A histogram of out-degrees -- how often a vertex is a source in the pull
// CSR, exactly so with an inverse CSR or a symmetric graph and a fair guess
// otherwise -- gives the degree from which on vertices get a slot; slots and
// rows with edges are numbered by prefix sums, and one pass rewrites the edge
// ids as words: it looks every source up in a bitmap of V / 8 bytes, which L1
// serves far better than a word per vertex, and only sources with a slot in
// their slot's number.
#include <algorithm>
#include <vector>

#include "gbx_pull.cuh"

namespace gbx {
namespace {

// Degree classes: exact below 64, then 64 steps per power of two.
constexpr uint32_t kDegreeBins = 64 + 26 * 64;
__host__ __device__ __forceinline__ uint32_t degree_bin(uint32_t d) {
    if (d < 64) return d;
#ifdef __CUDA_ARCH__
    const uint32_t e = 31u - __clz(d);
#else
    const uint32_t e = 31u - (uint32_t)__builtin_clz(d);
#endif
    return 64 + (e - 6) * 64 + ((d >> (e - 6)) & 63u);
}

__global__ void degree_bins_kernel(const uint32_t *deg, uint32_t V, uint32_t *bins) {
    __shared__ uint32_t h[kDegreeBins];
    for (uint32_t j = threadIdx.x; j < kDegreeBins; j += blockDim.x) h[j] = 0;
    __syncthreads();
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x)
        atomicAdd(&h[degree_bin(deg[v])], 1u);
    __syncthreads();
    for (uint32_t j = threadIdx.x; j < kDegreeBins; j += blockDim.x)
        if (h[j]) atomicAdd(bins + j, h[j]);
}

__global__ void pull_flags_kernel(const uint32_t *off, const uint32_t *deg, uint32_t V, uint32_t hot_bin,
                                  uint32_t *has_edges, uint32_t *is_hot, uint32_t *hot_bits) {
    const uint32_t step = gridDim.x * blockDim.x;  // a multiple of 32: a warp's lanes hold a word's 32 vertices
    for (uint64_t v0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u; v0 < V; v0 += step) {
        const uint64_t v = v0 + (threadIdx.x & 31);
        const bool hot = v < V && degree_bin(deg[v]) >= hot_bin;
        if (v < V) {
            has_edges[v] = off[v + 1] != off[v];
            is_hot[v] = hot;
        }
        const unsigned bits = __ballot_sync(0xffffffffu, hot);
        if ((threadIdx.x & 31) == 0) hot_bits[v0 / 32] = bits;
    }
}

// rows and slots
__global__ void pull_rows_kernel(const uint32_t *has_edges, const uint32_t *row_pos, const uint32_t *is_hot,
                                 const uint32_t *slot_pos, const uint32_t *deg, uint32_t V, uint2 *rows,
                                 uint32_t *row_degree, uint32_t *hot_ids) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
        const bool hot = is_hot[v];
        const uint32_t slot = hot ? slot_pos[v] : ~0u;
        if (has_edges[v]) {
            rows[row_pos[v]] = make_uint2(v, slot);
            row_degree[row_pos[v]] = deg[v];
        }
        if (hot) hot_ids[slot] = v;
    }
}

// what an edge carries: its source, or its source's slot
__global__ void pull_words_kernel(const uint32_t *src, uint32_t E, const uint32_t *hot_bits, const uint32_t *slot_pos,
                                  uint32_t *edges) {
    const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < E; i += 8 * step) {
        uint32_t u[8], bits[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) u[q] = i + q * step < E ? __ldcs(src + i + q * step) : 0u;
#pragma unroll
        for (int q = 0; q < 8; ++q) bits[q] = __ldg(hot_bits + (u[q] >> 5));
#pragma unroll
        for (int q = 0; q < 8; ++q)
            if ((bits[q] >> (u[q] & 31)) & 1u) u[q] = __ldg(slot_pos + u[q]) | kPullHot;
#pragma unroll
        for (int q = 0; q < 8; ++q)
            if (i + q * step < E) __stcs(edges + i + q * step, u[q]);
    }
}

__global__ void pull_ends_kernel(const uint32_t *off, uint32_t V, uint32_t *edges) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x)
        if (off[v + 1] != off[v]) edges[off[v + 1] - 1] |= kPullLast;
}

// Unit t begins at the row that holds its edge (pull_unit_edge), or at that
// edge when the row is longer than span; such a row holds the first edge of
// the unit after the one it begins in, so its pieces are those of the units
// from pull_unit_of(its first edge) to pull_unit_of(its last).
__global__ void pull_units_kernel(const uint32_t *off, const uint32_t *row_pos, gbx_pull_layout l) {
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t <= l.n_units; t += gridDim.x * blockDim.x) {
        if (t == l.n_units) {
            l.units[t] = make_uint4(l.E, l.n_rows, ~0u, 0u);
            continue;
        }
        const uint32_t e = pull_unit_edge(l, t);
        uint32_t lo = 0, hi = l.V;  // the last v with off[v] <= e
        while (hi - lo > 1) {
            const uint32_t mid = lo + (hi - lo) / 2;
            if (off[mid] <= e) lo = mid; else hi = mid;
        }
        const uint32_t b = off[lo], end = off[lo + 1];
        const bool cut = end - b > l.span && e > b;
        const uint32_t first = pull_unit_of(l, b);
        l.units[t] = make_uint4(end - b > l.span ? e : b, row_pos[lo], cut ? first : ~0u,
                                cut ? pull_unit_of(l, end - 1) - first + 1 : 0u);
    }
}

// Below kLayoutEdges edges a sweep is a chain of latencies, and a launch per
// sweep of the row engine is shorter than this engine's with its grid barrier.
// Up to kLayoutLocalEdges that holds as well for graphs without long rows,
// which the row engine cuts into pieces and joins. 20 PageRank iterations, us,
// row engine / this one: R-MAT of 36k edges 118 / 175, 200k (longest row 4,254)
// 219 / 176, 400k 354 / 185, 4M 595 / 396; local graphs of 400k edges (longest
// row 224) 144 / 161, 4M (875) 402 / 419, 8M (1,250) 657 / 715, 16M (1,968)
// 1,020 / 944, 32M 2,307 / 1,864. A graph's first SpMV, us, with the row plan
// and a row sweep / with the layout and its sweep: R-MAT of 400k edges 255 / 193,
// 3M 295 / 199, 16M 409 / 287, 64M 775 / 676; crawl of 16M edges 335 / 278, 48M
// 516 / 520, 142M 1,030 / 1,084 (the second call: 661 / 452).
constexpr uint32_t kLayoutEdges = 65536;
constexpr uint32_t kLayoutLocalEdges = 12'000'000;
constexpr uint32_t kLayoutLongRow = 3072;

int build_layout(gbx_graph *g, cudaStream_t s, gbx_pull_layout *l) {
    const uint32_t V = g->V, E = g->E;
    const uint32_t *off = g->pull_offsets();
    l->V = V;
    l->E = E;
    const int grid = (int)std::min<uint64_t>((V + 255) / 256, (uint64_t)num_sms() * 8);
    DevBuf<uint32_t> bins, has, hot, hot_bits, row_pos, slot_pos, tot;
    GBX_TRY(bins.alloc(kDegreeBins, s));
    GBX_TRY(has.alloc(V, s));
    GBX_TRY(hot.alloc(V, s));
    GBX_TRY(row_pos.alloc(V, s));
    GBX_TRY(slot_pos.alloc(V, s));
    GBX_TRY(tot.alloc(2, s));
    GBX_TRY(hot_bits.alloc(ceil_div(V, 32), s));
    GBX_CUDA(cudaMemsetAsync(bins.p, 0, kDegreeBins * 4, s));
    degree_bins_kernel<<<std::min(grid, num_sms() * 2), 256, 0, s>>>(g->out_degree, V, bins.p);
    GBX_LAUNCH_CHECK();
    std::vector<uint32_t> count(kDegreeBins);
    GBX_CUDA(cudaMemcpyAsync(count.data(), bins.p, kDegreeBins * 4, cudaMemcpyDeviceToHost, s));
    GBX_CUDA(cudaStreamSynchronize(s));
    // A slot costs every SM a sixteenth of a cycle per sweep (64 bytes per
    // cycle from L2), a gather saved saves one SM one cycle: no more slots
    // than edges per SM.
    const uint32_t most = std::min<uint32_t>(kHotMax, E / (uint32_t)num_sms());
    uint32_t bin = kDegreeBins, slots = 0;
    while (bin > 1 && slots + count[bin - 1] <= most) slots += count[--bin];
    l->hot = (slots + 3) & ~3u;
    pull_flags_kernel<<<grid, 256, 0, s>>>(off, g->out_degree, V, bin, has.p, hot.p, hot_bits.p);
    GBX_LAUNCH_CHECK();
    GBX_TRY(exclusive_scan_u32(has.p, row_pos.p, V, s, tot.p));
    GBX_TRY(exclusive_scan_u32(hot.p, slot_pos.p, V, s, tot.p + 1));
    GBX_CUDA(cudaMemcpyAsync(&l->n_rows, tot.p, 4, cudaMemcpyDeviceToHost, s));
    GBX_CUDA(cudaStreamSynchronize(s));
    // An equal number of units for every warp of the GPU, of at most
    // kPullSpanMax edges; where that is more than one, the last quarter of the
    // edges in units a quarter as long, so that no warp waits a whole unit for
    // the last one.
    const uint64_t warps = (uint64_t)num_sms() * kPullWarps;
    const uint64_t per_warp = E / warps + 1;
    const uint64_t rounds = (per_warp + kPullSpanMax - 1) / kPullSpanMax;
    l->span = l->tail_span = (uint32_t)((per_warp / rounds + 127) / 128 * 128);
    if (rounds > 1) {
        l->big = (uint32_t)(warps * (rounds - 1 - rounds / 4));
        l->tail_span = (l->span / 4 + 127) / 128 * 128;
    }
    const uint64_t left = E - std::min<uint64_t>(E, (uint64_t)l->big * l->span);
    if (left == 0) l->big = 0, l->tail_span = l->span;
    l->n_units = l->big + (uint32_t)(((l->big ? left : E) + l->tail_span - 1) / l->tail_span);
    GBX_TRY(dev_alloc((void **)&l->edges, ((size_t)E + kPullPad) * 4, s));
    GBX_TRY(dev_alloc((void **)&l->hot_ids, (size_t)std::max(l->hot, 1u) * 4, s));
    GBX_TRY(dev_alloc((void **)&l->rows, (size_t)std::max(l->n_rows, 1u) * sizeof(uint2), s));
    GBX_TRY(dev_alloc((void **)&l->units, ((size_t)l->n_units + 1) * sizeof(uint4), s));
    GBX_TRY(dev_alloc((void **)&l->work, pull_work_words(*l) * 4, s));
    GBX_TRY(dev_alloc((void **)&l->row_degree, (size_t)std::max(l->n_rows, 1u) * 4, s));
    GBX_TRY(dev_alloc((void **)&l->sums, (size_t)l->n_units * 8, s));
    GBX_TRY(dev_alloc((void **)&l->tickets, (size_t)l->n_units * 4, s));
    GBX_CUDA(cudaMemsetAsync(l->tickets, 0, (size_t)l->n_units * 4, s));
    GBX_CUDA(cudaMemsetAsync(l->edges + E, 0, kPullPad * 4, s));
    if (l->hot) GBX_CUDA(cudaMemsetAsync(l->hot_ids, 0xFF, (size_t)l->hot * 4, s));
    pull_rows_kernel<<<grid, 256, 0, s>>>(has.p, row_pos.p, hot.p, slot_pos.p, g->out_degree, V, l->rows,
                                        l->row_degree, l->hot_ids);
    GBX_LAUNCH_CHECK();
    const int egrid = (int)std::min<uint64_t>((E + 2047ull) / 2048, (uint64_t)num_sms() * 8);
    pull_words_kernel<<<egrid, 256, 0, s>>>(g->pull_src(), E, hot_bits.p, slot_pos.p, l->edges);
    GBX_LAUNCH_CHECK();
    pull_ends_kernel<<<grid, 256, 0, s>>>(off, V, l->edges);
    GBX_LAUNCH_CHECK();
    pull_units_kernel<<<ceil_div(l->n_units + 1, 256), 256, 0, s>>>(off, row_pos.p, *l);
    GBX_LAUNCH_CHECK();
    GBX_CUDA(cudaStreamSynchronize(s));  // complete before any other stream or thread sees it
    return GBX_OK;
}

}  // namespace

int get_pull_layout(gbx_graph *g, cudaStream_t s, gbx_pull_layout **out) {
    *out = nullptr;
    if (g->E < kLayoutEdges || g->E > 0x7FFFFFFFu || g->V > kIdMask) return GBX_OK;
    const uint32_t longest = g->in_offsets ? g->max_in_degree : g->max_out_degree;
    if (g->E < kLayoutLocalEdges && longest < kLayoutLongRow) return GBX_OK;
    bool captured = false;
    GBX_TRY(is_capturing(s, &captured));
    std::lock_guard<std::mutex> lock(g->pull_layout_mutex);
    if (!g->pull_layout && !captured && g->pull_layout_tries < 2) {
        gbx_pull_layout *l = new gbx_pull_layout();
        const int st = build_layout(g, s, l);
        if (st == GBX_OK) {
            g->pull_layout = l;
        } else {
            cudaStreamSynchronize(s);
            gbx_free_pull_layout(l);
            if (st != GBX_ERR_NOMEM) return st;
            // no room for it: the row engine needs none
            clear_error();
            ++g->pull_layout_tries;
            return GBX_OK;
        }
    }
    *out = g->pull_layout;
    return GBX_OK;
}

}  // namespace gbx

void gbx_free_pull_layout(gbx_pull_layout *l) {
    if (!l) return;
    gbx::dev_free(l->edges);
    gbx::dev_free(l->hot_ids);
    gbx::dev_free(l->rows);
    gbx::dev_free(l->units);
    gbx::dev_free(l->work);
    gbx::dev_free(l->row_degree);
    gbx::dev_free(l->sums);
    gbx::dev_free(l->tickets);
    delete l;
}
