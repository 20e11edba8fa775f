// Pull PageRank (the reference's pageRankPullGraphCSR, pageRank.c:245-368).
//
// Per iteration: for every vertex v a pull engine sums contrib[u] over v's
// in-edges, and the epilogue computes
//   next = base_pr + damp * sum           (base_pr = 1 - 0.85f, damp = 0.85f)
//   contrib_next[v] = next / outdeg(v)    (0 for dangling vertices)
//   |next - prev| -> FP64 error sum, active count (>= epsilon)
// so the reference's three V-sized passes (contrib, gather, update) become
// one sweep. Ranks and contributions ping-pong between two buffers. An
// iteration that follows one with no active vertex is not run, which
// reproduces the reference's early exit (stats->iterations = the index of the
// iteration with no active vertex). A final kernel divides by N (:344-350).
//
// The sweeps run on the hot-table engine (gbx_pull.cuh) in one persistent
// kernel, one CTA per SM: each iteration loads the hot sources' contributions
// into shared memory, deals the edge units and ends at a grid barrier. Those
// of small and some local graphs run as one launch each on the row engine
// (gbx_gather.cuh), which needs no layout; that loop (state reset, initial
// ranks, the iterations) is captured once per graph and (max_iterations,
// epsilon) as a CUDA graph and replayed by every later call. With epsilon = 0 no iteration's residual but the last is asked for,
// so ranks are written in the last two only; a row's epilogue is its degree
// and one contribution.
#include <algorithm>

#include "gbx_pull.cuh"

namespace gbx {

struct PrIterState {
    double err;
    unsigned active;
    unsigned cursor;  // next unit of the hot-table engine
};

struct PrTerm {
    const uint32_t *__restrict__ src;
    const float *__restrict__ contrib;
    // the in-edge stream is read once per iteration: evict-first, so it does
    // not push the gathered contributions out of L2
    __device__ __forceinline__ uint32_t src_of(uint32_t e) const { return __ldcs(src + e); }
    __device__ __forceinline__ float value(uint32_t, uint32_t u) const { return __ldg(contrib + u); }
};

struct PrEpi {
    const float *__restrict__ r_cur;
    float *__restrict__ r_next;
    float *__restrict__ contrib_next;
    const uint32_t *__restrict__ out_degree;
    PrIterState *state;  // this iteration's slot
    double epsilon;
    double inv_n;
    double err;
    unsigned active;
    bool reduce;  // accumulate the residual and the active count this iteration
    __device__ __forceinline__ void operator()(uint32_t v, float sum) {
        const float damp = 0.85f;
        const float base = 1.0f - 0.85f;
        float next = __fadd_rn(base, __fmul_rn(damp, sum));
        float prev = r_cur[v];
        r_next[v] = next;
        uint32_t d = out_degree[v];
        contrib_next[v] = d ? __fdiv_rn(next, (float)d) : 0.0f;
        if (reduce) {
            double e = (double)fabsf(__fsub_rn(next, prev));
            err += e * inv_n;
            active += (e >= epsilon) ? 1u : 0u;
        }
    }
    __device__ __forceinline__ void block_finish() {
        if (!reduce) return;
        __shared__ double sd[32];
        __shared__ unsigned su[32];
        double te = block_sum(err, sd);
        unsigned ta = block_sum(active, su);
        if (threadIdx.x == 0) {
            if (te != 0.0) atomicAdd(&state->err, te);
            if (ta) atomicAdd(&state->active, ta);
        }
    }
};

__global__ void pr_init_kernel(float *r, float *contrib, const uint32_t *out_degree, uint32_t V) {
    const float base = 1.0f - 0.85f;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
        r[v] = base;
        uint32_t d = out_degree[v];
        contrib[v] = d ? __fdiv_rn(base, (float)d) : 0.0f;
    }
}

// Iteration `it`: skip when the previous iteration converged.
template <class Term, class Epi>
__global__ void __launch_bounds__(kGatherThreads, kGatherBlocksPerSM)
    pr_iteration_kernel(const uint32_t *__restrict__ off, uint32_t V, gbx_gather_plan plan,
                        GatherGeometry geo, Term term, Epi epi, const PrIterState *prev) {
    if (prev && prev->active == 0) return;
    gather_rows_kernel_body(off, V, plan, geo, term, epi);
}

// final ranks: pick the buffer holding the last executed iteration
__global__ void pr_finish_kernel(const float *r0, const float *r1, const PrIterState *st,
                                 uint32_t max_it, uint32_t can_stop, uint32_t V, float *out, uint32_t *iters_out,
                                 gbx_pr_result *res_dev) {
    __shared__ uint32_t s_k;
    if (threadIdx.x == 0) {
        uint32_t k = max_it;
        for (uint32_t i = 0; can_stop && i < max_it; ++i)
            if (st[i].active == 0) { k = i; break; }
        s_k = k;
    }
    __syncthreads();
    uint32_t k = s_k;
    uint32_t executed = k < max_it ? k + 1 : max_it;
    const float *r = (executed & 1u) ? r1 : r0;
    const float nf = (float)V;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x)
        out[v] = __fdiv_rn(r[v], nf);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        res_dev->iterations = k;
        uint32_t last = executed ? executed - 1 : 0;
        res_dev->active_last = executed ? (can_stop ? st[last].active : V) : 0;
        res_dev->error_total = executed ? st[last].err : 0.0;
        if (iters_out) *iters_out = k;
    }
}

// Enqueue the row engine's loop: state reset, initial ranks, max_it iterations.
static int pr_enqueue_loop(gbx_graph *g, const gbx_gather_plan &plan, uint32_t max_it, double epsilon, float *rbuf,
                           float *cbuf, PrIterState *st, cudaStream_t s, uint32_t *kernels) {
    const uint32_t V = g->V;
    float *r[2] = {rbuf, rbuf + V};
    float *c[2] = {cbuf, cbuf + V};
    GBX_CUDA(cudaMemsetAsync(st, 0, sizeof(PrIterState) * (max_it ? max_it : 1), s));
    const int grid = (int)std::min<uint64_t>((V + 255) / 256, (uint64_t)num_sms() * 8);
    pr_init_kernel<<<grid, 256, 0, s>>>(r[0], c[0], g->out_degree, V);
    GBX_LAUNCH_CHECK();
    const GatherGeometry geo = gather_geometry(plan);
    const double inv_n = 1.0 / (double)V;
    for (uint32_t it = 0; it < max_it; ++it) {
        const int a = it & 1, b = a ^ 1;
        PrTerm term{g->pull_src(), c[a]};
        // with epsilon = 0 every vertex stays active, so only the last
        // iteration's residual (reported as error_total) is reduced
        const bool reduce = epsilon > 0.0 || it + 1 == max_it;
        PrEpi epi{r[a], r[b], c[b], g->out_degree, st + it, epsilon, inv_n, 0.0, 0u, reduce};
        pr_iteration_kernel<PrTerm, PrEpi><<<gather_grid(geo), kGatherThreads, 0, s>>>(
            g->pull_offsets(), V, plan, geo, term, epi, (it && epsilon > 0.0) ? st + it - 1 : nullptr);
        GBX_LAUNCH_CHECK();
    }
    *kernels = 1 + max_it;
    return GBX_OK;
}

// ---- hot-table engine -----------------------------------------------------------

// Contributions: slots first, then one entry per vertex (used by those
// without a slot). Other SMs wrote them in the previous iteration, so they are
// not read through the read-only path; the grid barrier's acquire drops what
// L1 holds of them.
struct PrHotTerm {
    const float *cold;
    struct Factors {};
    __device__ __forceinline__ void factors(uint32_t, uint32_t, uint32_t, Factors &) const {}
    __device__ __forceinline__ void scale(const Factors &, float (&)[4]) const {}
};

struct PrHotEpi {
    const float *r_cur;
    float *r_next;
    float *c_next;  // slots, then vertices
    uint32_t hot;
    const uint32_t *__restrict__ row_degree;  // out-degrees in row order
    double epsilon, inv_n;
    double err;
    unsigned active;
    bool write, reduce;
    __device__ __forceinline__ void prefetch(uint32_t row) const {
        asm volatile("prefetch.global.L1 [%0];" ::"l"(row_degree + row));
    }
    __device__ __forceinline__ void operator()(uint32_t row, uint32_t v, uint32_t slot, float sum) {
        const float next = __fadd_rn(1.0f - 0.85f, __fmul_rn(0.85f, sum));
        const uint32_t d = __ldg(row_degree + row);
        // dangling: nobody reads it, and it stays 0 where a graph without an
        // inverse lists such a vertex as a source
        if (d) c_next[slot != ~0u ? slot : hot + v] = __fdiv_rn(next, (float)d);
        if (write) {
            if (reduce) {
                const double e = (double)fabsf(__fsub_rn(next, r_cur[v]));
                err += e * inv_n;
                active += (e >= epsilon) ? 1u : 0u;
            }
            r_next[v] = next;
        }
    }
};

// floats per contribution buffer: the slots of both start on 16 bytes
__host__ __device__ inline size_t contrib_stride(uint32_t V, uint32_t hot) { return ((size_t)V + hot + 3) & ~(size_t)3; }

// both buffers of ranks and contributions at the first iteration's values
// (rows without in-edges keep them)
__global__ void pr_hot_init_kernel(float *r, float *c, const uint32_t *out_degree, uint32_t V, uint32_t hot,
                                   const uint32_t *hot_ids) {
    const float base = 1.0f - 0.85f;
    const uint32_t n = hot + V;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t v = i < hot ? hot_ids[i] : i - hot;
        const uint32_t d = v < V ? out_degree[v] : 0u;
        const float x = d ? __fdiv_rn(base, (float)d) : 0.0f;
        c[i] = x;
        c[i + contrib_stride(V, hot)] = x;
        if (i >= hot) {
            r[v] = base;
            r[v + V] = base;
        }
    }
}

struct PrHotArgs {
    gbx_pull_layout layout;
    float *r, *c;
    const uint32_t *row_degree;
    PrIterState *state;
    PullPieces pieces;
    GridSync *sync;
    uint32_t max_it;
    double epsilon;
};

__global__ void __launch_bounds__(kPullThreads, 1) pr_hot_kernel(PrHotArgs a) {
    extern __shared__ __align__(16) float s_hot[];
    __shared__ double sd[32];
    __shared__ unsigned su[32];
    const uint32_t V = a.layout.V, hot = a.layout.hot;
    const size_t stride = contrib_stride(V, hot);
    float *buf = s_hot + hot + 4 + (threadIdx.x >> 5) * kPullBuf;
    grid_barrier_init();
    for (uint32_t it = 0; it < a.max_it; ++it) {
        const uint32_t p = it & 1, q = p ^ 1;
        PrHotTerm term{a.c + p * stride + hot};
        // with epsilon = 0 every vertex stays active: only the last
        // iteration's residual (reported as error_total) is reduced
        const bool reduce = a.epsilon > 0.0 || it + 1 == a.max_it;
        const bool write = reduce || it + 2 == a.max_it;
        PrHotEpi epi{a.r + (size_t)p * V, a.r + (size_t)q * V, a.c + q * stride, hot, a.row_degree, a.epsilon,
                     1.0 / (double)V, 0.0, 0u, write, reduce};
        PullSweep<PrHotTerm, PrHotEpi> sweep{a.layout, (uint32_t)__cvta_generic_to_shared(s_hot), buf, term, epi,
                                               a.pieces};
        // the first unit's words do not wait for the slots
        typename PullSweep<PrHotTerm, PrHotEpi>::Start first{};
        if (first_unit() < a.layout.n_units) first = sweep.start(first_unit());
        load_hot(a.c + p * stride, hot, s_hot);
        deal_units(sweep, &a.state[it].cursor, first);
        if (reduce) {
            const double te = block_sum(epi.err, sd);
            const unsigned ta = block_sum(epi.active, su);
            if (threadIdx.x == 0) {
                if (te != 0.0) atomicAdd(&a.state[it].err, te);
                if (ta) atomicAdd(&a.state[it].active, ta);
            }
        }
        if (it + 1 == a.max_it) break;
        if (!grid_barrier(a.sync)) return;
        if (a.epsilon > 0.0 && __ldcg(&a.state[it].active) == 0) break;
    }
}

}  // namespace gbx

// Per-graph PageRank working memory and the row engine's captured loop
// (re-captured when max_iterations, epsilon or its buffers change). Calls on
// one graph object are serialised by the caller, as for every other entry point.
struct gbx_pr_cache {
    float *rbuf = nullptr;   // 2V: ping-pong ranks
    float *cbuf = nullptr;   // ping-pong contributions, 2V or 2 (slots + V)
    size_t cbuf_n = 0;
    // the result and the grid barrier's words, then one state per iteration
    struct Tail {
        gbx_pr_result res;
        gbx::GridSync sync;
    } *tail = nullptr;
    gbx::PrIterState *st = nullptr;  // behind *tail
    uint32_t cap = 0;                // states
    cudaStream_t cap_stream = nullptr;
    cudaGraphExec_t exec = nullptr;
    uint32_t key_it = 0, kernels = 0;
    double key_eps = -1.0;
    void drop_capture() {
        if (exec) cudaGraphExecDestroy(exec);
        exec = nullptr;
    }
};
static_assert(sizeof(gbx_pr_cache::Tail) % alignof(gbx::PrIterState) == 0, "states follow on their alignment");

void gbx_free_pr_cache(gbx_pr_cache *c) {
    if (!c) return;
    c->drop_capture();
    if (c->cap_stream) cudaStreamDestroy(c->cap_stream);
    cudaFree(c->rbuf);
    cudaFree(c->cbuf);
    cudaFree(c->tail);
    delete c;
}

using namespace gbx;

namespace {

int pr_cache(gbx_graph *g, const gbx_pull_layout *l, uint32_t max_it, gbx_pr_cache **out) {
    gbx_pr_cache *c = g->pr_cache;
    if (!c) c = g->pr_cache = new gbx_pr_cache();
    const size_t need = 2 * contrib_stride(g->V, l ? l->hot : 0);
    if (!c->rbuf) GBX_CUDA(cudaMalloc(&c->rbuf, sizeof(float) * 2 * (size_t)g->V));
    if (c->cbuf_n < need) {
        c->drop_capture();
        cudaFree(c->cbuf);
        c->cbuf = nullptr;
        c->cbuf_n = 0;
        GBX_CUDA(cudaMalloc(&c->cbuf, sizeof(float) * need));
        c->cbuf_n = need;
    }
    if (c->cap < std::max(max_it, 1u)) {
        c->drop_capture();
        cudaFree(c->tail);
        c->tail = nullptr;
        c->cap = 0;
        const uint32_t cap = std::max(max_it, 64u);
        GBX_CUDA(cudaMalloc(&c->tail, sizeof(*c->tail) + sizeof(PrIterState) * cap));
        c->st = reinterpret_cast<PrIterState *>(c->tail + 1);
        c->cap = cap;
    }
    if (!l && !c->cap_stream) GBX_CUDA(cudaStreamCreateWithFlags(&c->cap_stream, cudaStreamNonBlocking));
    *out = c;
    return GBX_OK;
}

// (Re)capture the row engine's loop on the cache's own stream.
int pr_capture(gbx_graph *g, const gbx_gather_plan &plan, uint32_t max_it, double epsilon, gbx_pr_cache *c) {
    if (c->exec && c->key_it == max_it && c->key_eps == epsilon) return GBX_OK;
    c->drop_capture();
    GBX_CUDA(cudaStreamBeginCapture(c->cap_stream, cudaStreamCaptureModeThreadLocal));
    uint32_t kernels = 0;
    const int st = pr_enqueue_loop(g, plan, max_it, epsilon, c->rbuf, c->cbuf, c->st, c->cap_stream, &kernels);
    cudaGraph_t graph = nullptr;
    const cudaError_t e = cudaStreamEndCapture(c->cap_stream, &graph);
    if (st != GBX_OK) {
        if (graph) cudaGraphDestroy(graph);
        return st;
    }
    GBX_CUDA(e);
    const cudaError_t ei = cudaGraphInstantiate(&c->exec, graph, 0);
    cudaGraphDestroy(graph);
    GBX_CUDA(ei);
    c->key_it = max_it;
    c->key_eps = epsilon;
    c->kernels = kernels;
    return GBX_OK;
}

// the persistent kernel over the hot-table layout
int pr_run_hot(gbx_graph *g, const gbx_pull_layout &l, uint32_t max_it, double epsilon, gbx_pr_cache *c,
               cudaStream_t s) {
    const uint32_t V = g->V;
    GBX_CUDA(cudaMemsetAsync(c->tail, 0, sizeof(*c->tail) + sizeof(PrIterState) * max_it, s));
    const int grid = (int)std::min<uint64_t>((V + l.hot + 255ull) / 256, (uint64_t)num_sms() * 8);
    pr_hot_init_kernel<<<grid, 256, 0, s>>>(c->rbuf, c->cbuf, g->out_degree, V, l.hot, l.hot_ids);
    GBX_LAUNCH_CHECK();
    PrHotArgs a{l, c->rbuf, c->cbuf, l.row_degree, c->st, {l.sums, l.tickets}, &c->tail->sync, max_it, epsilon};
    const size_t smem = pull_smem(l);
    GBX_CUDA(cudaFuncSetAttribute(pr_hot_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPullSmemLimit));
    // a CTA per SM, fewer where there is less than a unit per warp
    const unsigned ctas = std::min<unsigned>((unsigned)num_sms(), ceil_div(l.n_units, kPullWarps));
    void *args[] = {&a};
    GBX_CUDA(cudaLaunchCooperativeKernel((const void *)pr_hot_kernel, dim3(ctas), dim3(kPullThreads), args, smem, s));
    GBX_LAUNCH_CHECK();
    return GBX_OK;
}

}  // namespace

int gbx::pagerank_pull(gbx_graph *g, uint32_t max_iterations, double epsilon, float *ranks, gbx_pr_result *result,
                       cudaStream_t s, bool by_rows) {
    const uint32_t V = g->V;
    gbx_pull_layout *layout = nullptr;
    if (max_iterations && !by_rows) GBX_TRY(get_pull_layout(g, s, &layout));
    gbx_gather_plan *plan = nullptr;
    if (!layout) GBX_TRY(get_pull_plan(g, s, &plan));
    OutArray<float> out;
    GBX_TRY(out.bind(ranks, V, s));
    gbx_pr_cache *c = nullptr;
    GBX_TRY(pr_cache(g, layout, max_iterations, &c));
    if (layout) {
        GBX_TRY(pr_run_hot(g, *layout, max_iterations, epsilon, c, s));
    } else {
        GBX_TRY(pr_capture(g, *plan, max_iterations, epsilon, c));
        GBX_CUDA(cudaGraphLaunch(c->exec, s));
        for (uint32_t k = 0; k < c->kernels; ++k) note_launch();
    }
    const int grid = (int)std::min<uint64_t>((V + 255) / 256, (uint64_t)num_sms() * 8);
    pr_finish_kernel<<<grid, 256, 0, s>>>(c->rbuf, c->rbuf + V, c->st, max_iterations, epsilon > 0.0 ? 1u : 0u, V,
                                          out.d, nullptr, &c->tail->res);
    GBX_LAUNCH_CHECK();
    GBX_TRY(out.finish(s));
    gbx_pr_cache::Tail h;
    GBX_CUDA(cudaMemcpyAsync(&h, c->tail, sizeof(h), cudaMemcpyDeviceToHost, s));
    GBX_CUDA(cudaStreamSynchronize(s));
    if (layout && h.sync.error) {
        GBX_CUDA(cudaMemset(layout->tickets, 0, sizeof(unsigned) * (size_t)layout->n_units));  // a sweep was left half done
        GBX_REQUIRE(false, GBX_ERR_DEVICE_TIMEOUT, "PageRank: a grid barrier wait ran out");
    }
    if (result) *result = h.res;
    return GBX_OK;
}

extern "C" int gbx_pagerank_pull(gbx_graph *g, uint32_t max_iterations, double epsilon,
                                 float *ranks, gbx_pr_result *result, void *stream) {
    clear_error();
    GBX_REQUIRE(g && ranks, GBX_ERR_INVALID, "graph or ranks is NULL");
    GBX_REQUIRE(epsilon >= 0.0, GBX_ERR_INVALID, "epsilon must be >= 0");
    GBX_TRY(ensure_device());
    return pagerank_pull(g, max_iterations, epsilon, ranks, result, (cudaStream_t)stream, false);
}
