// SpMV pull (the reference's SPMVPullGraphCSR, SPMV.c:117-215):
// y[v] += sum over pull edges (u->v) of w_uv * x[u], repeated `iterations`
// times with y never reset. The hot-table engine (gbx_pull.cuh), with the hot
// vertices' x gathered once per call, or for small and some local graphs the
// row engine (gbx_gather.cuh) computes each row's sum and adds it to y.
#include <algorithm>

#include "gbx_pull.cuh"

namespace gbx {

struct SpmvTerm {
    const uint32_t *__restrict__ src;
    const float *__restrict__ val;  // may be null
    float dflt;
    const float *__restrict__ x;
    // index and value streams are read once: evict-first, keeping x in L2
    __device__ __forceinline__ uint32_t src_of(uint32_t e) const { return __ldcs(src + e); }
    __device__ __forceinline__ float value(uint32_t e, uint32_t u) const {
        float w = val ? __ldcs(val + e) : dflt;
        return __fmul_rn(w, __ldg(x + u));
    }
};

struct SpmvEpi {
    float *__restrict__ y;
    __device__ __forceinline__ void operator()(uint32_t v, float sum) { y[v] = __fadd_rn(y[v], sum); }
    __device__ __forceinline__ void block_finish() {}
};

// ---- hot-table engine -----------------------------------------------------------

struct SpmvHotTerm {
    const float *__restrict__ val;  // may be null
    float dflt;
    const float *cold;  // x
    bool wide;  // val starts on a 16-byte boundary
    struct Factors {
        float w[4];
    };
    __device__ __forceinline__ void factors(uint32_t e, uint32_t e0, uint32_t e1, Factors &f) const {
        if (!val) {  // (an edge outside the unit counts 0 * 0, also where dflt is not finite)
#pragma unroll
            for (int k = 0; k < 4; ++k) f.w[k] = e + k >= e0 && e + k < e1 ? dflt : 0.f;
        } else if (wide && e >= e0 && e + 4 <= e1) {
            const float4 w = __ldcs(reinterpret_cast<const float4 *>(val + e));
            f.w[0] = w.x, f.w[1] = w.y, f.w[2] = w.z, f.w[3] = w.w;
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) f.w[k] = e + k >= e0 && e + k < e1 ? __ldcs(val + e + k) : 0.f;
        }
    }
    __device__ __forceinline__ void scale(const Factors &f, float (&v)[4]) const {
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = __fmul_rn(f.w[k], v[k]);
    }
};

struct SpmvHotEpi {
    float *__restrict__ y;
    __device__ __forceinline__ void prefetch(uint32_t) const {}
    __device__ __forceinline__ void operator()(uint32_t, uint32_t v, uint32_t, float sum) const { y[v] = __fadd_rn(y[v], sum); }
};

__global__ void spmv_hot_values_kernel(const float *x, const uint32_t *hot_ids, uint32_t hot, uint32_t V, float *out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= hot) return;
    const uint32_t v = hot_ids[i];
    out[i] = v < V ? x[v] : 0.f;
}

__global__ void __launch_bounds__(kPullThreads, 1)
    spmv_hot_kernel(gbx_pull_layout layout, const float *hot_x, SpmvHotTerm term, SpmvHotEpi epi, PullPieces pieces,
                    unsigned *cursor) {
    extern __shared__ __align__(16) float s_hot[];
    PullSweep<SpmvHotTerm, SpmvHotEpi> sweep{layout, (uint32_t)__cvta_generic_to_shared(s_hot),
                                             s_hot + layout.hot + 4 + (threadIdx.x >> 5) * kPullBuf, term, epi, pieces};
    typename PullSweep<SpmvHotTerm, SpmvHotEpi>::Start first{};
    if (first_unit() < layout.n_units) first = sweep.start(first_unit());
    load_hot(hot_x, layout.hot, s_hot);
    deal_units(sweep, cursor, first);
}

// Working memory is the call's own, so that sweeps of one graph on several
// streams do not meet; a captured call's is the layout's. So is, where there
// is none to be had, that of a call that holds the graph's lock to its end.
static int spmv_run_hot(gbx_graph *g, const gbx_pull_layout &l, SpmvHotTerm term, float *y, uint32_t iterations,
                        cudaStream_t s) {
    bool captured = false;
    GBX_TRY(is_capturing(s, &captured));
    DevBuf<float> own;
    std::unique_lock<std::mutex> lent(g->pull_layout_mutex, std::defer_lock);
    if (!captured && own.alloc(pull_work_words(l), s) != GBX_OK) {
        clear_error();
        lent.lock();
    }
    float *const hot_x = own.p ? own.p : l.work, *const sums = hot_x + std::max(l.hot, 4u);
    unsigned *const tickets = reinterpret_cast<unsigned *>(sums + 2 * (size_t)l.n_units);
    unsigned *const cursors = tickets + l.n_units;
    GBX_CUDA(cudaMemsetAsync(tickets, 0, ((size_t)l.n_units + kPullCursors) * sizeof(unsigned), s));
    if (l.hot) {
        spmv_hot_values_kernel<<<ceil_div(l.hot, 256), 256, 0, s>>>(term.cold, l.hot_ids, l.hot, l.V, hot_x);
        GBX_LAUNCH_CHECK();
    }
    const size_t smem = pull_smem(l);
    GBX_CUDA(cudaFuncSetAttribute(spmv_hot_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPullSmemLimit));
    const unsigned ctas = std::min<unsigned>((unsigned)num_sms(), ceil_div(l.n_units, kPullWarps));
    for (uint32_t it = 0; it < iterations; ++it) {
        const uint32_t at = it % kPullCursors;
        if (it && at == 0) GBX_CUDA(cudaMemsetAsync(cursors, 0, kPullCursors * sizeof(unsigned), s));
        spmv_hot_kernel<<<ctas, kPullThreads, smem, s>>>(l, hot_x, term, SpmvHotEpi{y}, PullPieces{sums, tickets},
                                                         cursors + at);
        GBX_LAUNCH_CHECK();
    }
    if (lent.owns_lock()) GBX_CUDA(cudaStreamSynchronize(s));
    return GBX_OK;
}

}  // namespace gbx

using namespace gbx;

extern "C" int gbx_spmv(gbx_graph *g, const float *values, float default_value, const float *x,
                        float *y, uint32_t iterations, void *stream) {
    clear_error();
    GBX_REQUIRE(g && x && y, GBX_ERR_INVALID, "graph, x or y is NULL");
    GBX_TRY(ensure_device());
    cudaStream_t s = (cudaStream_t)stream;
    const uint32_t V = g->V;
    gbx_pull_layout *layout = nullptr;
    if (iterations) GBX_TRY(get_pull_layout(g, s, &layout));
    gbx_gather_plan *plan = nullptr;
    if (!layout) GBX_TRY(get_pull_plan(g, s, &plan));
    InArray<float> xin, vin;
    GBX_TRY(xin.bind(x, V, s));
    const float *vals = nullptr;
    if (values) {
        GBX_TRY(vin.bind(values, g->E, s));
        vals = vin.d;
    } else {
        vals = g->pull_weight();
    }
    // y is read and written: stage host y in and out
    OutArray<float> yout;
    GBX_TRY(yout.bind(y, V, s));
    if (yout.to_host()) GBX_CUDA(cudaMemcpyAsync(yout.d, y, (size_t)V * 4, cudaMemcpyHostToDevice, s));
    if (layout) {
        const bool wide = ((uintptr_t)vals & 15u) == 0;
        GBX_TRY(spmv_run_hot(g, *layout, SpmvHotTerm{vals, default_value, xin.d, wide}, yout.d, iterations, s));
    } else {
        SpmvTerm term{g->pull_src(), vals, default_value, xin.d};
        SpmvEpi epi{yout.d};
        for (uint32_t it = 0; it < iterations; ++it)
            GBX_TRY(launch_gather(g->pull_offsets(), V, *plan, term, epi, s));
    }
    GBX_TRY(yout.finish(s));
    if (yout.to_host()) GBX_CUDA(cudaStreamSynchronize(s));
    return GBX_OK;
}
