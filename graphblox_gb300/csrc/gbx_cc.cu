// Connected components (the reference's connectedComponentsGraphCSR,
// connectedComponents.c:268-629). Every variant hooks roots high->low only
// and compresses fully, so components[v] is the smallest vertex id of v's
// component -- identical labels to the reference for all three variants.
//
//  1 Afforest (default, :379-535): two neighbour rounds linking v with its
//    r-th neighbour, compress, count 1024 sampled vertices' labels in one CTA,
//    then link the remaining edges of every vertex outside the most frequent
//    one's component (plus all in-edges when the inverse CSR is present, as
//    the DIRECTED build does). RMAT-22, 128M edges: 571 -> 148 us, of which
//    the two rounds take 90 (a random sector per vertex and the claims).
//  0 Shiloach-Vishkin sweeps (:293-377): hook on roots, compress, repeat.
//  2 label propagation (:537-629): atomicMin both ways until stable.
#include <algorithm>

#include "gbx_internal.cuh"

namespace gbx {

__device__ __forceinline__ uint32_t ld_volatile(const uint32_t *p) {
    return *(const volatile uint32_t *)p;
}

// linkNodes (connectedComponents.c:177-196). The first two reads may come from
// L1: what it holds of a label is an earlier one, an ancestor of the vertex
// all the same, and once most vertices hang under one root every read of its
// label through L2 would queue at the same line. Those that decide go past L1.
__device__ __forceinline__ void cc_link(uint32_t u, uint32_t v, uint32_t *comp) {
    uint32_t p1 = comp[u];
    uint32_t p2 = comp[v];
    for (int guard = 0; p1 != p2 && guard < (1 << 20); ++guard) {
        uint32_t high = p1 > p2 ? p1 : p2;
        uint32_t low = p1 + (p2 - high);
        uint32_t phigh = ld_volatile(comp + high);
        if (phigh == low) break;
        if (phigh == high && atomicCAS(comp + high, high, low) == high) break;
        p1 = ld_volatile(comp + ld_volatile(comp + high));
        p2 = ld_volatile(comp + low);
    }
}

__global__ void cc_init_kernel(uint32_t *comp, uint32_t V) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x)
        comp[v] = v;
}

// compressNodes (connectedComponents.c:199-210). Through L1 (an older label is
// an ancestor too, and a root's label does not change here); four vertices per
// thread. RMAT-22: 55 us with reads of the one hot label past L1.
__global__ void cc_compress_kernel(uint32_t *comp, uint32_t V) {
    const uint32_t step = gridDim.x * blockDim.x;
    for (uint64_t v0 = blockIdx.x * blockDim.x + threadIdx.x; v0 < V; v0 += 4ull * step) {
        uint32_t c[4], up[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) c[q] = v0 + (uint64_t)q * step < V ? comp[v0 + (uint64_t)q * step] : 0u;
#pragma unroll
        for (int q = 0; q < 4; ++q) up[q] = comp[c[q]];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint64_t v = v0 + (uint64_t)q * step;
            if (v >= V || c[q] == up[q]) continue;
            do {
                c[q] = up[q];
                up[q] = comp[c[q]];
            } while (c[q] != up[q]);
            comp[v] = c[q];
        }
    }
}

__global__ void cc_neighbor_round_kernel(const uint32_t *off, const uint32_t *dest, uint32_t *comp,
                                         uint32_t V, uint32_t r) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
        uint32_t b = off[v], e = off[v + 1];
        if (b + r < e) cc_link(v, dest[b + r], comp);
    }
}

// The most frequent label among `ns` sampled vertices (of equally frequent
// ones the smallest): a count per label in a shared-memory hash table, one
// addition per distinct label of a warp (5 us; sorting them and one thread
// scanning the runs took 40).
__global__ void __launch_bounds__(1024) cc_sample_kernel(const uint32_t *comp, uint32_t V, uint32_t ns,
                                                         uint64_t seed, uint32_t *out) {
    constexpr uint32_t kSlots = 2048;
    __shared__ uint32_t key[kSlots], count[kSlots];
    __shared__ unsigned long long best;
    const uint32_t t = threadIdx.x;
    key[t] = key[t + 1024] = 0xFFFFFFFFu;
    count[t] = count[t + 1024] = 0;
    if (t == 0) best = 0;
    uint64_t x = seed + 0x9E3779B97F4A7C15ull * (t + 1);
    x ^= x >> 30; x *= 0xBF58476D1CE4E5B9ull; x ^= x >> 27; x *= 0x94D049BB133111EBull; x ^= x >> 31;
    const uint32_t mine = t < ns ? comp[(uint32_t)(x % V)] : 0xFFFFFFFFu;
    __syncthreads();
    const unsigned peers = __match_any_sync(0xffffffffu, mine);
    if (mine != 0xFFFFFFFFu && (t & 31) == (uint32_t)__ffs(peers) - 1) {
        uint32_t at = (mine * 2654435761u) >> 21;
        for (;;) {  // at most 1024 labels in 2048 slots: a free one is met
            const uint32_t held = atomicCAS(key + at, 0xFFFFFFFFu, mine);
            if (held == 0xFFFFFFFFu || held == mine) break;
            at = (at + 1) & (kSlots - 1);
        }
        atomicAdd(count + at, (uint32_t)__popc(peers));
    }
    __syncthreads();
    for (uint32_t i = t; i < kSlots; i += 1024)
        if (count[i]) atomicMax(&best, ((unsigned long long)count[i] << 32) | (0xFFFFFFFFu - key[i]));
    __syncthreads();
    if (t == 0) *out = 0xFFFFFFFFu - (uint32_t)best;
}

// Afforest final link over edges from index `skip_first`: a warp looks at 32
// vertices at once and takes the rows of those outside the skipped component
// one after the other, so the many inside it cost one coalesced read
// (RMAT-22: 16 us; a warp per vertex, one label read after the other: 245).
__global__ void cc_final_link_kernel(const uint32_t *off, const uint32_t *dest, const uint32_t *ioff,
                                     const uint32_t *isrc, uint32_t *comp, uint32_t V,
                                     uint32_t skip_first, const uint32_t *skip_label) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t skip = *skip_label;
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5, groups = (V + 31) / 32;
    for (uint32_t gr = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; gr < groups; gr += nw) {
        const uint32_t v = gr * 32 + lane;
        const bool out = v < V && ld_volatile(comp + v) != skip;
        uint32_t b = 0, e = 0, ib = 0, ie = 0;
        if (out) {
            b = off[v] + skip_first;
            e = off[v + 1];
            if (ioff) {
                ib = ioff[v];
                ie = ioff[v + 1];
            }
        }
        unsigned rows = __ballot_sync(0xffffffffu, b < e || ib < ie);
        while (rows) {
            const int k = __ffs(rows) - 1;
            rows &= rows - 1;
            const uint32_t u = gr * 32 + k;
            const uint32_t rb = __shfl_sync(0xffffffffu, b, k), re = __shfl_sync(0xffffffffu, e, k);
            for (uint32_t j = rb + lane; j < re; j += 32) cc_link(u, dest[j], comp);
            if (ioff) {
                const uint32_t jb = __shfl_sync(0xffffffffu, ib, k), je = __shfl_sync(0xffffffffu, ie, k);
                for (uint32_t j = jb + lane; j < je; j += 32) cc_link(u, isrc[j], comp);
            }
        }
    }
}

// Shiloach-Vishkin hooking sweep: hook the higher root under the lower one
__global__ void cc_sv_hook_kernel(const uint32_t *off, const uint32_t *dest, uint32_t *comp,
                                  uint32_t V, unsigned *change) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    bool changed = false;
    for (uint32_t v = gw; v < V; v += nw) {
        uint32_t b = off[v], e = off[v + 1];
        for (uint32_t j = b + lane; j < e; j += 32) {
            uint32_t u = dest[j];
            uint32_t cs = ld_volatile(comp + v), cd = ld_volatile(comp + u);
            if (cs == cd) continue;
            uint32_t high = cs > cd ? cs : cd, low = cs + (cd - high);
            if (ld_volatile(comp + high) == high && atomicCAS(comp + high, high, low) == high)
                changed = true;
        }
    }
    if (__any_sync(0xffffffffu, changed) && lane == 0) atomicOr(change, 1u);
}

// label propagation: min label across every edge, both directions
__global__ void cc_lp_kernel(const uint32_t *off, const uint32_t *dest, uint32_t *comp, uint32_t V,
                             unsigned *change) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    bool changed = false;
    for (uint32_t v = gw; v < V; v += nw) {
        uint32_t b = off[v], e = off[v + 1];
        for (uint32_t j = b + lane; j < e; j += 32) {
            uint32_t u = dest[j];
            uint32_t cv = ld_volatile(comp + v), cu = ld_volatile(comp + u);
            if (cv < cu) changed |= atomicMin(comp + u, cv) > cv;
            else if (cu < cv) changed |= atomicMin(comp + v, cu) > cu;
        }
    }
    if (__any_sync(0xffffffffu, changed) && lane == 0) atomicOr(change, 1u);
}

}  // namespace gbx

using namespace gbx;

extern "C" int gbx_cc(gbx_graph *g, int variant, uint32_t *components, uint32_t *iterations,
                      void *stream) {
    clear_error();
    GBX_REQUIRE(g && components, GBX_ERR_INVALID, "graph or components is NULL");
    GBX_REQUIRE(variant >= 0 && variant <= 2, GBX_ERR_INVALID, "variant must be 0, 1 or 2");
    GBX_TRY(ensure_device());
    cudaStream_t s = (cudaStream_t)stream;
    const uint32_t V = g->V;
    OutArray<uint32_t> out;
    GBX_TRY(out.bind(components, V, s));
    uint32_t *comp = out.d;
    const unsigned grid = std::min<unsigned>(ceil_div(V, 256), (unsigned)num_sms() * 8);
    const unsigned wgrid = std::min<unsigned>(ceil_div((uint64_t)V * 32, 256), (unsigned)num_sms() * 16);
    cc_init_kernel<<<grid, 256, 0, s>>>(comp, V);
    GBX_LAUNCH_CHECK();
    uint32_t iters = 0;
    DevBuf<unsigned> flag;
    GBX_TRY(flag.alloc(2, s));
    if (variant == 1) {
        const uint32_t rounds = 2;
        for (uint32_t r = 0; r < rounds; ++r) {
            cc_neighbor_round_kernel<<<grid, 256, 0, s>>>(g->offsets, g->dest, comp, V, r);
            GBX_LAUNCH_CHECK();
            cc_compress_kernel<<<grid, 256, 0, s>>>(comp, V);
            GBX_LAUNCH_CHECK();
        }
        uint32_t ns = V < 1024 ? V / 2 : 1024;
        if (ns == 0) ns = 1;
        cc_sample_kernel<<<1, 1024, 0, s>>>(comp, V, ns, 27491095ull, flag.p);
        GBX_LAUNCH_CHECK();
        cc_final_link_kernel<<<wgrid, 256, 0, s>>>(g->offsets, g->dest, g->in_offsets, g->in_src,
                                                   comp, V, rounds, flag.p);
        GBX_LAUNCH_CHECK();
        cc_compress_kernel<<<grid, 256, 0, s>>>(comp, V);
        GBX_LAUNCH_CHECK();
        iters = rounds;
    } else {
        const uint32_t cap = V + 2;  // each sweep merges at least one pair of trees
        unsigned h = 1;
        while (h) {
            GBX_REQUIRE(iters < cap, GBX_ERR_ITER_CAP, "CC sweep cap reached");
            GBX_CUDA(cudaMemsetAsync(flag.p, 0, 4, s));
            if (variant == 0) {
                // forward edges hook both endpoints' trees, so in-edges add nothing
                cc_sv_hook_kernel<<<wgrid, 256, 0, s>>>(g->offsets, g->dest, comp, V, flag.p);
                GBX_LAUNCH_CHECK();
                cc_compress_kernel<<<grid, 256, 0, s>>>(comp, V);
            } else {
                cc_lp_kernel<<<wgrid, 256, 0, s>>>(g->offsets, g->dest, comp, V, flag.p);
            }
            GBX_LAUNCH_CHECK();
            GBX_CUDA(cudaMemcpyAsync(&h, flag.p, 4, cudaMemcpyDeviceToHost, s));
            GBX_CUDA(cudaStreamSynchronize(s));
            iters++;
        }
    }
    GBX_TRY(out.finish(s));
    GBX_CUDA(cudaStreamSynchronize(s));
    if (iterations) *iterations = iters;
    return GBX_OK;
}
