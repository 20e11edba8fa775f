// Device preprocessing: the CSR build from an edge list and the degree
// reordering, i.e. the GPU form of graphCSRPreProcessingStep's sort / dedup /
// map steps (graphCSR.c:243-327) and of reorderGraphProcessDegree
// (reorder.c:275-380).
#include <algorithm>

#include "gbx_internal.cuh"
#include "gbx_sort.cuh"

namespace gbx {

static unsigned grid1d(uint64_t n) {
    uint64_t b = (n + 255) / 256;
    uint64_t cap = (uint64_t)num_sms() * 8;
    return (unsigned)std::max<uint64_t>(1, std::min(b, cap));
}

__global__ void max_u32_of_kernel(const uint32_t *a, uint32_t n, uint32_t *out) {
    uint32_t m = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) m = max(m, a[i]);
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

__global__ void max_id_kernel(const uint32_t *s, const uint32_t *d, uint32_t n, uint32_t *out) {
    uint32_t m = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        m = max(m, max(s[i], d[i]));
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

// Largest id of an edge list (device scalar read back), 0 for no edges.
static int max_edge_id(const uint32_t *s, const uint32_t *d, uint32_t n, cudaStream_t st, uint32_t *out) {
    *out = 0;
    if (!n) return GBX_OK;
    DevBuf<uint32_t> r;
    GBX_TRY(r.alloc(1, st));
    GBX_CUDA(cudaMemsetAsync(r.p, 0, 4, st));
    max_id_kernel<<<grid1d(n), 256, 0, st>>>(s, d, n, r.p);
    GBX_LAUNCH_CHECK();
    GBX_CUDA(cudaMemcpyAsync(out, r.p, 4, cudaMemcpyDeviceToHost, st));
    GBX_CUDA(cudaStreamSynchronize(st));
    return GBX_OK;
}

// mapVerticesWithInOutDegree_base (vertex.c:204-328) on a source-sorted edge
// list: each run of equal sources writes its first position (idx) and its end
// (into deg); degrees_from_runs_kernel turns the end into the run length. No
// atomics: a hub's run would otherwise take one atomic per edge on one address.
// kept: the edge count when only the device knows it yet. Four edges per
// thread and, where the list allows it, per load.
__global__ void map_vertices_kernel(const uint32_t *s, uint32_t n, const uint32_t *kept, uint32_t V, uint32_t *deg,
                                    uint32_t *idx) {
    if (kept) n = min(n, *kept);
    const bool wide = ((uintptr_t)s & 15u) == 0;
    const uint64_t step = (uint64_t)gridDim.x * blockDim.x * 4;
    for (uint64_t i0 = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) * 4; i0 < n; i0 += step) {
        const uint32_t i = (uint32_t)i0, m = min(4u, n - i);
        uint32_t v[4];
        if (wide && m == 4) {
            const uint4 q = *reinterpret_cast<const uint4 *>(s + i);
            v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
        } else {
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q) v[q] = q < m ? s[i + q] : 0u;
        }
        uint32_t before = i ? s[i - 1] & kIdMask : 0u;
        const uint32_t after = i + m < n ? s[i + m] & kIdMask : 0u;
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q) {
            if (q >= m) break;
            const uint32_t x = v[q] & kIdMask;
            const uint32_t next = q + 1 < m ? v[(q + 1) & 3] & kIdMask : after;
            if (x < V) {
                if (i + q == 0 || x != before) idx[x] = i + q;
                if (i + q + 1 == n || x != next) deg[x] = i + q + 1;
            }
            before = x;
        }
    }
}

__global__ void degrees_from_runs_kernel(uint32_t *deg, const uint32_t *idx, uint32_t V) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x)
        if (deg[v]) deg[v] -= idx[v];
}

// deg[key] += 1 for the active lanes, one atomic per distinct key in the warp
// (edge lists sorted by source repeat a key along the warp; hubs repeat
// everywhere, and one address taking every increment serialises the atomics)
__device__ __forceinline__ void count_keys(uint32_t *deg, uint32_t key, unsigned active) {
    const uint32_t lane = threadIdx.x & 31;
    if ((active >> lane) & 1u) {
        const unsigned peers = __match_any_sync(active, key);
        if (lane == (uint32_t)(__ffs(peers) - 1)) atomicAdd(deg + key, (uint32_t)__popc(peers));
    }
}

// Degrees and, in the same read of the edges, the largest id: an edge with an
// end outside [0, V) raises *max_id to at least V and is not counted. Four
// edges per lane are loaded before the first is counted.
__global__ void degree_count_kernel(const uint32_t *s, const uint32_t *d, uint32_t n, uint32_t V, int lmode,
                                    uint32_t *deg, uint32_t *max_id) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;  // a multiple of 32
    uint32_t m = 0;
    for (uint64_t base = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) & ~31ull; base < n; base += 4 * stride) {
        uint32_t a[4], b[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint64_t i = base + q * stride + lane;
            a[q] = i < n ? s[i] : 0u;
            b[q] = i < n ? d[i] : 0u;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint64_t i = base + q * stride + lane;
            const uint32_t top = max(a[q], b[q]);
            m = max(m, top);
            const unsigned active = __ballot_sync(0xffffffffu, i < n && top < V);
            if (lmode == 2 || lmode == 3) count_keys(deg, b[q], active);
            if (lmode != 2) count_keys(deg, a[q], active);
        }
    }
    m = __reduce_max_sync(0xffffffffu, m);
    if (lane == 0) atomicMax(max_id, m);
}

__global__ void new_labels_kernel(const uint32_t *sorted_ids, uint32_t V, uint32_t *newlab) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < V; i += gridDim.x * blockDim.x)
        newlab[sorted_ids[i]] = V - 1 - i;
}

// Four edges per thread: eight id loads, then eight gathers in flight.
__global__ void relabel_edges_kernel(uint32_t *s, uint32_t *d, uint32_t n, const uint32_t *newlab) {
    const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += 4 * step) {
        uint32_t a[4], b[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint64_t j = i + q * step;
            a[q] = j < n ? __ldcs(s + j) : 0u;
            b[q] = j < n ? __ldcs(d + j) : 0u;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            a[q] = __ldg(newlab + a[q]);
            b[q] = __ldg(newlab + b[q]);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint64_t j = i + q * step;
            if (j < n) {
                __stcs(s + j, a[q]);
                __stcs(d + j, b[q]);
            }
        }
    }
}

// label_array[v] = labels[label_array[v]]; inverse[label_array[v]] = v  (reorder.c:368-373)
__global__ void compose_labels_kernel(uint32_t *labels, uint32_t *inv, uint32_t V, const uint32_t *newlab) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
        uint32_t l = newlab[labels[v]];
        labels[v] = l;
        inv[l] = v;
    }
}

// ---- bucketed reorder modes (DBG, HUBSort, HUBCluster, Corder) -------------
struct BucketThresholds {
    uint32_t t[11];
    uint32_t n;
};

// key[v] = n-1 - bucket(v): a stable ascending sort of (key, id) lists the
// highest bucket first, ids ascending inside a bucket (reorder.c:439-572)
__global__ void bucket_key_kernel(const uint32_t *deg, uint32_t V, BucketThresholds th, uint32_t *key) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
        uint32_t i = 0;
        while (deg[v] > th.t[i]) ++i;  // th.t[th.n-1] = UINT32_MAX ends the scan
        key[v] = th.n - 1 - i;
    }
}

// newlab[sorted[i]] = i
__global__ void rank_labels_kernel(const uint32_t *sorted, uint32_t n, uint32_t *newlab) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        newlab[sorted[i]] = i;
}

// HUBSort: hot flag (degree above t0) per vertex
__global__ void hot_flag_kernel(const uint32_t *deg, uint32_t V, uint32_t t0, uint32_t *flag) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x)
        flag[v] = deg[v] > t0 ? 1u : 0u;
}

// hot vertices (ascending ids) and their degrees at their rank; cold vertices
// labelled H + (their rank among cold vertices) = H + v - (hot before v)
__global__ void hot_split_kernel(const uint32_t *deg, const uint32_t *flag, const uint32_t *pos, uint32_t V,
                                 const uint32_t *hot_total, uint32_t *hot_ids, uint32_t *hot_deg,
                                 uint32_t *newlab) {
    const uint32_t H = *hot_total;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
        if (flag[v]) {
            hot_ids[pos[v]] = v;
            hot_deg[pos[v]] = deg[v];
        } else {
            newlab[v] = H + v - pos[v];
        }
    }
}

// bad[0] counts labels out of range or taken twice (seen[] starts zeroed)
__global__ void permutation_check_kernel(const uint32_t *lab, uint32_t V, uint32_t *seen, unsigned *bad) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
        const uint32_t l = lab[v];
        if (l >= V || atomicExch(seen + l, 1u) != 0u) atomicAdd(bad, 1u);
    }
}

// ---- mask mode (maskGraphProcess, reorder.c:1164-1475) --------------------
// The vertex at position i of the bucket order takes the first region with
// room left (reorder.c:1408-1436): HOT below e0, WARM below e1, LUKEWARM
// below e2 (cumulative region ends), COLD after.
__global__ void mask_hints_kernel(const uint32_t *sorted, uint32_t V, uint64_t e0, uint64_t e1, uint64_t e2,
                                  uint32_t *mask) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < V; i += gridDim.x * blockDim.x)
        mask[sorted[i]] = i < e0 ? 0xC0000000u : i < e1 ? 0x80000000u : i < e2 ? 0x40000000u : 0u;
}

// maskEdgeList (reorder.c:1639-1657): every id ORed with its vertex's hint
__global__ void mask_edges_kernel(uint32_t *s, uint32_t *d, uint32_t n, const uint32_t *mask) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t a = s[i], b = d[i];
        s[i] = a | mask[a];
        d[i] = b | mask[b];
    }
}

static int bits_for(uint32_t maxv) {
    int b = 0;
    while (b < 32 && (maxv >> b)) ++b;
    return b;
}

}  // namespace gbx

using namespace gbx;

extern "C" int gbx_csr_build(uint32_t num_edges, const uint32_t *src, const uint32_t *dst,
                             const float *w, int symmetric, int dedup, int sort_mode,
                             uint32_t num_vertices, uint32_t *out_degree, uint32_t *edges_idx,
                             uint32_t *src_out, uint32_t *dst_out, float *w_out,
                             uint32_t *num_edges_out, void *stream) {
    clear_error();
    GBX_REQUIRE(num_edges == 0 || (src && dst), GBX_ERR_INVALID, "src/dst is NULL");
    GBX_REQUIRE(out_degree && edges_idx && num_edges_out, GBX_ERR_INVALID, "output is NULL");
    GBX_REQUIRE(num_vertices > 0, GBX_ERR_INVALID, "num_vertices must be > 0");
    GBX_REQUIRE(!dedup || sort_mode == 1 || sort_mode == 3, GBX_ERR_INVALID,
                "dedup needs a (source,destination) sort (sort_mode 1)");
    GBX_REQUIRE(!symmetric || num_edges <= 0x7FFFFFFFu, GBX_ERR_INVALID, "too many edges");
    GBX_TRY(ensure_device());
    cudaStream_t s = (cudaStream_t)stream;
    const uint32_t E = num_edges, E2 = symmetric ? 2 * num_edges : num_edges, V = num_vertices;
    InArray<uint32_t> isrc, idst;
    InArray<float> iw;
    GBX_TRY(isrc.bind(src, E, s));
    GBX_TRY(idst.bind(dst, E, s));
    GBX_TRY(iw.bind(w_out ? w : nullptr, E, s));
    // outputs the caller does not want, or wants in host memory, go to working memory
    DevBuf<uint32_t> ss, sd;
    OutArray<uint32_t> os, od, odeg, oidx;
    OutArray<float> ow;
    GBX_TRY(os.bind(src_out, E2, s));
    GBX_TRY(od.bind(dst_out, E2, s));
    GBX_TRY(ow.bind(w_out, E2, s));
    if (!src_out) GBX_TRY(ss.alloc(E2, s));
    if (!dst_out) GBX_TRY(sd.alloc(E2, s));
    uint32_t *fs = src_out ? os.d : ss.p;
    DevBuf<SortControl> ctl;
    GBX_TRY(sort_edges(EdgeView{isrc.d, idst.d, E, symmetric}, iw.d, sort_mode == 1 || sort_mode == 3, dedup != 0, V,
                       fs, dst_out ? od.d : sd.p, ow.d, &ctl, s));
    GBX_TRY(odeg.bind(out_degree, V, s));
    GBX_TRY(oidx.bind(edges_idx, V, s));
    GBX_CUDA(cudaMemsetAsync(odeg.d, 0, (size_t)V * 4, s));
    GBX_CUDA(cudaMemsetAsync(oidx.d, 0, (size_t)V * 4, s));
    if (E2) {
        map_vertices_kernel<<<grid1d(ceil_div(E2, 4)), 256, 0, s>>>(fs, E2, dedup ? &ctl.p->kept : nullptr, V, odeg.d,
                                                                    oidx.d);
        GBX_LAUNCH_CHECK();
        degrees_from_runs_kernel<<<grid1d(V), 256, 0, s>>>(odeg.d, oidx.d, V);
        GBX_LAUNCH_CHECK();
    }
    SortControl h;
    GBX_CUDA(cudaMemcpyAsync(&h, ctl.p, sizeof(h), cudaMemcpyDeviceToHost, s));
    GBX_CUDA(cudaStreamSynchronize(s));
    GBX_TRY(check_sort(h));
    const uint32_t Eout = dedup ? h.kept : E2;
    GBX_TRY(odeg.finish(s));
    GBX_TRY(oidx.finish(s));
    os.n = od.n = ow.n = Eout;
    GBX_TRY(os.finish(s));
    GBX_TRY(od.finish(s));
    GBX_TRY(ow.finish(s));
    if (odeg.to_host() || oidx.to_host() || os.to_host() || od.to_host() || ow.to_host())
        GBX_CUDA(cudaStreamSynchronize(s));
    *num_edges_out = Eout;
    return GBX_OK;
}

extern "C" int gbx_degree_reorder(uint32_t num_vertices, uint32_t num_edges, uint32_t *src,
                                  uint32_t *dst, int lmode, uint32_t *labels,
                                  uint32_t *inverse_labels, void *stream) {
    clear_error();
    GBX_REQUIRE(num_vertices > 0, GBX_ERR_INVALID, "num_vertices must be > 0");
    GBX_REQUIRE(num_edges == 0 || (src && dst), GBX_ERR_INVALID, "src/dst is NULL");
    GBX_REQUIRE(labels && inverse_labels, GBX_ERR_INVALID, "labels is NULL");
    GBX_REQUIRE(lmode != 10, GBX_ERR_UNSUPPORTED,
                "lmode 10 (random order) draws per-thread random degrees in the reference and is not "
                "reproducible; relabel with explicit labels (gbx_relabel) instead");
    GBX_REQUIRE(lmode != 11, GBX_ERR_INVALID, "lmode 11 (labels from a file): call gbx_relabel with the labels");
    GBX_REQUIRE((lmode >= 1 && lmode <= 9) || lmode == 12 || lmode == 13, GBX_ERR_INVALID,
                "lmode must be 1-9, 12 or 13");
    GBX_TRY(ensure_device());
    cudaStream_t s = (cudaStream_t)stream;
    const uint32_t V = num_vertices, E = num_edges;
    OutArray<uint32_t> os, od, ol, oi;
    GBX_TRY(os.bind(src, E, s));
    GBX_TRY(od.bind(dst, E, s));
    GBX_TRY(ol.bind(labels, V, s));
    GBX_TRY(oi.bind(inverse_labels, V, s));
    if (os.to_host() && E) GBX_CUDA(cudaMemcpyAsync(os.d, src, (size_t)E * 4, cudaMemcpyHostToDevice, s));
    if (od.to_host() && E) GBX_CUDA(cudaMemcpyAsync(od.d, dst, (size_t)E * 4, cudaMemcpyHostToDevice, s));
    if (ol.to_host()) GBX_CUDA(cudaMemcpyAsync(ol.d, labels, (size_t)V * 4, cudaMemcpyHostToDevice, s));
    DevBuf<uint32_t> deg, ids, newlab, mx;
    GBX_TRY(deg.alloc(V, s));
    GBX_TRY(ids.alloc(V, s));
    GBX_TRY(newlab.alloc(V, s));
    GBX_TRY(mx.alloc(2, s));  // largest degree, largest id
    GBX_CUDA(cudaMemsetAsync(deg.p, 0, (size_t)V * 4, s));
    GBX_CUDA(cudaMemsetAsync(mx.p, 0, 8, s));
    // reorderGraphGenerateInOutDegrees (reorder.c:1483-1552): in-degrees for
    // 2, 5, 7, 9, in + out for 3, out-degrees for every other mode
    const bool in_deg = lmode == 2 || lmode == 5 || lmode == 7 || lmode == 9;
    const int count_mode = in_deg ? 2 : (lmode == 3 ? 3 : 1);
    if (E) {
        degree_count_kernel<<<grid1d(ceil_div(E, 4)), 256, 0, s>>>(os.d, od.d, E, V, count_mode, deg.p, mx.p + 1);
        GBX_LAUNCH_CHECK();
    }
    max_u32_of_kernel<<<grid1d(V), 256, 0, s>>>(deg.p, V, mx.p);
    GBX_LAUNCH_CHECK();
    uint32_t hm[2];
    GBX_CUDA(cudaMemcpyAsync(hm, mx.p, 8, cudaMemcpyDeviceToHost, s));
    GBX_CUDA(cudaStreamSynchronize(s));
    const uint32_t hmax = hm[0];
    GBX_REQUIRE(E == 0 || hm[1] < V, GBX_ERR_INVALID, "vertex id %u >= num_vertices %u", hm[1], V);
    // thresholds of the bucketed modes: t0 = avg <= 1 ? 1 : avg/2 (HUBCluster:
    // avg), doubling, last UINT32_MAX; avg = E/V in uint32 as the reference's
    // EdgeList.avg_degree
    BucketThresholds th{};
    th.n = (lmode == 4 || lmode == 5 || lmode == 12 || lmode == 13) ? 11u : (lmode >= 6 && lmode <= 9 ? 2u : 0u);
    if (th.n) {
        const uint32_t avg = E / V;
        th.t[0] = (lmode == 8 || lmode == 9) ? avg : (avg <= 1 ? 1u : avg / 2);
        for (uint32_t i = 1; i + 1 < th.n; ++i) th.t[i] = th.t[i - 1] * 2u;
        th.t[th.n - 1] = 0xFFFFFFFFu;
    }
    if (th.n == 0) {
        // reorderGraphListDegree (reorder.c:296-380): stable ascending sort of
        // (degree, id), label N-1-rank
        GBX_TRY(radix_sort_pairs(deg.p, ids.p, V, bits_for(hmax), s, true));
        new_labels_kernel<<<grid1d(V), 256, 0, s>>>(ids.p, V, newlab.p);
        GBX_LAUNCH_CHECK();
    } else if (lmode == 6 || lmode == 7) {
        // HUBSort (reorder.c:814-982): hot vertices (degree above t0) stably
        // sorted by degree and labelled in reverse, cold ones after, in id order
        DevBuf<uint32_t> flag, pos, hot_deg, tot;
        GBX_TRY(flag.alloc(V, s));
        GBX_TRY(pos.alloc(V, s));
        GBX_TRY(hot_deg.alloc(V, s));
        GBX_TRY(tot.alloc(1, s));
        hot_flag_kernel<<<grid1d(V), 256, 0, s>>>(deg.p, V, th.t[0], flag.p);
        GBX_LAUNCH_CHECK();
        GBX_TRY(exclusive_scan_u32(flag.p, pos.p, V, s, tot.p));
        hot_split_kernel<<<grid1d(V), 256, 0, s>>>(deg.p, flag.p, pos.p, V, tot.p, ids.p, hot_deg.p, newlab.p);
        GBX_LAUNCH_CHECK();
        uint32_t H = 0;
        GBX_CUDA(cudaMemcpyAsync(&H, tot.p, 4, cudaMemcpyDeviceToHost, s));
        GBX_CUDA(cudaStreamSynchronize(s));
        GBX_TRY(radix_sort_pairs(hot_deg.p, ids.p, H, bits_for(hmax), s));
        if (H) {
            new_labels_kernel<<<grid1d(H), 256, 0, s>>>(ids.p, H, newlab.p);
            GBX_LAUNCH_CHECK();
        }
    } else {
        // DBG / Corder (11 buckets) and HUBCluster (2): buckets from the
        // highest, ids ascending inside a bucket
        bucket_key_kernel<<<grid1d(V), 256, 0, s>>>(deg.p, V, th, deg.p);
        GBX_LAUNCH_CHECK();
        GBX_TRY(radix_sort_pairs(deg.p, ids.p, V, bits_for(th.n - 1), s, true));
        rank_labels_kernel<<<grid1d(V), 256, 0, s>>>(ids.p, V, newlab.p);
        GBX_LAUNCH_CHECK();
    }
    if (E) {
        relabel_edges_kernel<<<grid1d(E), 256, 0, s>>>(os.d, od.d, E, newlab.p);
        GBX_LAUNCH_CHECK();
    }
    compose_labels_kernel<<<grid1d(V), 256, 0, s>>>(ol.d, oi.d, V, newlab.p);
    GBX_LAUNCH_CHECK();
    GBX_TRY(os.finish(s));
    GBX_TRY(od.finish(s));
    GBX_TRY(ol.finish(s));
    GBX_TRY(oi.finish(s));
    GBX_CUDA(cudaStreamSynchronize(s));
    return GBX_OK;
}

extern "C" int gbx_relabel(uint32_t num_vertices, uint32_t num_edges, uint32_t *src, uint32_t *dst,
                           const uint32_t *new_labels, uint32_t *labels, uint32_t *inverse_labels, void *stream) {
    clear_error();
    GBX_REQUIRE(num_vertices > 0, GBX_ERR_INVALID, "num_vertices must be > 0");
    GBX_REQUIRE(num_edges == 0 || (src && dst), GBX_ERR_INVALID, "src/dst is NULL");
    GBX_REQUIRE(new_labels && labels && inverse_labels, GBX_ERR_INVALID, "labels is NULL");
    GBX_TRY(ensure_device());
    cudaStream_t s = (cudaStream_t)stream;
    const uint32_t V = num_vertices, E = num_edges;
    InArray<uint32_t> nl;
    GBX_TRY(nl.bind(new_labels, V, s));
    DevBuf<uint32_t> seen;
    DevBuf<unsigned> bad;
    GBX_TRY(seen.alloc(V, s));
    GBX_TRY(bad.alloc(1, s));
    GBX_CUDA(cudaMemsetAsync(seen.p, 0, (size_t)V * 4, s));
    GBX_CUDA(cudaMemsetAsync(bad.p, 0, 4, s));
    permutation_check_kernel<<<grid1d(V), 256, 0, s>>>(nl.d, V, seen.p, bad.p);
    GBX_LAUNCH_CHECK();
    unsigned hbad = 0;
    GBX_CUDA(cudaMemcpyAsync(&hbad, bad.p, 4, cudaMemcpyDeviceToHost, s));
    GBX_CUDA(cudaStreamSynchronize(s));
    GBX_REQUIRE(hbad == 0, GBX_ERR_INVALID, "new_labels is not a permutation of [0, %u): %u bad entries", V,
                hbad);
    OutArray<uint32_t> os, od, ol, oi;
    GBX_TRY(os.bind(src, E, s));
    GBX_TRY(od.bind(dst, E, s));
    GBX_TRY(ol.bind(labels, V, s));
    GBX_TRY(oi.bind(inverse_labels, V, s));
    if (os.to_host() && E) GBX_CUDA(cudaMemcpyAsync(os.d, src, (size_t)E * 4, cudaMemcpyHostToDevice, s));
    if (od.to_host() && E) GBX_CUDA(cudaMemcpyAsync(od.d, dst, (size_t)E * 4, cudaMemcpyHostToDevice, s));
    if (ol.to_host()) GBX_CUDA(cudaMemcpyAsync(ol.d, labels, (size_t)V * 4, cudaMemcpyHostToDevice, s));
    uint32_t id_max = 0;
    GBX_TRY(max_edge_id(os.d, od.d, E, s, &id_max));
    GBX_REQUIRE(E == 0 || id_max < V, GBX_ERR_INVALID, "vertex id %u >= num_vertices %u", id_max, V);
    if (E) {
        relabel_edges_kernel<<<grid1d(E), 256, 0, s>>>(os.d, od.d, E, nl.d);
        GBX_LAUNCH_CHECK();
    }
    compose_labels_kernel<<<grid1d(V), 256, 0, s>>>(ol.d, oi.d, V, nl.d);
    GBX_LAUNCH_CHECK();
    GBX_TRY(os.finish(s));
    GBX_TRY(od.finish(s));
    GBX_TRY(ol.finish(s));
    GBX_TRY(oi.finish(s));
    GBX_CUDA(cudaStreamSynchronize(s));
    return GBX_OK;
}

extern "C" int gbx_mask_graph(uint32_t num_vertices, uint32_t num_edges, uint32_t *src, uint32_t *dst,
                              int mmode, uint32_t cache_size, uint32_t *mask_array, void *stream) {
    clear_error();
    GBX_REQUIRE(num_vertices > 0, GBX_ERR_INVALID, "num_vertices must be > 0");
    GBX_REQUIRE(num_edges == 0 || (src && dst), GBX_ERR_INVALID, "src/dst is NULL");
    GBX_REQUIRE(mask_array, GBX_ERR_INVALID, "mask_array is NULL");
    GBX_REQUIRE(mmode >= 1 && mmode <= 6, GBX_ERR_INVALID, "mmode must be 1-6");
    GBX_TRY(ensure_device());
    cudaStream_t s = (cudaStream_t)stream;
    const uint32_t V = num_vertices, E = num_edges;
    OutArray<uint32_t> os, od, om;
    GBX_TRY(os.bind(src, E, s));
    GBX_TRY(od.bind(dst, E, s));
    GBX_TRY(om.bind(mask_array, V, s));
    if (os.to_host() && E) GBX_CUDA(cudaMemcpyAsync(os.d, src, (size_t)E * 4, cudaMemcpyHostToDevice, s));
    if (od.to_host() && E) GBX_CUDA(cudaMemcpyAsync(od.d, dst, (size_t)E * 4, cudaMemcpyHostToDevice, s));
    uint32_t id_max = 0;
    GBX_TRY(max_edge_id(os.d, od.d, E, s, &id_max));
    GBX_REQUIRE(E == 0 || id_max < V, GBX_ERR_INVALID,
                "vertex id %u >= num_vertices %u (ids must not carry mask bits yet)", id_max, V);
    DevBuf<uint32_t> key, ids, seen;
    GBX_TRY(key.alloc(V, s));
    GBX_TRY(ids.alloc(V, s));
    GBX_TRY(seen.alloc(1, s));  // the largest id again, not read
    GBX_CUDA(cudaMemsetAsync(seen.p, 0, 4, s));
    GBX_CUDA(cudaMemsetAsync(key.p, 0, (size_t)V * 4, s));
    // maskGraphProcessGenerateInOutDegrees (reorder.c:1260-1306): in-degrees
    // for 2, 4, in + out for 5, 6, out-degrees otherwise
    const int count_mode = (mmode == 2 || mmode == 4) ? 2 : (mmode == 5 || mmode == 6) ? 3 : 1;
    if (E) {
        degree_count_kernel<<<grid1d(ceil_div(E, 4)), 256, 0, s>>>(os.d, od.d, E, V, count_mode, key.p, seen.p);
        GBX_LAUNCH_CHECK();
    }
    // DBG's 11 buckets (reorder.c:1214-1228), highest first, ids ascending
    BucketThresholds th{};
    th.n = 11;
    const uint32_t avg = E / V;
    th.t[0] = avg <= 1 ? 1u : avg / 2;
    for (uint32_t i = 1; i + 1 < th.n; ++i) th.t[i] = th.t[i - 1] * 2u;
    th.t[th.n - 1] = 0xFFFFFFFFu;
    bucket_key_kernel<<<grid1d(V), 256, 0, s>>>(key.p, V, th, key.p);
    GBX_LAUNCH_CHECK();
    GBX_TRY(radix_sort_pairs(key.p, ids.p, V, bits_for(th.n - 1), s, true));
    // region sizes (reorder.c:1329-1345) with cs = cache_size / 4: V/4 each
    // when V - cs < 2 cs, else cs*8, *4, *4 in uint32 as the reference
    const uint32_t cs = cache_size >> 2;
    uint32_t r0, r1, r2;
    if ((int64_t)V - (int64_t)cs < 2 * (int64_t)cs) {
        r0 = r1 = r2 = V / 4;
    } else {
        r0 = cs * 8u;
        r1 = r0 * 4u;
        r2 = r1 * 4u;
    }
    const uint64_t e0 = r0, e1 = e0 + r1, e2 = e1 + r2;
    mask_hints_kernel<<<grid1d(V), 256, 0, s>>>(ids.p, V, e0, e1, e2, om.d);
    GBX_LAUNCH_CHECK();
    GBX_TRY(om.finish(s));
    if ((mmode == 1 || mmode == 2) && E) {
        mask_edges_kernel<<<grid1d(E), 256, 0, s>>>(os.d, od.d, E, om.d);
        GBX_LAUNCH_CHECK();
        GBX_TRY(os.finish(s));
        GBX_TRY(od.finish(s));
    }
    GBX_CUDA(cudaStreamSynchronize(s));
    return GBX_OK;
}
