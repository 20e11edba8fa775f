// Sorting of pairs and of whole edges (gbx_sort.cu).
#pragma once

#include "gbx_internal.cuh"

namespace gbx {

// E edges; symmetric: followed by every edge reversed (edgeList.c:559-576)
struct EdgeView {
    const uint32_t *src, *dst;
    uint32_t E;
    int symmetric;
    __host__ __device__ uint32_t count() const { return symmetric ? 2 * E : E; }
};

// Device words a sort leaves behind.
struct SortControl {
    unsigned error;       // a wait ran out
    unsigned trivial;     // bit k: digit k is the same in every element
    uint32_t max_id;      // largest id, mask bits included
    uint32_t max_vertex;  // largest id without them
    uint32_t kept;        // edges kept by the removal of repeats
    uint32_t pad[11];
    unsigned ticket[16];  // next tile of each pass
};

int check_sort(const SortControl &h);  // GBX_ERR_DEVICE_TIMEOUT when a wait ran out

// Stable sort of (key, value) pairs by the `bits` low key bits, in place.
// iota: the values on entry are 0, 1, 2, ... and are not read. Synchronizes
// the stream to learn whether a wait ran out (the pairs are unusable then).
int radix_sort_pairs(uint32_t *keys, uint32_t *vals, uint32_t n, int bits, cudaStream_t s, bool iota = false);

// Edges sorted by source (by_dst: by (source, destination)), stably, into
// src_out / dst_out / w_out (device, room for e.count() edges; w_out may be
// null; w null: weights 1). The outputs may be the input arrays. dedup:
// without self loops and repeats. Enqueued on s after one synchronization
// that checks the ids (GBX_ERR_INVALID when a vertex is not below
// num_vertices, nothing written); *ctl is read by the caller afterwards.
int sort_edges(const EdgeView &e, const float *w, bool by_dst, bool dedup, uint32_t num_vertices, uint32_t *src_out,
               uint32_t *dst_out, float *w_out, DevBuf<SortControl> *ctl, cudaStream_t s);

}  // namespace gbx
