// Batched BFS and PageRank over many graphs in one persistent launch.
// No reference counterpart as a batch: each graph gets exactly the per-graph
// results of the reference's breadthFirstSearchGraphCSR (BFS.c:103-127, the
// direction-optimising loop :335-485) and pageRankPullGraphCSR
// (pageRank.c:245-368), the same as gbx_bfs / gbx_pagerank_pull.
//
// Layout (gbx_batch): the graphs' CSRs packed back to back. Packed vertex
// vertex_base[g] + v is graph g's vertex v; offsets[] (total V + 1) hold
// global edge positions; dest / in_src hold graph-local ids. A device work
// queue deals whole graphs to CTAs, largest edge count first.
//
// One CTA owns one graph at a time, so a level or an iteration ends with
// __syncthreads instead of a grid barrier, and the per-graph working set
// lives in shared memory:
//   BFS: visited / frontier / next bitmaps (3 x V/8 bytes); neighbour tests
//        are shared-memory bit probes. Top-down flattens the out-edges of 32
//        frontier vertices per warp; bottom-up gives each warp 32 unvisited
//        vertices, one lane each, scanning in-edges until a frontier parent.
//   PR:  contributions (4V bytes) in shared memory; the gather streams the
//        graph's in-edges as words (a batch's first PageRank call lays them
//        out) and reads contributions from shared memory.
// Graphs too large for the shared-memory capacity use the same code on a
// per-CTA global scratch slot.
#include <algorithm>
#include <mutex>
#include <numeric>
#include <vector>

#include "gbx_internal.cuh"

struct gbx_batch {
    int device = 0;
    uint32_t G = 0, V = 0, E = 0;
    uint32_t max_v = 0;
    uint32_t *vbase = nullptr;       // G+1
    uint32_t *offsets = nullptr;     // V+1, global edge positions
    uint32_t *dest = nullptr;        // E, graph-local ids
    uint32_t *in_offsets = nullptr;  // V+1 or null (pull = forward CSR)
    uint32_t *in_src = nullptr;      // E or null
    uint32_t *order = nullptr;       // G, graph ids by descending edge count
    std::vector<uint32_t> h_vbase;   // host copy of vbase
    // PageRank's in-edge words (built by its first call): graph g's start
    // wbase[g] units of 16 bytes into words, its rows with edges at rows + vbase[g]
    uint4 *words = nullptr;
    uint32_t *wbase = nullptr;       // G
    uint2 *rows = nullptr;           // V: {vertex, out-degree}
    // G * 33: where each warp's part begins: {edge, row | top bit: it began earlier}
    uint2 *starts = nullptr;
    std::mutex words_mutex;
    const uint32_t *poff() const { return in_offsets ? in_offsets : offsets; }
    const uint32_t *psrc() const { return in_offsets ? in_src : dest; }
};

namespace gbx {

constexpr int kBbThreads = 512;
constexpr int kBbWarps = kBbThreads / 32;
constexpr uint32_t kBbWordsCap = 4096;  // bitmap words in shared memory: V <= 131072
constexpr int kBpThreads = 1024;
constexpr int kBpWarps = kBpThreads / 32;
constexpr uint32_t kBpSmemV = 46976;   // contributions in shared memory (188 KB), a multiple of 32
constexpr uint32_t kBpShortV = 32768;  // ids that leave a 16-bit word's top bit free
constexpr uint32_t kBpBuf = 288;       // pending row sums of a warp: fewer than 32, and a group's 256

__device__ __forceinline__ uint32_t bb_next_graph(uint32_t *cursor, uint32_t G, const uint32_t *order,
                                                  uint32_t *s_slot) {
    __syncthreads();
    if (threadIdx.x == 0) {
        const uint32_t i = atomicAdd(cursor, 1u);
        *s_slot = i < G ? order[i] : 0xFFFFFFFFu;
    }
    __syncthreads();
    return *s_slot;
}

struct BbArgs {
    uint32_t G;
    const uint32_t *vbase, *off, *dest, *poff, *psrc, *order, *sources;
    uint32_t *dist;
    int32_t *parent;
    gbx_bfs_result *res;
    uint32_t *cursor;
    uint32_t *scratch;  // per CTA: 3 * scratch_words
    uint32_t scratch_words;
    uint32_t alpha, beta;
};

// ---- BFS -----------------------------------------------------------------------
__global__ void __launch_bounds__(kBbThreads, 2) bfs_batched_kernel(BbArgs a) {
    extern __shared__ uint32_t s_bits[];  // 3 * kBbWordsCap
    __shared__ uint32_t s_pre[kBbWarps][33];
    __shared__ uint32_t s_slot, s_nf;
    __shared__ unsigned long long s_mf;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (;;) {
        const uint32_t g = bb_next_graph(a.cursor, a.G, a.order, &s_slot);
        if (g == 0xFFFFFFFFu) break;
        const uint32_t vb = a.vbase[g], Vg = a.vbase[g + 1] - vb;
        const uint32_t words = (Vg + 31) / 32;
        uint32_t *S, *F, *N;
        if (words <= kBbWordsCap) {
            S = s_bits;
            F = s_bits + kBbWordsCap;
            N = s_bits + 2 * kBbWordsCap;
        } else {
            uint32_t *base = a.scratch + (size_t)blockIdx.x * 3 * a.scratch_words;
            S = base;
            F = base + a.scratch_words;
            N = base + 2 * a.scratch_words;
        }
        const uint32_t *off = a.off + vb;  // off[v], v local; values are global edge positions
        const uint32_t *poff = a.poff + vb;
        const uint32_t src = a.sources[g];
        const uint32_t Eg = off[Vg] - off[0];
        for (uint32_t w = threadIdx.x; w < words; w += blockDim.x) {
            S[w] = 0;
            F[w] = 0;
            N[w] = 0;
        }
        for (uint32_t v = threadIdx.x; v < Vg; v += blockDim.x) a.dist[vb + v] = 0;
        if (threadIdx.x == 0) {
            s_nf = 0;
            s_mf = 0;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            S[src >> 5] = 1u << (src & 31);
            F[src >> 5] = 1u << (src & 31);
            if (a.parent) a.parent[vb + src] = (int32_t)src;
        }
        __syncthreads();
        const uint32_t deg_src = off[src + 1] - off[src];
        unsigned long long mf = deg_src, edges_total = deg_src;
        uint32_t processed = 1, iteration = 1, L = 0, td = 0, bu = 0, nf_prev = 0;
        bool in_bu = false;
        for (uint32_t step = 0; step <= Vg; ++step) {
            const unsigned long long mu = (unsigned long long)Eg - edges_total;
            bool use_bu;
            if (in_bu)
                use_bu = true;
            else
                use_bu = mf > mu / a.alpha;
            uint32_t my_nf = 0;
            unsigned long long my_mf = 0;
            if (use_bu) {
                // each warp owns whole words of S and N: no atomics on them
                for (uint32_t w = warp; w < words; w += kBbWarps) {
                    const uint32_t valid = (w + 1) * 32 <= Vg ? 0xFFFFFFFFu : ((1u << (Vg & 31)) - 1u);
                    const uint32_t unv = ~S[w] & valid;
                    if (!unv) continue;
                    const uint32_t v = w * 32 + lane;
                    uint32_t found = 0xFFFFFFFFu;
                    if ((unv >> lane) & 1u) {
                        const uint32_t b = poff[v], e = poff[v + 1];
                        for (uint32_t j = b; j < e; ++j) {
                            const uint32_t u = __ldg(a.psrc + j);
                            if ((F[u >> 5] >> (u & 31)) & 1u) {
                                found = u;
                                break;
                            }
                        }
                    }
                    const uint32_t hit = __ballot_sync(0xFFFFFFFFu, found != 0xFFFFFFFFu);
                    if (found != 0xFFFFFFFFu) {
                        a.dist[vb + v] = L + 1;
                        if (a.parent) a.parent[vb + v] = (int32_t)found;
                        my_mf += off[v + 1] - off[v];
                    }
                    if (lane == 0 && hit) {
                        S[w] |= hit;
                        N[w] = hit;
                        my_nf += __popc(hit);
                    }
                }
                bu++;
            } else {
                for (uint32_t w = warp; w < words; w += kBbWarps) {
                    const uint32_t fw = F[w];
                    if (!fw) continue;
                    const uint32_t u = w * 32 + lane;
                    const bool mine = (fw >> lane) & 1u;
                    const uint32_t eb = mine ? off[u] : 0;
                    const uint32_t deg = mine ? off[u + 1] - eb : 0;
                    // exclusive prefix of the 32 degrees
                    uint32_t incl = deg;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                        if (lane >= (uint32_t)o) incl += t;
                    }
                    const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
                    s_pre[warp][lane] = incl - deg;
                    if (lane == 31) s_pre[warp][32] = total;
                    __syncwarp();
                    for (uint32_t j = lane; j < total; j += 32) {
                        // owner: last k with s_pre[k] <= j (degree-0 lanes share a prefix; take the last)
                        uint32_t lo = 0, hi = 31;
                        while (lo < hi) {
                            const uint32_t mid = (lo + hi + 1) >> 1;
                            if (s_pre[warp][mid] <= j) lo = mid; else hi = mid - 1;
                        }
                        const uint32_t k = lo;
                        const uint32_t uu = w * 32 + k;
                        const uint32_t e = off[uu] + (j - s_pre[warp][k]);
                        const uint32_t v = __ldg(a.dest + e);
                        const uint32_t bit = 1u << (v & 31);
                        if (S[v >> 5] & bit) continue;
                        const uint32_t old = atomicOr(&S[v >> 5], bit);
                        if (old & bit) continue;
                        atomicOr(&N[v >> 5], bit);
                        a.dist[vb + v] = L + 1;
                        if (a.parent) a.parent[vb + v] = (int32_t)uu;
                        my_nf++;
                        my_mf += off[v + 1] - off[v];
                    }
                    __syncwarp();
                }
                td++;
            }
            my_nf = warp_sum(my_nf);
            my_mf = warp_sum(my_mf);
            if (lane == 0 && (my_nf || my_mf)) {
                atomicAdd(&s_nf, my_nf);
                atomicAdd(&s_mf, my_mf);
            }
            __syncthreads();
            const uint32_t nf = s_nf;
            const unsigned long long nmf = s_mf;
            __syncthreads();
            if (threadIdx.x == 0) {
                s_nf = 0;
                s_mf = 0;
            }
            // the old frontier becomes the next output bitmap
            for (uint32_t w = threadIdx.x; w < words; w += blockDim.x) F[w] = 0;
            uint32_t *t = F;
            F = N;
            N = t;
            __syncthreads();
            processed += nf;
            iteration++;
            edges_total += nmf;
            if (nf == 0) break;
            L++;
            if (use_bu) {
                // the reference stays bottom-up while the frontier grows or is large
                in_bu = nf > nf_prev || nf > Vg / a.beta;
                nf_prev = nf;
            } else {
                nf_prev = nf;
            }
            mf = nmf;
        }
        // unreached vertices: parent = -out_degree, or -1 without out-edges
        if (a.parent) {
            for (uint32_t v = threadIdx.x; v < Vg; v += blockDim.x) {
                if (!((S[v >> 5] >> (v & 31)) & 1u)) {
                    const uint32_t d = off[v + 1] - off[v];
                    a.parent[vb + v] = d ? -(int32_t)d : -1;
                }
            }
        }
        if (threadIdx.x == 0 && a.res) {
            gbx_bfs_result r;
            r.processed_nodes = processed;
            r.iteration = iteration;
            r.depth = L;
            r.top_down_steps = td;
            r.bottom_up_steps = bu;
            r.reserved = 0;
            r.edges_traversed = edges_total;
            a.res[g] = r;
        }
    }
}

// ---- PageRank --------------------------------------------------------------------
// A graph's in-edges are a stream of words in row order: the source's id and,
// in the top bit, whether the edge is its row's last; 16 bits each for graphs
// of up to 32,768 vertices, else 32. The CTA's 32 warps take equal parts of
// the stream, 256 edges at a time, eight consecutive ones per lane: a lane adds
// up its row pieces and a segmented scan joins them across the warp, so no
// row is too long or too short for its lane and no offsets are read. Row sums
// collect in shared memory and leave 32 at a time through the epilogue, which
// writes the vertex's next contribution. A row cut by a part's end leaves
// pieces that one warp joins after the barrier. Every order of additions is
// fixed: ranks repeat bit for bit.
//
// Bound: the shared-memory pipe (65%: a gather of 32 random words takes 3 to 4
// cycles, and scans' shuffles go the same way) and the issue slots (65%: 190
// instructions per 256 edges). 2,048 graphs, 30 iterations, 6.5G edge visits:
// 7.9 ms; 11.0 without spreading the banks and with a scan per group of a long
// row, 9.1 with equal edges per warp. Rows taken one per lane or one per warp,
// ids in 32 bits: 20.9 ms.
//
// Distance of the ranks from 64 bits, relative L2, against that form (which
// compensated every addition of rows above 32 edges): 14 R-MAT batches of 16 to
// 2,048 graphs 3.5% nearer on average; in made-up batches of one row length,
// rows of 2 to 32 edges 20% nearer, 33 to 400 4% to 11% further off, longer ones
// 7% nearer. With the errors of lanes and scan carried along all of them are 10%
// to 20% nearer, and a pass over the 2,048 graphs takes 9.9 ms instead of 9.0.
struct BpArgs {
    uint32_t G;
    const uint32_t *vbase, *off, *order;
    const uint4 *words;
    const uint32_t *wbase;
    const uint2 *starts, *rows;
    float *ranks;       // output, also one rank buffer
    float *rother;      // second rank buffer (V)
    float *next;        // per CTA: next contributions where two buffers do not fit shared memory
    float *scratch;     // per CTA: contributions of graphs above kBpSmemV
    uint32_t max_v;     // floats per CTA in next and scratch
    uint32_t smem_v;    // floats of contributions in shared memory
    uint32_t *cursor;
    uint32_t max_it;
    double epsilon;
    gbx_pr_result *res;
};

__device__ __forceinline__ void kahan_add(float &sum, float &comp, float x) {
    const float y = __fsub_rn(x, comp);
    const float t = __fadd_rn(sum, y);
    comp = __fsub_rn(__fsub_rn(t, sum), y);
    sum = t;
}

// A warp's part of a graph's word stream: whole groups of 256 edges, with an
// equal share of the cost; a row costs about as much as this many edges (its
// sum and epilogue against a group's 150 instructions).
constexpr uint32_t kBpRowCost = 4;
constexpr uint32_t kBpStarts = kBpWarps + 1;

// inclusive segmented scan over the warp: lane's value added to those below it
// down to the nearest lane (itself included) that starts a segment
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
template <class T>
__device__ __forceinline__ T segmented_scan(T x, bool starts) {
    const uint32_t lane = threadIdx.x & 31;
    const unsigned m = __ballot_sync(0xffffffffu, starts) & (0xffffffffu >> (31 - lane));
    const uint32_t back = m ? lane - (31u - __clz(m)) : lane;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T t = __shfl_up_sync(0xffffffffu, x, o);
        if ((uint32_t)o <= back) x = add_rn(x, t);
    }
    return x;
}

// bank-spreading place of a contribution inside its 32 vertices: R-MAT ids have
// few one bits, and a quarter of the edges would meet in bank 0
__host__ __device__ __forceinline__ uint32_t bp_place(uint32_t v) { return v ^ (((v >> 5) ^ (v >> 10)) & 31u); }

struct BpRow {  // one row's epilogue
    float *rc, *rn, *c_next;
    double epsilon, inv_n;
    bool write, reduce;
    double err;
    uint32_t active;
    __device__ __forceinline__ void operator()(uint2 row, float sum) {
        const float next = __fadd_rn(1.0f - 0.85f, __fmul_rn(0.85f, sum));
        if (row.y) c_next[bp_place(row.x)] = __fdiv_rn(next, (float)row.y);
        if (write) {
            if (reduce) {
                const double d = (double)fabsf(__fsub_rn(next, rc[row.x]));
                err += d * inv_n;
                active += d >= epsilon ? 1u : 0u;
            }
            rn[row.x] = next;
        }
    }
};

// Shared memory of the parts' ends: a row begun in an earlier part and ended
// here leaves its piece in head; what follows the part's last row end (or the
// whole part) in tail. Pieces of the largest rows meet here: joined in 64 bits,
// the sum is rounded once.
struct BpEnds {
    double head[kBpWarps], tail[kBpWarps];
    uint32_t has_end[kBpWarps];
};

// This warp's part of one sweep. kShort: 16-bit words.
//
// The open row -- the one whose end is not reached yet -- is held as `carry`
// (its edges in the group where it began) and, for groups without any row end,
// a compensated sum per lane; a long row therefore costs no scan until its
// end, where the lanes are joined in 64 bits. What decides when an iteration
// stops is the ranks of the largest rows: their sums are rounded once.
template <bool kShort>
__device__ __forceinline__ void bp_sweep(const uint4 *words, uint2 start, uint32_t e1, const uint2 *rows, const float *c,
                                         float *buf, BpEnds &ends_of, BpRow &epi) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lt = (1u << lane) - 1u;
    const uint32_t e0 = start.x;
    uint32_t row = start.y & 0x7FFFFFFFu, pending = 0;
    bool cut = start.y >> 31, any = false, spread = false;  // spread: the lanes hold some of the open row
    float carry = 0.f, ls = 0.f, lc = 0.f;
    constexpr uint32_t kPerLane = kShort ? 1 : 2;  // 16-byte loads per group
    const uint4 *w = words + (size_t)(e0 / 8 + lane) * kPerLane;
    uint4 ahead[kPerLane];
    if (e0 < e1) {
#pragma unroll
        for (uint32_t i = 0; i < kPerLane; ++i) ahead[i] = __ldcs(w + i);
    }
    for (uint32_t at = e0; at < e1; at += 256) {
        uint32_t id[8], ends;
        if constexpr (kShort) {
            const uint4 x = ahead[0];
            id[0] = x.x & 0x7FFFu, id[1] = (x.x >> 16) & 0x7FFFu;
            id[2] = x.y & 0x7FFFu, id[3] = (x.y >> 16) & 0x7FFFu;
            id[4] = x.z & 0x7FFFu, id[5] = (x.z >> 16) & 0x7FFFu;
            id[6] = x.w & 0x7FFFu, id[7] = (x.w >> 16) & 0x7FFFu;
            // flags of word i to bits 2i and 2i + 16, the upper ones then down to 2i + 1
            const uint32_t f = ((x.x & 0x80008000u) >> 15) | ((x.y & 0x80008000u) >> 13) |
                               ((x.z & 0x80008000u) >> 11) | ((x.w & 0x80008000u) >> 9);
            ends = (f | (f >> 15)) & 0xFFu;
        } else {
            const uint4 x = ahead[0], y = ahead[kPerLane - 1];
            const uint32_t z[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
            ends = 0;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                id[k] = z[k] & 0x7FFFFFFFu;
                ends |= (z[k] >> 31) << k;
            }
        }
        w += 32 * kPerLane;
        const uint32_t left = e1 - at;
        if (left > 256) {
#pragma unroll
            for (uint32_t i = 0; i < kPerLane; ++i) ahead[i] = __ldcs(w + i);
        }
        float x[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) x[k] = c[id[k]];
        if (left < 256) {  // words past the stream's end are vertex 0 without a row end
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (lane * 8 + k >= left) x[k] = 0.f;
        }
        const unsigned m = __ballot_sync(0xffffffffu, ends != 0);
        if (m == 0) {
            float acc = x[0];
#pragma unroll
            for (int k = 1; k < 8; ++k) acc = __fadd_rn(acc, x[k]);
            kahan_add(ls, lc, acc);
            spread = true;
            continue;
        }
        // where this lane's row sums go
        const uint32_t mine = __popc(ends);
        uint32_t upto = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= (uint32_t)o) upto += t;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, upto, 31);
        float *out = buf + pending + upto - mine;
        float *const first_out = out;
        float acc = 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            acc = __fadd_rn(acc, x[k]);
            if ((ends >> k) & 1u) {
                *out++ = acc;
                acc = 0.f;
            }
        }
        const float scan = segmented_scan(acc, ends != 0);
        float in = __shfl_up_sync(0xffffffffu, scan, 1);
        if (lane == 0) in = 0.f;
        double open = 0.0;  // the open row's earlier groups
        if (spread) open = warp_sum((double)ls - (double)lc);
        if (ends) {
            const float sum = __fadd_rn(in, *first_out);
            if (m & lt) {
                *first_out = sum;
            } else if (spread || cut) {
                const double whole = open + (double)carry + (double)in + (double)*first_out;
                *first_out = __double2float_rn(whole);
                if (cut) ends_of.head[warp] = whole;
            } else {
                *first_out = __fadd_rn(sum, carry);
            }
        }
        carry = __shfl_sync(0xffffffffu, scan, 31);
        ls = lc = 0.f;
        spread = false;
        any = true;
        __syncwarp();
        pending += total;
        uint32_t first = cut;
        row += first;
        cut = false;
        for (; pending - first >= 32; first += 32, row += 32) epi(__ldg(rows + row + lane), buf[first + lane]);
        if (first) {
            pending -= first;
            const float t = lane < pending ? buf[first + lane] : 0.f;
            __syncwarp();
            if (lane < pending) buf[lane] = t;
        }
        __syncwarp();
    }
    if (lane < pending) epi(__ldg(rows + row + lane), buf[lane]);
    double tail = (double)carry;
    if (spread) tail += warp_sum((double)ls - (double)lc);
    if (lane == 0) {
        ends_of.tail[warp] = tail;
        ends_of.has_end[warp] = any;
    }
    __syncwarp();
}

__global__ void __launch_bounds__(kBpThreads, 1) pr_batched_kernel(BpArgs a) {
    extern __shared__ __align__(16) float s_mem[];  // contributions [smem_v], pending row sums
    __shared__ BpEnds s_ends;
    __shared__ uint32_t s_slot, s_active;
    __shared__ double s_err;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float *buf = s_mem + a.smem_v + warp * kBpBuf;
    const float base = 1.0f - 0.85f;
    const bool can_stop = a.epsilon > 0.0;
    for (;;) {
        const uint32_t g = bb_next_graph(a.cursor, a.G, a.order, &s_slot);
        if (g == 0xFFFFFFFFu) break;
        const uint32_t vb = a.vbase[g], Vg = a.vbase[g + 1] - vb;
        const uint32_t *off = a.off + vb;
        const uint4 *words = a.words + a.wbase[g];
        const uint2 *rows = a.rows + vb;
        const uint2 start = a.starts[g * kBpStarts + warp];
        const uint32_t stop = a.starts[g * kBpStarts + warp + 1].x;
        // lane i of warp 0 finishes the row that the end of part i - 1 cuts
        const uint32_t part = a.starts[g * kBpStarts + lane].y;
        const uint2 part_row = part >> 31 ? rows[part & 0x7FFFFFFFu] : make_uint2(0u, 0u);
        // contributions: two buffers in shared memory, or one there and the
        // next ones in global memory, or both in global memory
        const uint32_t room = (Vg + 31) & ~31u;
        const bool in_smem = room <= a.smem_v, both = 2 * room <= a.smem_v;
        float *c = in_smem ? s_mem : a.scratch + (size_t)blockIdx.x * a.max_v;
        float *cn = both ? s_mem + room : a.next + (size_t)blockIdx.x * a.max_v;
        uint32_t cur = 0;  // c within s_mem, where it is there
        float *rc = a.ranks + vb, *rn = a.rother + vb;
        for (uint32_t v = threadIdx.x; v < Vg; v += blockDim.x) {
            rc[v] = rn[v] = base;  // rows without in-edges keep it
            const uint32_t d = off[v + 1] - off[v];
            c[bp_place(v)] = cn[bp_place(v)] = d ? __fdiv_rn(base, (float)d) : 0.0f;
        }
        if (threadIdx.x == 0) {
            s_active = 0;
            s_err = 0.0;
        }
        __syncthreads();
        uint32_t k = a.max_it, executed = 0, active_last = 0;
        double err_last = 0.0;
        for (uint32_t it = 0; it < a.max_it; ++it) {
            // with epsilon = 0 only the last iteration's residual is asked
            // for, and ranks are written in the last two
            const bool reduce = can_stop || it + 1 == a.max_it;
            BpRow epi{rc, rn, cn, a.epsilon, 1.0 / (double)Vg, reduce || it + 2 == a.max_it, reduce, 0.0, 0u};
            if (in_smem && Vg <= kBpShortV)
                bp_sweep<true>(words, start, stop, rows, s_mem + cur, buf, s_ends, epi);
            else if (in_smem)
                bp_sweep<false>(words, start, stop, rows, s_mem + cur, buf, s_ends, epi);
            else
                bp_sweep<false>(words, start, stop, rows, c, buf, s_ends, epi);
            __syncthreads();
            if (warp == 0) {  // rows cut by a part's end
                const bool cut = part >> 31, ended = s_ends.has_end[lane];
                const double scan = segmented_scan(s_ends.tail[lane], ended || !cut);
                const double in = __shfl_up_sync(0xffffffffu, scan, 1);
                if (cut && ended)
                    epi(part_row, __double2float_rn(in + s_ends.head[lane]));
            }
            if (reduce) {
                const double err = warp_sum(epi.err);
                const uint32_t active = warp_sum(epi.active);
                if (lane == 0) {
                    atomicAdd(&s_err, err);
                    atomicAdd(&s_active, active);
                }
            }
            __syncthreads();
            if (both || !in_smem) {
                float *t = c;
                c = cn;
                cn = t;
                cur = room - cur;
            } else {
                for (uint32_t i = threadIdx.x; i < room / 4; i += blockDim.x)
                    reinterpret_cast<float4 *>(c)[i] = reinterpret_cast<const float4 *>(cn)[i];
            }
            float *t = rc;
            rc = rn;
            rn = t;
            executed = it + 1;
            if (!both && in_smem) __syncthreads();  // the copy
            if (reduce) {
                active_last = can_stop ? s_active : Vg;
                err_last = s_err;
                __syncthreads();
                if (can_stop && active_last == 0) {
                    k = it;
                    break;
                }
                if (threadIdx.x == 0) {
                    s_active = 0;
                    s_err = 0.0;
                }
                __syncthreads();
            }
        }
        // final ranks / N into the output buffer
        float *out = a.ranks + vb;
        const float nf = (float)Vg;
        for (uint32_t v = threadIdx.x; v < Vg; v += blockDim.x) out[v] = __fdiv_rn(rc[v], nf);
        if (threadIdx.x == 0 && a.res) {
            gbx_pr_result r;
            r.iterations = k;
            r.active_last = executed ? active_last : 0;
            r.error_total = executed ? err_last : 0.0;
            a.res[g] = r;
        }
    }
}

// first_edge[g]: graph g's first in-edge; first_edge[G]: past the last graph's
__global__ void bp_bounds_kernel(const uint32_t *vbase, uint32_t G, const uint32_t *poff, uint32_t *first_edge) {
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g <= G; g += gridDim.x * blockDim.x)
        first_edge[g] = poff[vbase[g]];
}

// One CTA lays a graph's words out.
__global__ void __launch_bounds__(kBpThreads)
    bp_layout_kernel(uint32_t G, const uint32_t *order, const uint32_t *vbase, const uint32_t *off,
                     const uint32_t *poff, const uint32_t *psrc, const uint32_t *wbase, uint32_t smem_v, uint4 *words,
                     uint2 *rows, uint2 *starts) {
    __shared__ uint32_t s_wsum[kBpWarps], s_base;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint32_t i = blockIdx.x; i < G; i += gridDim.x) {
        const uint32_t g = order[i];
        const uint32_t vb = vbase[g], Vg = vbase[g + 1] - vb;
        const uint32_t *po = poff + vb;
        const uint32_t first = po[0], edges = po[Vg] - first;
        const bool is_short = Vg <= kBpShortV && ((Vg + 31) & ~31u) <= smem_v;
        uint16_t *w16 = reinterpret_cast<uint16_t *>(words + wbase[g]);
        uint32_t *w32 = reinterpret_cast<uint32_t *>(words + wbase[g]);
        if (threadIdx.x == 0) s_base = 0;
        __syncthreads();
        // rows with edges, in order
        for (uint32_t v0 = 0; v0 < Vg; v0 += kBpThreads) {
            const uint32_t v = v0 + threadIdx.x;
            const bool has = v < Vg && po[v + 1] != po[v];
            const unsigned b = __ballot_sync(0xffffffffu, has);
            if (lane == 0) s_wsum[warp] = __popc(b);
            __syncthreads();
            uint32_t p = s_base + __popc(b & ((1u << lane) - 1u));
            for (uint32_t w = 0; w < warp; ++w) p += s_wsum[w];
            if (has) rows[vb + p] = make_uint2(v, off[vb + v + 1] - off[vb + v]);
            __syncthreads();
            if (threadIdx.x == kBpThreads - 1) s_base = p + has;
            __syncthreads();
        }
        const uint32_t rows_g = s_base;
        // words (the stream is padded to whole groups with vertex 0)
        for (uint32_t e = threadIdx.x; e < (edges + 255) / 256 * 256; e += kBpThreads) {
            const uint32_t u = e < edges ? bp_place(psrc[first + e]) : 0u;
            if (is_short) w16[e] = (uint16_t)u; else w32[e] = u;
        }
        __syncthreads();
        for (uint32_t v = threadIdx.x; v < Vg; v += kBpThreads) {
            if (po[v + 1] == po[v]) continue;
            const uint32_t e = po[v + 1] - 1 - first;
            if (is_short) w16[e] |= 0x8000u; else w32[e] |= 0x80000000u;
        }
        // the parts' first edges: part k begins at the first group with at
        // least k / 32 of the cost before it
        const uint32_t groups = (edges + 255) / 256;
        const uint64_t total = (uint64_t)edges + (uint64_t)kBpRowCost * rows_g;
        auto row_at = [&](uint32_t e) {  // the last row that begins at or before e
            uint32_t lo = 0, hi = rows_g;
            while (hi - lo > 1) {
                const uint32_t mid = lo + (hi - lo) / 2;
                if (po[rows[vb + mid].x] - first <= e) lo = mid; else hi = mid;
            }
            return lo;
        };
        for (uint32_t j = threadIdx.x; j <= groups; j += blockDim.x) {
            const uint32_t e = min(j * 256, edges);
            const uint32_t row = j < groups ? row_at(e) : rows_g;
            const uint64_t cost = (uint64_t)e + (uint64_t)kBpRowCost * row;
            const uint64_t before = j ? (uint64_t)(j - 1) * 256 + (uint64_t)kBpRowCost * row_at((j - 1) * 256) : 0;
            for (uint32_t k = 0; k < kBpStarts; ++k) {
                const uint64_t want = total * k / kBpWarps;
                if (cost < want || (j && before >= want)) continue;
                const bool cut = e < edges && po[rows[vb + row].x] - first < e;
                starts[g * kBpStarts + k] = make_uint2(e, e < edges ? row | (cut ? 0x80000000u : 0u) : 0u);
            }
        }
        __syncthreads();
    }
}

// ---- validation ------------------------------------------------------------------
// One block per graph: offsets non-decreasing inside [off[vb], off[vb+Vg]],
// neighbour ids below Vg. Sets *bad on any violation.
__global__ void batch_check_kernel(const uint32_t *vbase, uint32_t G, const uint32_t *off, const uint32_t *ids,
                                   uint32_t E, uint32_t *bad) {
    for (uint32_t g = blockIdx.x; g < G; g += gridDim.x) {
        const uint32_t vb = vbase[g], Vg = vbase[g + 1] - vb;
        for (uint32_t v = threadIdx.x; v < Vg; v += blockDim.x) {
            const uint32_t b = off[vb + v], e = off[vb + v + 1];
            if (e < b || e > E) {
                atomicOr(bad, 1u);
                continue;
            }
            for (uint32_t j = b; j < e; ++j)
                if (ids[j] >= Vg) {
                    atomicOr(bad, 2u);
                    break;
                }
        }
    }
}

}  // namespace gbx

using namespace gbx;

namespace {

template <typename T>
int upload(T **dst, const T *src, size_t n, cudaStream_t s) {
    GBX_CUDA(cudaMalloc(dst, std::max<size_t>(n, 1) * sizeof(T)));
    if (n) GBX_CUDA(cudaMemcpyAsync(*dst, src, n * sizeof(T), cudaMemcpyDefault, s));
    return GBX_OK;
}

template <typename T>
int to_host(std::vector<T> &out, const T *src, size_t n, cudaStream_t s) {
    out.resize(n);
    if (n) GBX_CUDA(cudaMemcpyAsync(out.data(), src, n * sizeof(T), cudaMemcpyDefault, s));
    return GBX_OK;
}

int batch_create(gbx_batch *b, uint32_t G, const uint32_t *vertex_base, const uint32_t *offsets,
                 const uint32_t *dest, const uint32_t *in_offsets, const uint32_t *in_src, cudaStream_t s) {
    std::vector<uint32_t> vb;
    GBX_TRY(to_host(vb, vertex_base, (size_t)G + 1, s));
    GBX_CUDA(cudaStreamSynchronize(s));
    GBX_REQUIRE(vb[0] == 0, GBX_ERR_INVALID, "vertex_base[0] must be 0");
    for (uint32_t g = 0; g < G; ++g)
        GBX_REQUIRE(vb[g + 1] > vb[g], GBX_ERR_INVALID, "graph %u has no vertices", g);
    const uint32_t V = vb[G];
    std::vector<uint32_t> off;
    GBX_TRY(to_host(off, offsets, (size_t)V + 1, s));
    GBX_CUDA(cudaStreamSynchronize(s));
    GBX_REQUIRE(off[0] == 0, GBX_ERR_INVALID, "offsets[0] must be 0");
    const uint32_t E = off[V];
    b->G = G;
    b->V = V;
    b->E = E;
    std::vector<uint32_t> order(G);
    std::vector<uint64_t> eg(G);
    for (uint32_t g = 0; g < G; ++g) {
        eg[g] = (uint64_t)(off[vb[g + 1]] - off[vb[g]]) + (vb[g + 1] - vb[g]);
        b->max_v = std::max(b->max_v, vb[g + 1] - vb[g]);
    }
    std::iota(order.begin(), order.end(), 0u);
    std::stable_sort(order.begin(), order.end(), [&](uint32_t x, uint32_t y) { return eg[x] > eg[y]; });
    GBX_REQUIRE(dest || E == 0, GBX_ERR_INVALID, "dest is NULL");
    GBX_TRY(upload(&b->vbase, vb.data(), vb.size(), s));
    GBX_TRY(upload(&b->offsets, off.data(), off.size(), s));
    GBX_TRY(upload(&b->dest, dest, E, s));
    GBX_TRY(upload(&b->order, order.data(), order.size(), s));
    if (in_offsets) {
        GBX_REQUIRE(in_src || E == 0, GBX_ERR_INVALID, "in_offsets without in_src");
        GBX_TRY(upload(&b->in_offsets, in_offsets, (size_t)V + 1, s));
        GBX_TRY(upload(&b->in_src, in_src, E, s));
    }
    DevBuf<uint32_t> bad;
    GBX_TRY(bad.alloc(1, s));
    GBX_CUDA(cudaMemsetAsync(bad.p, 0, 4, s));
    const unsigned grid = std::max(1u, std::min<unsigned>(G, (unsigned)num_sms() * 16));
    batch_check_kernel<<<grid, 256, 0, s>>>(b->vbase, G, b->offsets, b->dest, E, bad.p);
    GBX_LAUNCH_CHECK();
    if (b->in_offsets) {
        batch_check_kernel<<<grid, 256, 0, s>>>(b->vbase, G, b->in_offsets, b->in_src, E, bad.p);
        GBX_LAUNCH_CHECK();
    }
    uint32_t hbad = 0;
    GBX_CUDA(cudaMemcpyAsync(&hbad, bad.p, 4, cudaMemcpyDeviceToHost, s));
    GBX_CUDA(cudaStreamSynchronize(s));
    b->h_vbase = std::move(vb);
    GBX_REQUIRE(hbad == 0, GBX_ERR_INVALID, "packed CSR rejected: %s",
                (hbad & 1) ? "offsets decrease or exceed the edge count" : "a neighbour id is not below its graph's vertex count");
    return GBX_OK;
}

void batch_free(gbx_batch *b) {
    cudaFree(b->vbase);
    cudaFree(b->offsets);
    cudaFree(b->dest);
    cudaFree(b->in_offsets);
    cudaFree(b->in_src);
    cudaFree(b->order);
    dev_free(b->words);
    dev_free(b->wbase);
    dev_free(b->rows);
    dev_free(b->starts);
    delete b;
}

// Shared memory of pr_batched_kernel: contributions (room for two buffers of
// the largest graph where that fits) and the warps' pending row sums.
uint32_t bp_smem_v(const gbx_batch *b) {
    const uint32_t room = (b->max_v + 31) & ~31u;
    return std::min(kBpSmemV, 2 * (uint64_t)room <= kBpSmemV ? 2 * room : room);
}

// The word layout, complete on return (any stream may use it).
int bp_layout(gbx_batch *b, cudaStream_t s) {
    std::lock_guard<std::mutex> lock(b->words_mutex);
    if (b->starts) return GBX_OK;
    const uint32_t smem_v = bp_smem_v(b);
    // The words are the in-edges, which a graph may have more or fewer of than
    // out-edges: a caller's in-edge CSR need not be the forward one's transpose.
    std::vector<uint32_t> first_edge((size_t)b->G + 1);
    DevBuf<uint32_t> bounds;
    GBX_TRY(bounds.alloc(first_edge.size(), s));
    bp_bounds_kernel<<<std::min<unsigned>(ceil_div(first_edge.size(), 256), (unsigned)num_sms() * 8), 256, 0, s>>>(
        b->vbase, b->G, b->poff(), bounds.p);
    GBX_LAUNCH_CHECK();
    GBX_CUDA(cudaMemcpyAsync(first_edge.data(), bounds.p, first_edge.size() * 4, cudaMemcpyDeviceToHost, s));
    GBX_CUDA(cudaStreamSynchronize(s));
    std::vector<uint32_t> wbase(b->G);
    uint64_t at = 0;
    for (uint32_t g = 0; g < b->G; ++g) {
        const uint32_t v = b->h_vbase[g + 1] - b->h_vbase[g], edges = first_edge[g + 1] - first_edge[g];
        wbase[g] = (uint32_t)at;
        at += ((uint64_t)edges + 255) / 256 * (v <= kBpShortV && ((v + 31) & ~31u) <= smem_v ? 32 : 64);
    }
    auto build = [&]() -> int {
        GBX_TRY(dev_alloc((void **)&b->words, std::max<uint64_t>(at, 1) * sizeof(uint4), s));
        GBX_TRY(dev_alloc((void **)&b->wbase, (size_t)b->G * 4, s));
        GBX_TRY(dev_alloc((void **)&b->rows, (size_t)b->V * sizeof(uint2), s));
        uint2 *starts = nullptr;
        GBX_TRY(dev_alloc((void **)&starts, (size_t)b->G * kBpStarts * sizeof(uint2), s));
        b->starts = starts;
        GBX_CUDA(cudaMemcpyAsync(b->wbase, wbase.data(), (size_t)b->G * 4, cudaMemcpyHostToDevice, s));
        const unsigned grid = std::min<unsigned>(b->G, (unsigned)num_sms() * 2);
        bp_layout_kernel<<<grid, kBpThreads, 0, s>>>(b->G, b->order, b->vbase, b->offsets, b->poff(), b->psrc(), b->wbase, smem_v,
                                              b->words, b->rows, b->starts);
        GBX_LAUNCH_CHECK();
        GBX_CUDA(cudaStreamSynchronize(s));
        return GBX_OK;
    };
    const int st = build();
    if (st != GBX_OK) {
        cudaStreamSynchronize(s);
        dev_free(b->words);
        dev_free(b->wbase);
        dev_free(b->rows);
        dev_free(b->starts);
        b->words = nullptr;
        b->wbase = nullptr;
        b->rows = b->starts = nullptr;
    }
    return st;
}

}  // namespace

extern "C" int gbx_batch_create(gbx_batch **out, uint32_t num_graphs, const uint32_t *vertex_base,
                                const uint32_t *offsets, const uint32_t *dest, const uint32_t *in_offsets,
                                const uint32_t *in_src, void *stream) {
    clear_error();
    GBX_REQUIRE(out, GBX_ERR_INVALID, "out is NULL");
    *out = nullptr;
    GBX_REQUIRE(num_graphs > 0 && vertex_base && offsets, GBX_ERR_INVALID, "empty batch or NULL tables");
    GBX_TRY(ensure_device());
    gbx_batch *b = new gbx_batch();
    cudaGetDevice(&b->device);
    const int st = batch_create(b, num_graphs, vertex_base, offsets, dest, in_offsets, in_src, (cudaStream_t)stream);
    if (st != GBX_OK) {
        cudaStreamSynchronize((cudaStream_t)stream);
        batch_free(b);
        return st;
    }
    *out = b;
    return GBX_OK;
}

extern "C" int gbx_batch_destroy(gbx_batch *b) {
    clear_error();
    if (!b) return GBX_OK;
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(b->device);
    cudaDeviceSynchronize();
    batch_free(b);
    cudaSetDevice(prev);
    return GBX_OK;
}

extern "C" int gbx_batch_info(const gbx_batch *b, uint32_t *num_graphs, uint32_t *num_vertices,
                              uint32_t *num_edges) {
    clear_error();
    GBX_REQUIRE(b, GBX_ERR_INVALID, "batch is NULL");
    if (num_graphs) *num_graphs = b->G;
    if (num_vertices) *num_vertices = b->V;
    if (num_edges) *num_edges = b->E;
    return GBX_OK;
}

extern "C" int gbx_bfs_batched(gbx_batch *b, const uint32_t *sources, uint32_t *distances, int32_t *parents,
                               gbx_bfs_result *results, void *stream) {
    clear_error();
    GBX_REQUIRE(b && sources && distances, GBX_ERR_INVALID, "batch, sources or distances is NULL");
    GBX_TRY(ensure_device());
    cudaStream_t s = (cudaStream_t)stream;
    std::vector<uint32_t> hs;
    GBX_TRY(to_host(hs, sources, b->G, s));
    GBX_CUDA(cudaStreamSynchronize(s));
    const std::vector<uint32_t> &vb = b->h_vbase;
    for (uint32_t g = 0; g < b->G; ++g)
        GBX_REQUIRE(hs[g] < vb[g + 1] - vb[g], GBX_ERR_INVALID, "source %u of graph %u is not below its %u vertices",
                    hs[g], g, vb[g + 1] - vb[g]);
    InArray<uint32_t> src_d;
    GBX_TRY(src_d.bind(sources, b->G, s));
    OutArray<uint32_t> dist;
    OutArray<int32_t> par;
    OutArray<gbx_bfs_result> res;
    GBX_TRY(dist.bind(distances, b->V, s));
    GBX_TRY(par.bind(parents, b->V, s));
    GBX_TRY(res.bind(results, b->G, s));
    DevBuf<uint32_t> cursor, scratch;
    GBX_TRY(cursor.alloc(1, s));
    GBX_CUDA(cudaMemsetAsync(cursor.p, 0, 4, s));
    const size_t smem = (size_t)3 * kBbWordsCap * sizeof(uint32_t);
    GBX_CUDA(cudaFuncSetAttribute(bfs_batched_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int occ = 0;
    GBX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, bfs_batched_kernel, kBbThreads, smem));
    const unsigned grid = std::max(1u, std::min<unsigned>((unsigned)num_sms() * std::max(occ, 1), b->G));
    const uint32_t words_max = (b->max_v + 31) / 32;
    BbArgs a;
    a.scratch_words = 0;
    a.scratch = nullptr;
    if (words_max > kBbWordsCap) {
        a.scratch_words = words_max;
        GBX_TRY(scratch.alloc((size_t)grid * 3 * words_max, s));
        a.scratch = scratch.p;
    }
    a.G = b->G;
    a.vbase = b->vbase;
    a.off = b->offsets;
    a.dest = b->dest;
    a.poff = b->poff();
    a.psrc = b->psrc();
    a.order = b->order;
    a.sources = src_d.d;
    a.dist = dist.d;
    a.parent = par.d;
    a.res = res.d;
    a.cursor = cursor.p;
    a.alpha = 15;
    a.beta = 18;
    bfs_batched_kernel<<<grid, kBbThreads, smem, s>>>(a);
    GBX_LAUNCH_CHECK();
    GBX_TRY(dist.finish(s));
    GBX_TRY(par.finish(s));
    GBX_TRY(res.finish(s));
    GBX_CUDA(cudaStreamSynchronize(s));
    return GBX_OK;
}

extern "C" int gbx_pr_batched(gbx_batch *b, uint32_t max_iterations, double epsilon, float *ranks,
                              gbx_pr_result *results, void *stream) {
    clear_error();
    GBX_REQUIRE(b && ranks, GBX_ERR_INVALID, "batch or ranks is NULL");
    GBX_REQUIRE(epsilon >= 0.0, GBX_ERR_INVALID, "epsilon must be >= 0");
    GBX_TRY(ensure_device());
    cudaStream_t s = (cudaStream_t)stream;
    GBX_TRY(bp_layout(b, s));
    OutArray<float> out;
    OutArray<gbx_pr_result> res;
    GBX_TRY(out.bind(ranks, b->V, s));
    GBX_TRY(res.bind(results, b->G, s));
    DevBuf<float> other, next, scratch;
    DevBuf<uint32_t> cursor;
    GBX_TRY(other.alloc(b->V, s));
    GBX_TRY(cursor.alloc(1, s));
    GBX_CUDA(cudaMemsetAsync(cursor.p, 0, 4, s));
    const uint32_t smem_v = bp_smem_v(b), room = (b->max_v + 31) & ~31u;
    const size_t smem = ((size_t)smem_v + kBpWarps * kBpBuf) * sizeof(float);
    // the limit holds for the process: always the most that any batch takes
    GBX_CUDA(cudaFuncSetAttribute(pr_batched_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)((kBpSmemV + kBpWarps * kBpBuf) * sizeof(float))));
    const unsigned grid = std::min<unsigned>((unsigned)num_sms(), b->G);
    if (2 * (uint64_t)room > smem_v) GBX_TRY(next.alloc((size_t)grid * room, s));
    if (room > smem_v) GBX_TRY(scratch.alloc((size_t)grid * room, s));
    BpArgs a;
    a.G = b->G;
    a.vbase = b->vbase;
    a.off = b->offsets;
    a.order = b->order;
    a.words = b->words;
    a.wbase = b->wbase;
    a.starts = b->starts;
    a.rows = b->rows;
    a.ranks = out.d;
    a.rother = other.p;
    a.next = next.p;
    a.scratch = scratch.p;
    a.max_v = room;
    a.smem_v = smem_v;
    a.cursor = cursor.p;
    a.max_it = max_iterations;
    a.epsilon = epsilon;
    a.res = res.d;
    pr_batched_kernel<<<grid, kBpThreads, smem, s>>>(a);
    GBX_LAUNCH_CHECK();
    GBX_TRY(out.finish(s));
    GBX_TRY(res.finish(s));
    GBX_CUDA(cudaStreamSynchronize(s));
    return GBX_OK;
}
