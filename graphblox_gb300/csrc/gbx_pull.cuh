// Hot-table pull engine: the repeated form of the pull sweep of
// gbx_gather.cuh. Which of the two a graph gets depends on the graph alone
// (get_pull_layout), so that equal calls give equal bits whatever was called
// before them.
//
// What bounds a pull sweep is the gather of one 4-byte value per edge. An
// access that misses L1 costs one 32-byte sector from L2, and an SM gets one
// sector per cycle whatever the table's size and the loads in flight: 297 G
// random loads/s on 152 SMs, measured with tables of 1 to 64 MB. The row
// engine reaches 150-210 G edges/s of it: its warps wait for the words of
// their edges, then for the gathers, then add up. Two things differ here.
//
// Work is cut by edges, not by rows: a unit is a run of up to `span` edges of
// the pull order, and the last edge of every row carries a flag, so a unit
// needs no row offsets and no search. A lane takes four consecutive edges from
// one 16-byte load, adds up its row pieces, and a segmented scan over the warp
// joins them; row sums collect in shared memory and leave 32 at a time through
// the epilogue. That leaves registers to keep three groups of 128 edges under
// way per warp: one being added up, one being gathered, one whose words are on
// their way.
//
// Few sources make up much of a skewed graph's edges. The kHotMax most used
// get a slot, an edge's word carries the slot instead of the vertex id, and
// each SM keeps the slots' values in shared memory (RMAT-22: 20,000 of 4.2M
// vertices cover 43% of the edges). More slots cover more edges but leave L1
// less room, and every miss in flight holds a sector of it: a sweep of RMAT-22
// takes 236 us without slots, 188 with 16,000, 184 with 20,000, 178 with
// 28,000, 198 with 40,000 and 316 with 52,000; SpMV over a crawl graph, whose
// ids are local and hit L1, 416, 433, 430, 459, 629 and 1055 us (both with
// plain additions).
//
// Rows of up to `span` edges lie in one unit; longer rows are cut where a unit
// begins, each piece leaves a partial sum, and the warp that brings the last
// one adds them up in order (compensated per lane) and runs the epilogue. Every
// order of additions is fixed by the layout: results repeat bit for bit. Rows
// without edges are in no unit.
//
// Against the row engine (RMAT-22, 65M edges): a PageRank iteration 332 -> 187
// us, SpMV 453 -> 229 us; SpMV over 142M crawl edges 641 -> 458 us.
#pragma once

#include <algorithm>

#include "gbx_coop.cuh"
#include "gbx_gather.cuh"

// edge words
constexpr uint32_t kPullLast = 0x80000000u;  // last edge of its row
constexpr uint32_t kPullHot = 0x40000000u;   // the rest is a slot, not a vertex

struct gbx_pull_layout {
    uint32_t V = 0, E = 0;
    uint32_t hot = 0;                // slots, a multiple of 4
    uint32_t n_rows = 0;             // rows with edges
    // Units: the first `big` of span edges, the others of tail_span
    uint32_t n_units = 0, big = 0, span = 0, tail_span = 0;
    uint32_t *edges = nullptr;       // device [E + kPullPad]: edge words
    uint32_t *hot_ids = nullptr;     // device [hot]: vertex of a slot, ~0 for an unused one
    uint2 *rows = nullptr;           // device [n_rows]: {vertex, its slot or ~0}
    // device [n_units + 1]: {first edge, row of that edge, the unit where that
    // row begins when it is cut (else ~0), units of the cut row}
    uint4 *units = nullptr;
    // device [pull_work_words]: working memory of captured SpMV calls (the
    // graph that a capture makes outlives any allocation of the call)
    float *work = nullptr;
    // PageRank's, allocated here so that a graph that has a layout lacks
    // nothing: device [n_rows] out-degrees in row order, piece sums
    // [2 * n_units] and tickets [n_units], zero between sweeps
    uint32_t *row_degree = nullptr;
    float *sums = nullptr;
    unsigned *tickets = nullptr;
};

__host__ __device__ inline uint32_t pull_unit_edge(const gbx_pull_layout &l, uint32_t t) {
    return t <= l.big ? t * l.span : l.big * l.span + (t - l.big) * l.tail_span;
}
__host__ __device__ inline uint32_t pull_unit_of(const gbx_pull_layout &l, uint32_t e) {
    return e < l.big * l.span ? e / l.span : l.big + (e - l.big * l.span) / l.tail_span;
}

namespace gbx {

constexpr int kPullThreads = 1024;      // one CTA per SM, 64 registers per thread
constexpr int kPullWarps = kPullThreads / 32;
constexpr uint32_t kPullPad = 512;      // readable words past the last edge
constexpr uint32_t kPullBuf = 160;      // pending row sums of a warp: fewer than 32, and a group's 128
constexpr uint32_t kHotMax = 20000;     // 80 KB of slots beside 20 KB of pending sums
// Edges per unit: a unit costs a chain of three loads before its first
// additions (RMAT-22, PageRank iteration: 1280 193 us, 2048 181, 3072 178).
constexpr uint32_t kPullSpanMax = 3072;

// shared memory: the slots, four zeros (the first is the value of no edge),
// the warps' pending sums
constexpr size_t pull_smem_of(uint32_t hot) { return ((size_t)hot + 4 + kPullWarps * kPullBuf) * sizeof(float); }
inline size_t pull_smem(const gbx_pull_layout &l) { return pull_smem_of(l.hot); }
// A kernel's limit on dynamic shared memory holds for the process: it is
// always set to the most that any layout takes, so that no thread lowers it
// between another one's setting and launch.
constexpr int kPullSmemLimit = (int)pull_smem_of(kHotMax);

// A running sum and the errors of its additions: of any two numbers (Knuth
// 1969, two-sum), or in half the instructions where the sum mostly is the
// larger one (Kahan 1965). Past an infinity the errors are not finite and
// the plain sum is the value.
struct PullSum {
    float s = 0.f, err = 0.f;
    __device__ __forceinline__ void add(float x) {
        const float t = __fadd_rn(s, x), y = __fsub_rn(t, s);
        err = __fadd_rn(err, __fadd_rn(__fsub_rn(s, __fsub_rn(t, y)), __fsub_rn(x, y)));
        s = t;
    }
    __device__ __forceinline__ void add_small(float x) {
        const float t = __fadd_rn(s, x);
        err = __fadd_rn(err, __fsub_rn(x, __fsub_rn(t, s)));
        s = t;
    }
    __device__ __forceinline__ float value() const { return fabsf(err) < INFINITY ? __fadd_rn(s, err) : s; }
};

// Memory of one sweep in flight: piece sums [2 * units] and tickets [units]
// (zero between sweeps).
struct PullPieces {
    float *sums;
    unsigned *tickets;
};

// Working memory of SpMV sweeps, one run of words: the slots' values, piece
// sums, then tickets and cursors (zeroed by the call).
constexpr uint32_t kPullCursors = 64;
inline size_t pull_work_words(const gbx_pull_layout &l) {
    return (size_t)std::max(l.hot, 4u) + 3 * (size_t)l.n_units + kPullCursors;
}

// Term:  const float *cold            values by vertex
//        struct Factors; void factors(uint32_t e, uint32_t e0, uint32_t e1, Factors &)   of edges e..e+3
//        void scale(const Factors &, float (&v)[4])
// Epi:   void prefetch(uint32_t row)
//        void operator()(uint32_t row, uint32_t v, uint32_t slot, float sum)   once per row with edges
template <class Term, class Epi>
struct PullSweep {
    const gbx_pull_layout &l;
    uint32_t s_hot;  // shared-memory address of the slots
    float *buf;      // this warp's pending sums
    const Term &term;
    Epi &epi;
    PullPieces pieces;

    // up to 32 rows from `row` on leave through the epilogue
    __device__ __forceinline__ void emit(uint32_t row, const float *sums, uint32_t n) {
        const uint32_t lane = threadIdx.x & 31;
        if (lane < n) {
            const uint2 r = __ldg(l.rows + row + lane);
            epi(row + lane, r.x, r.y, sums[lane]);
        }
    }

    // one more piece of a cut row: the warp that brings the last one finishes it
    __device__ __forceinline__ void piece(uint32_t slot, float sum, uint32_t first, uint32_t count, uint32_t row) {
        const uint32_t lane = threadIdx.x & 31;
        unsigned t = 0;
        if (lane == 0) {
            // what the epilogue reads, while the ticket is on its way
            asm volatile("prefetch.global.L1 [%0];" ::"l"(l.rows + row));
            epi.prefetch(row);
            // release: the sum is visible before the ticket; acquire: the
            // last one sees every sum (the shuffle hands that to the warp)
            pieces.sums[slot] = sum;
            asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;"
                         : "=r"(t)
                         : "l"(pieces.tickets + first)
                         : "memory");
        }
        t = __shfl_sync(0xffffffffu, t, 0);
        if (t != count - 1) return;
        __syncwarp();
        PullSum k;
        for (uint32_t i = lane; i < count; i += 32)
            k.add(__ldcg(pieces.sums + 2 * (size_t)(first + i) + (i ? 0 : 1)));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float err = __shfl_xor_sync(0xffffffffu, k.err, o);
            k.add(__shfl_xor_sync(0xffffffffu, k.s, o));
            k.err = __fadd_rn(k.err, err);
        }
        const float total = k.value();
        if (lane == 0) {
            const uint2 r = __ldg(l.rows + row);
            epi(row, r.x, r.y, total);
            pieces.tickets[first] = 0;
        }
        __syncwarp();
    }

    // The values and row ends of edges e .. e+3. One of the two loads runs per
    // lane, both into the same register, so nothing waits here.
    __device__ __forceinline__ void gather(uint4 w, uint32_t e, uint32_t e0, uint32_t e1, bool whole, float (&v)[4],
                                           uint32_t &ends) const {
        uint32_t x[4] = {w.x, w.y, w.z, w.w};
        if (!whole) {  // the unit's first or last group: other edges become the zero past the slots
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (e + k < e0 || e + k >= e1) x[k] = kPullHot | l.hot;
        }
        ends = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t id = x[k] & kIdMask;
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "setp.ne.u32 p, %1, 0;\n\t"
                "@p ld.shared.f32 %0, [%2];\n\t"
                "@!p ld.global.f32 %0, [%3];\n\t}"
                : "=f"(v[k])
                : "r"(x[k] & kPullHot), "r"(s_hot + id * 4), "l"(term.cold + id));
            ends |= (x[k] >> 31) << k;
        }
    }

    // A unit's record and first words.
    struct Start {
        uint4 me, next, w0, w1;
    };
    __device__ __forceinline__ Start start(uint32_t u) const {
        Start st;
        st.me = __ldg(l.units + u);
        st.next = __ldg(l.units + u + 1);
        const uint4 *words = reinterpret_cast<const uint4 *>(l.edges) + st.me.x / 4 + (threadIdx.x & 31);
        st.w0 = __ldcs(words);
        st.w1 = __ldcs(words + 32);
        return st;
    }

    // Three groups of 128 edges are under way: one being added up, one whose
    // gathers (and factors) are in flight, one whose words are.
    __device__ __forceinline__ void unit(uint32_t u, const Start &st) {
        const uint32_t lane = threadIdx.x & 31;
        const uint32_t lt = (1u << lane) - 1u;
        const uint4 me = st.me, next = st.next;
        const uint32_t e0 = me.x, e1 = next.x;
        if (e0 == e1) return;  // several units' first edges lie in one short row: the last has it
        uint32_t row = me.y;          // row of the first pending sum
        uint32_t pending = 0;         // sums in buf
        bool cut = me.z != ~0u;       // the first row began in an earlier unit
        PullSum carry;                // the current row's edges of earlier groups
        uint32_t e = (e0 & ~3u) + lane * 4;
        const uint4 *words = reinterpret_cast<const uint4 *>(l.edges) + e / 4;
        float v1[4];
        uint32_t ends1;
        typename Term::Factors f1;
        uint4 w = st.w1;
        // the first rows' descriptions, needed when their sums are complete
        asm volatile("prefetch.global.L1 [%0];" ::"l"(l.rows + min(row + lane, l.n_rows - 1)));
        epi.prefetch(min(row + lane, l.n_rows - 1));
        gather(st.w0, e, e0, e1, e0 == (e0 & ~3u) && e0 + 128 <= e1, v1, ends1);
        term.factors(e, e0, e1, f1);
        for (uint32_t at = e0 & ~3u; at < e1; at += 128) {
            float v[4] = {v1[0], v1[1], v1[2], v1[3]};
            const uint32_t ends = ends1;
            const typename Term::Factors f = f1;
            e += 128;
            words += 32;
            if (at + 128 < e1) {
                const uint4 now = w;
                if (at + 256 < e1) w = __ldcs(words + 32);
                gather(now, e, e0, e1, at + 256 <= e1, v1, ends1);
                term.factors(e, e0, e1, f1);
            }
            term.scale(f, v);
            // this lane's pieces: the sum up to its first row end, sums of
            // rows inside, the sum after its last row end
            PullSum acc, head;
            float done[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (k == 0) acc.s = v[0]; else acc.add_small(v[k]);
                done[k] = acc.s;
                if ((ends >> k) & 1u) {
                    if ((ends & ((1u << k) - 1u)) == 0) head = acc;
                    acc = PullSum();
                }
            }
            // segmented scan of the trailing pieces; a lane with a row end starts a segment
            const unsigned m = __ballot_sync(0xffffffffu, ends != 0);
            const unsigned upto = m & (lt | (1u << lane));
            const uint32_t back = upto ? lane - (31u - __clz(upto)) : lane;
            // (inside 8 lanes: longer chains are joined below)
            float scan = acc.value();
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) {
                const float t = __shfl_up_sync(0xffffffffu, scan, o);
                if ((uint32_t)o <= min(back, lane % 8u)) scan = __fadd_rn(scan, t);
            }
            // the open row's sum after this lane: earlier groups, whole runs
            // of 8 lanes, and the lanes of the lane's own run
            PullSum open;
            if (upto == 0) open = carry;
#pragma unroll
            for (int b = 8; b < 32; b += 8) {
                const float run = __shfl_sync(0xffffffffu, scan, b - 1);
                open.add_small(lane >= (uint32_t)b && (upto >> b) == 0 ? run : 0.f);
            }
            open.add_small(scan);
            if (m) {
                PullSum in;
                in.s = __shfl_up_sync(0xffffffffu, open.s, 1);
                in.err = __shfl_up_sync(0xffffffffu, open.err, 1);
                if (lane == 0) in = carry;
                in.add_small(head.s);
                in.err = __fadd_rn(in.err, head.err);
                // row sums go to buf in row order
                uint32_t pos = pending, total = 0;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const unsigned b = __ballot_sync(0xffffffffu, (ends >> k) & 1u);
                    pos += __popc(b & lt);
                    total += __popc(b);
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if ((ends >> k) & 1u) {
                        buf[pos++] = (ends & ((1u << k) - 1u)) ? done[k] : in.value();
                    }
                }
                __syncwarp();
                pending += total;
                uint32_t start = 0;
                if (cut) {  // the first of them ends a cut row
                    piece(2 * u, buf[0], me.z, me.w, row);
                    cut = false;
                    start = 1;
                    ++row;
                }
                for (; pending - start >= 32; start += 32, row += 32) emit(row, buf + start, 32);
                if (start) {
                    pending -= start;
                    const float t = lane < pending ? buf[start + lane] : 0.f;
                    __syncwarp();
                    if (lane < pending) buf[lane] = t;
                    __syncwarp();
                }
            }
            carry.s = __shfl_sync(0xffffffffu, open.s, 31);
            carry.err = __shfl_sync(0xffffffffu, open.err, 31);
        }
        emit(row, buf, pending);
        row += pending;
        __syncwarp();
        // the last row goes on in the next unit: it began here, or the whole
        // unit lies inside it
        if (next.z != ~0u && (cut || next.z == u))
            piece(cut ? 2 * u : 2 * u + 1, carry.value(), next.z, next.w, row);
    }
};

// Every unit once: a warp's first two are fixed, so that small sweeps take no
// ticket, the others come from the cursor. The next unit is known while one
// is worked on; its record and first edge words are fetched ahead.
// `first`: start() of the warp's first unit, where there is one.
__device__ __forceinline__ uint32_t first_unit() { return (blockIdx.x * blockDim.x + threadIdx.x) >> 5; }

template <class Sweep>
__device__ __forceinline__ void deal_units(Sweep &sweep, unsigned *cursor, typename Sweep::Start first) {
    const gbx_pull_layout &l = sweep.l;
    const uint32_t lane = threadIdx.x & 31, warps = (gridDim.x * blockDim.x) >> 5;
    uint32_t u = first_unit(), next = u + warps;
    while (u < l.n_units) {
        uint32_t ticket = 0;
        if (next < l.n_units) {
            if (lane == 0) {
                ticket = atomicAdd(cursor, 1u);
                asm volatile("prefetch.global.L1 [%0];" ::"l"(l.units + next));
            }
            asm volatile("prefetch.global.L2 [%0];" ::"l"(l.edges + pull_unit_edge(l, next) + lane * 8));
        }
        sweep.unit(u, first);
        u = next;
        if (u >= l.n_units) break;
        first = sweep.start(u);
        next = 2 * warps + __shfl_sync(0xffffffffu, ticket, 0);
    }
}

// this CTA's slot values, by all its threads; ends with a barrier
__device__ __forceinline__ void load_hot(const float *values, uint32_t hot, float *s_hot) {
    const float4 *in = reinterpret_cast<const float4 *>(values);
    for (uint32_t i = threadIdx.x; i < hot / 4; i += blockDim.x) reinterpret_cast<float4 *>(s_hot)[i] = __ldcg(in + i);
    if (threadIdx.x < 4) s_hot[hot + threadIdx.x] = 0.f;
    __syncthreads();
}

// The layout of g's pull CSR, built on first use (not while s captures); *out
// null: the graph's sweeps run on the row engine of gbx_gather.cuh.
int get_pull_layout(gbx_graph *g, cudaStream_t s, gbx_pull_layout **out);

inline int is_capturing(cudaStream_t s, bool *yes) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    GBX_CUDA(cudaStreamIsCapturing(s, &cap));
    *yes = cap != cudaStreamCaptureStatusNone;
    return GBX_OK;
}

}  // namespace gbx
