// Stable LSD radix sort, 8 or 9 bits per pass, one kernel per pass: of (uint32
// key, uint32 value) pairs for the degree reordering (radixSortEdgesByDegree,
// reorder.c:223-269), the in-edge orders and the CSR segments, and of whole
// edges with an optional weight for the CSR build
// (radixSortEdgesBySourceAndDestination, radixsort.c:285-339).
//
// An edge is one 64-bit key, source above destination in `id_bits` bits each,
// so one sort orders by (source, destination) and the edges themselves move:
// nothing is permuted through an index afterwards. The first pass reads the
// caller's arrays, the last one writes them.
//
// One histogram kernel counts the digits of every pass at once. A pass then
// reads and writes each element once: a CTA takes the next tile (tickets are
// given in order, so a tile's predecessors have all started), ranks it stably
// -- a warp owns kSortItems * 32 consecutive elements, 32 at a time with peer
// masks built from ballots --, publishes its digit counts, sorts the tile
// through shared memory and meanwhile adds up the counts of the tiles before
// it (decoupled look-back, Merrill and Garland 2016): each thread owns a digit
// and walks back over its predecessors' published words, four in flight, until
// it meets an inclusive one. Writes leave in digit order, so a digit's
// elements of a tile (12 or 24 on average) are one contiguous run.
//
// Measured on 67M weighted edges (RMAT-22, 44 key bits): 530 us per pass of
// 9 bits (24 bytes an edge: 3.0 TB/s), where a pass over (key, index) pairs
// with a histogram kernel of its own and element-wise scattered writes took
// 1,520 us and the edges and weights were gathered through the index after six
// of them. What bounds a pass is shared by the issue slots (49%) and the
// shared-memory pipe (53%) that rank and stage the tile; HBM is at 45%.
// 512 threads x 12 elements x 2 CTAs per SM: 498 us per 8-bit pass, 384 x 12 x 3
// 518, 256 x 16 x 4 550, 512 x 8 x 3 537, 256 x 12 x 5 566, 1024 x 12 x 1 640;
// match.any in place of the ballots was 15% slower.
#include <algorithm>

#include "gbx_sort.cuh"

namespace gbx {

namespace {

constexpr int kMaxBits = 9;
constexpr uint32_t kMaxRadix = 1u << kMaxBits;
constexpr int kMaxPasses = 8;
constexpr int kSortThreads = 512;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortItems = 12;
constexpr int kSortCtas = 2;  // per SM: 64 registers per thread
constexpr uint32_t kSortTile = kSortThreads * kSortItems;

// Look-back words: count (34 bits), status (2 bits), epoch. A word counts only
// for the pass whose epoch it carries, so one clear serves all passes.
constexpr uint64_t kCountMask = (1ull << 34) - 1;
constexpr int kStatusShift = 34, kEpochShift = 36;
constexpr uint64_t kPartial = 1, kInclusive = 2;
constexpr unsigned kSpinLimit = 1u << 21;  // polls of about 0.5 us before a wait gives up

__device__ __forceinline__ uint64_t ld_relaxed(const uint64_t *p) {
    uint64_t v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed(uint64_t *p, uint64_t v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ uint64_t lookback_word(uint32_t epoch, uint64_t status, uint64_t count) {
    return ((uint64_t)epoch << kEpochShift) | (status << kStatusShift) | count;
}

// Sum of column `col` over the tiles before `tile`. Sets *error and returns 0
// when a wait runs out here or elsewhere.
__device__ uint64_t lookback(const uint64_t *state, uint32_t width, uint32_t col, uint32_t tile, uint32_t epoch,
                             unsigned *error) {
    uint64_t sum = 0;
    int64_t t = (int64_t)tile - 1;
    unsigned spins = 0;
    while (t >= 0) {
        uint64_t w[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) w[q] = t - q >= 0 ? ld_relaxed(state + (uint64_t)(t - q) * width + col) : 0;
        bool moved = false;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if ((uint32_t)(w[q] >> kEpochShift) != epoch) break;
            sum += w[q] & kCountMask;
            if (((w[q] >> kStatusShift) & 3) == kInclusive) return sum;
            --t;
            moved = true;
        }
        if (moved) continue;
        if (++spins > kSpinLimit) atomicExch(error, 1u);
        if ((spins & 255u) == 0 && *(volatile unsigned *)error) return 0;
    }
    return sum;
}

// The same for one column, by a whole warp: 32 predecessors per step.
__device__ uint64_t lookback_warp(const uint64_t *state, uint32_t tile, uint32_t epoch, unsigned *error) {
    const uint32_t lane = threadIdx.x & 31;
    uint64_t sum = 0;
    int64_t t = (int64_t)tile - 1;
    unsigned spins = 0;
    while (t >= 0) {
        const uint64_t w = t >= lane ? ld_relaxed(state + (t - lane)) : lookback_word(epoch, kInclusive, 0);
        const unsigned ready = __ballot_sync(0xffffffffu, (uint32_t)(w >> kEpochShift) == epoch);
        const uint32_t usable = ready == 0xffffffffu ? 32u : (uint32_t)__ffs(~ready) - 1u;
        const unsigned incl =
            __ballot_sync(0xffffffffu, lane < usable && ((w >> kStatusShift) & 3) == kInclusive);
        const uint32_t take = incl ? (uint32_t)__ffs(incl) : usable;
        uint64_t part = lane < take ? w & kCountMask : 0;
        part = warp_sum(part);
        sum += part;
        if (incl) return sum;
        t -= take;
        if (take) continue;
        if (++spins > kSpinLimit && lane == 0) atomicExch(error, 1u);
        if ((spins & 255u) == 0 && __shfl_sync(0xffffffffu, *(volatile unsigned *)error, 0)) return 0;
    }
    return sum;
}

// ---- digit histograms of every pass -----------------------------------------

// hist[k][kMaxRadix] counts the `bits`-bit digits at lo + k * bits
template <typename K>
__device__ __forceinline__ void count_digits(K key, int lo, int bits, int passes, uint32_t (*h)[kMaxRadix]) {
    const uint32_t m = (1u << bits) - 1;
    for (int k = 0; k < passes; ++k) atomicAdd(&h[k][(uint32_t)(key >> (lo + bits * k)) & m], 1u);
}

__device__ __forceinline__ void clear_digits(uint32_t (*h)[kMaxRadix], int passes) {
    for (uint32_t j = threadIdx.x; j < (uint32_t)passes * kMaxRadix; j += blockDim.x) (&h[0][0])[j] = 0;
    __syncthreads();
}

__device__ __forceinline__ void flush_digits(uint32_t (*h)[kMaxRadix], int passes, uint32_t *hist) {
    __syncthreads();
    for (uint32_t j = threadIdx.x; j < (uint32_t)passes * kMaxRadix; j += blockDim.x)
        if (const uint32_t c = (&h[0][0])[j]) atomicAdd(hist + j, c);
}

__global__ void __launch_bounds__(256)
    key_hist_kernel(const uint32_t *__restrict__ keys, uint32_t n, int bits, int passes, uint32_t *hist) {
    __shared__ uint32_t h[4][kMaxRadix];
    clear_digits(h, passes);
    const uint64_t step = (uint64_t)gridDim.x * 256;
    for (uint64_t i = (uint64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += 4 * step) {
        uint32_t k[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) k[q] = i + q * step < n ? keys[i + q * step] : 0u;
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (i + q * step < n) count_digits(k[q], 0, bits, passes, h);
    }
    flush_digits(h, passes, hist);
}

// digits of the packed edges, and the largest ids
__global__ void __launch_bounds__(256)
    edge_hist_kernel(EdgeView e, int id_bits, int lo, int bits, int passes, uint32_t *hist, SortControl *ctl) {
    __shared__ uint32_t h[kMaxPasses][kMaxRadix];
    clear_digits(h, passes);
    uint32_t m = 0, mm = 0;
    const uint64_t step = (uint64_t)gridDim.x * 256;
    for (uint64_t i = (uint64_t)blockIdx.x * 256 + threadIdx.x; i < e.E; i += 4 * step) {
        uint32_t a[4], b[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint64_t j = i + q * step;
            a[q] = j < e.E ? e.src[j] : 0u;
            b[q] = j < e.E ? e.dst[j] : 0u;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (i + q * step >= e.E) continue;
            m = max(m, max(a[q], b[q]));
            mm = max(mm, max(a[q] & kIdMask, b[q] & kIdMask));
            count_digits(((uint64_t)a[q] << id_bits) | b[q], lo, bits, passes, h);
            if (e.symmetric) count_digits(((uint64_t)b[q] << id_bits) | a[q], lo, bits, passes, h);
        }
    }
    m = __reduce_max_sync(0xffffffffu, m);
    mm = __reduce_max_sync(0xffffffffu, mm);
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&ctl->max_id, m);
        atomicMax(&ctl->max_vertex, mm);
    }
    flush_digits(h, passes, hist);
}

// exclusive prefix sums of each pass's counts (one CTA per pass; the counts of
// an 8-bit digit end in zeros)
__global__ void __launch_bounds__(kMaxRadix) digit_base_kernel(uint32_t *hist, uint32_t n, SortControl *ctl) {
    __shared__ uint32_t wsum[kMaxRadix / 32];
    uint32_t *h = hist + blockIdx.x * kMaxRadix;
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t c = h[threadIdx.x];
    if (c == n) atomicOr(&ctl->trivial, 1u << blockIdx.x);
    uint32_t incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += t;
    }
    if (lane == 31) wsum[wid] = incl;
    __syncthreads();
    uint32_t before = 0;
    for (uint32_t w = 0; w < wid; ++w) before += wsum[w];
    h[threadIdx.x] = before + incl - c;
}

// ---- one pass -----------------------------------------------------------------

template <typename K>
struct PassArgs {
    EdgeView edges;        // input of an edge sort's first pass (kin null)
    const K *kin;
    K *kout;               // output; null: the edge arrays below
    uint32_t *src_out, *dst_out;
    const uint32_t *vin;   // values; null in a pair sort: the element's index
    uint32_t *vout;
    uint32_t n;
    int shift, id_bits;
    uint32_t epoch;
    const uint32_t *base;  // first output position of each digit
    uint64_t *state;       // look-back words [tiles][digits]
    unsigned *ticket, *error;
};

// Keys and values of elements first + r * 32 (r < kSortItems); past the end of
// the list: the largest digit, behind every real one. A full tile's loads are
// unconditional, so that they are all in flight together.
__device__ __forceinline__ void load_edges(const PassArgs<uint64_t> &a, uint32_t first, uint32_t left,
                                           uint64_t (&key)[kSortItems]) {
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        key[r] = ~0ull;
        if ((uint32_t)r * 32 >= left) continue;
        const uint32_t i = first + r * 32;
        const bool back = i >= a.edges.E;  // a reversed copy
        const uint32_t j = back ? i - a.edges.E : i;
        const uint32_t s = __ldcs(a.edges.src + j), d = __ldcs(a.edges.dst + j);
        key[r] = back ? ((uint64_t)d << a.id_bits) | s : ((uint64_t)s << a.id_bits) | d;
    }
}
__device__ __forceinline__ void load_edges(const PassArgs<uint32_t> &, uint32_t, uint32_t, uint32_t (&)[kSortItems]) {}

__device__ __forceinline__ uint64_t ld_stream(const uint64_t *p) { return __ldcs((const unsigned long long *)p); }
__device__ __forceinline__ uint32_t ld_stream(const uint32_t *p) { return __ldcs(p); }

template <typename K>
__device__ __forceinline__ void load_keys(const PassArgs<K> &a, uint32_t first, uint32_t left, K (&key)[kSortItems]) {
    if (sizeof(K) == 8 && !a.kin) {
        load_edges(a, first, left, key);
    } else if (left > (kSortItems - 1) * 32u) {
#pragma unroll
        for (int r = 0; r < kSortItems; ++r) key[r] = ld_stream(a.kin + first + r * 32);
    } else {
#pragma unroll
        for (int r = 0; r < kSortItems; ++r) key[r] = r * 32u < left ? ld_stream(a.kin + first + r * 32) : ~K(0);
    }
}

template <typename K>
__device__ __forceinline__ void load_values(const PassArgs<K> &a, uint32_t first, uint32_t left,
                                            uint32_t (&val)[kSortItems]) {
    const bool edges = sizeof(K) == 8 && !a.kin;
    if (!a.vin) {
#pragma unroll
        for (int r = 0; r < kSortItems; ++r) val[r] = first + r * 32;
    } else if (left > (kSortItems - 1) * 32u && !(edges && a.edges.symmetric)) {
#pragma unroll
        for (int r = 0; r < kSortItems; ++r) val[r] = __ldcs(a.vin + first + r * 32);
    } else {
#pragma unroll
        for (int r = 0; r < kSortItems; ++r) {
            const uint32_t i = first + r * 32;
            val[r] = r * 32u < left ? __ldcs(a.vin + (edges && i >= a.edges.E ? i - a.edges.E : i)) : 0u;
        }
    }
}

template <typename K, bool kValues, int kBits>
__global__ void __launch_bounds__(kSortThreads, kSortCtas) radix_pass_kernel(PassArgs<K> a) {
    constexpr uint32_t kRadix = 1u << kBits, kDigit = kRadix - 1;
    static_assert(kRadix <= kSortThreads, "one thread per digit");
    extern __shared__ __align__(16) unsigned char smem[];
    K *skey = reinterpret_cast<K *>(smem);
    uint32_t *sval = reinterpret_cast<uint32_t *>(skey + kSortTile);
    // per-warp digit counts, dead before the tile is staged over them
    uint16_t(*whist)[kRadix] = reinterpret_cast<uint16_t(*)[kRadix]>(smem);
    static_assert(kSortWarps * kRadix * 2 <= kSortTile * sizeof(uint32_t), "counts must fit the staging area");
    __shared__ uint32_t s_goff[kRadix];  // a digit's first output position less its first in the tile
    __shared__ uint32_t s_wsum[kRadix / 32];
    __shared__ uint32_t s_tile, s_stop;
    const uint32_t tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    if (tid == 0) {
        s_tile = atomicAdd(a.ticket, 1u);
        s_stop = 0;
    }
    for (uint32_t j = tid; j < kSortWarps * kRadix / 2; j += kSortThreads) reinterpret_cast<uint32_t *>(smem)[j] = 0;
    __syncthreads();
    const uint32_t tile = s_tile;
    const uint64_t base = (uint64_t)tile * kSortTile;
    const uint32_t valid = (uint32_t)min((uint64_t)kSortTile, a.n - base);
    // this lane's first element, and how far the end of the list is from it
    const uint32_t at = wid * (kSortItems * 32) + lane;
    const uint32_t first = (uint32_t)base + at, left = valid > at ? valid - at : 0u;
    K key[kSortItems];
    load_keys(a, first, left, key);
    uint32_t pos[kSortItems];
    const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        const uint32_t d = (uint32_t)(key[r] >> a.shift) & kDigit;
        unsigned peers = 0xffffffffu;
#pragma unroll
        for (int b = 0; b < kBits; ++b) {
            const bool on = (d >> b) & 1u;
            const unsigned m = __ballot_sync(0xffffffffu, on);
            peers &= on ? m : ~m;
        }
        const uint32_t before = whist[wid][d];
        __syncwarp();
        if ((peers & lt) == 0) whist[wid][d] = (uint16_t)(before + __popc(peers));
        __syncwarp();
        pos[r] = before + __popc(peers & lt);
    }
    uint32_t val[kSortItems];
    if (kValues) load_values(a, first, left, val);
    __syncthreads();
    uint32_t count = 0, incl = 0;
    if (tid < kRadix) {
#pragma unroll
        for (int w = 0; w < kSortWarps; ++w) count += whist[w][tid];
        st_relaxed(a.state + (uint64_t)tile * kRadix + tid,
                   lookback_word(a.epoch, tile ? kPartial : kInclusive, count));
        incl = count;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o) incl += t;
        }
        if (lane == 31) s_wsum[wid] = incl;
    }
    __syncthreads();
    if (tid < kRadix) {
        uint32_t run = incl - count;
        for (uint32_t w = 0; w < wid; ++w) run += s_wsum[w];
        incl = run;  // from here on: the digit's first position in the tile
#pragma unroll
        for (int w = 0; w < kSortWarps; ++w) {
            const uint32_t c = whist[w][tid];
            whist[w][tid] = (uint16_t)run;
            run += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        const uint32_t d = (uint32_t)(key[r] >> a.shift) & kDigit;
        pos[r] += whist[wid][d];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        skey[pos[r]] = key[r];
        if (kValues) sval[pos[r]] = val[r];
    }
    if (tid < kRadix) {
        uint64_t prefix = 0;
        if (tile) {
            prefix = lookback(a.state, kRadix, tid, tile, a.epoch, a.error);
            st_relaxed(a.state + (uint64_t)tile * kRadix + tid, lookback_word(a.epoch, kInclusive, prefix + count));
        }
        s_goff[tid] = a.base[tid] + (uint32_t)prefix - incl;
        if (*(volatile unsigned *)a.error) s_stop = 1;
    }
    __syncthreads();
    if (s_stop) return;  // a wait ran out: positions are unknown, nothing is written
    if (sizeof(K) == 8 && !a.kout) {  // the last pass of an edge sort
#pragma unroll
        for (int r = 0; r < kSortItems; ++r) {
            const uint32_t j = tid + r * kSortThreads;
            if (j >= valid) break;
            const uint64_t k = skey[j];
            const uint32_t p = s_goff[(uint32_t)(k >> a.shift) & kDigit] + j;
            a.src_out[p] = (uint32_t)(k >> a.id_bits);
            a.dst_out[p] = (uint32_t)(k & ((1ull << a.id_bits) - 1));
            if (kValues) a.vout[p] = sval[j];
        }
        return;
    }
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        const uint32_t j = tid + r * kSortThreads;
        if (j >= valid) break;
        const K k = skey[j];
        const uint32_t p = s_goff[(uint32_t)(k >> a.shift) & kDigit] + j;
        a.kout[p] = k;
        if (kValues) a.vout[p] = sval[j];
    }
}

template <typename K, bool kValues, int kBits>
int launch_pass_of(const PassArgs<K> &a, cudaStream_t s) {
    const size_t smem = kSortTile * (sizeof(K) + (kValues ? 4 : 0));
    GBX_CUDA(cudaFuncSetAttribute(radix_pass_kernel<K, kValues, kBits>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)smem));
    radix_pass_kernel<K, kValues, kBits><<<ceil_div(a.n, kSortTile), kSortThreads, smem, s>>>(a);
    GBX_LAUNCH_CHECK();
    return GBX_OK;
}

template <typename K, bool kValues>
int launch_pass(const PassArgs<K> &a, int bits, cudaStream_t s) {
    return bits == 9 ? launch_pass_of<K, kValues, 9>(a, s) : launch_pass_of<K, kValues, 8>(a, s);
}

// Bits per digit for a key of `total` bits: nine where that saves a pass. A
// nine-bit pass has runs half as long and twice the look-back words and costs
// 7% more (44 bits, 67M weighted edges: 6 passes of 490 us, 5 of 530 us).
int digit_bits(int total) { return (total + 8) / 9 < (total + 7) / 8 ? 9 : 8; }

// ---- removal of repeats and self loops ------------------------------------------

// removeDulpicatesSelfLoopEdges on sorted edges (edgeList.c:255-321): an edge
// stays when it is no self loop and differs from the one before it; a kept
// weight is truncated through uint32 as the reference's uint32_t tempWeight
// does (edgeList.c:260,273). One read and one write of each edge: the
// positions come from the same look-back as the sort's, one word per tile.
constexpr int kUniqueThreads = 512, kUniqueItems = 8;
constexpr uint32_t kUniqueTile = kUniqueThreads * kUniqueItems;

__global__ void __launch_bounds__(kUniqueThreads)
    unique_edges_kernel(const uint64_t *__restrict__ keys, const uint32_t *__restrict__ w, uint32_t n, int id_bits,
                        uint32_t epoch, uint64_t *state, unsigned *ticket, SortControl *ctl, uint32_t *src_out,
                        uint32_t *dst_out, float *w_out) {
    __shared__ uint32_t s_wsum[kUniqueThreads / 32];
    __shared__ uint32_t s_tile, s_base, s_stop;
    const uint32_t tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    if (tid == 0) s_tile = atomicAdd(ticket, 1u);
    __syncthreads();
    const uint32_t tile = s_tile;
    const uint64_t first = (uint64_t)tile * kUniqueTile + wid * (kUniqueItems * 32);
    const uint64_t idm = (1ull << id_bits) - 1;
    uint64_t key[kUniqueItems];
#pragma unroll
    for (int r = 0; r < kUniqueItems; ++r) {
        const uint64_t i = first + r * 32 + lane;
        key[r] = i < n ? __ldcs((const unsigned long long *)keys + i) : ~0ull;
    }
    uint64_t last = first && first < n ? keys[first - 1] : 0;  // the element before the warp's first
    uint32_t val[kUniqueItems];
    if (w) {
#pragma unroll
        for (int r = 0; r < kUniqueItems; ++r) {
            const uint64_t i = first + r * 32 + lane;
            val[r] = i < n ? __ldcs(w + i) : 0u;
        }
    }
    unsigned kept[kUniqueItems];
    uint32_t mine = 0;
#pragma unroll
    for (int r = 0; r < kUniqueItems; ++r) {
        const uint64_t i = first + r * 32 + lane;
        uint64_t prev = __shfl_up_sync(0xffffffffu, key[r], 1);
        if (lane == 0) prev = last;
        last = __shfl_sync(0xffffffffu, key[r], 31);
        const bool k = i < n && (key[r] >> id_bits) != (key[r] & idm) && (i == 0 || key[r] != prev);
        kept[r] = __ballot_sync(0xffffffffu, k);
        mine += __popc(kept[r]);
    }
    if (lane == 0) s_wsum[wid] = mine;
    __syncthreads();
    if (wid == 0) {
        const uint32_t c = lane < kUniqueThreads / 32 ? s_wsum[lane] : 0u;
        uint32_t incl = c;
#pragma unroll
        for (int o = 1; o < kUniqueThreads / 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o) incl += t;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, incl, kUniqueThreads / 32 - 1);
        if (lane == 0) st_relaxed(state + tile, lookback_word(epoch, tile ? kPartial : kInclusive, total));
        __syncwarp();
        const uint64_t prefix = lookback_warp(state, tile, epoch, &ctl->error);
        if (lane < kUniqueThreads / 32) s_wsum[lane] = incl - c;
        if (lane == 0) {
            if (tile) st_relaxed(state + tile, lookback_word(epoch, kInclusive, prefix + total));
            s_base = (uint32_t)prefix;
            s_stop = *(volatile unsigned *)&ctl->error;
            if ((uint64_t)(tile + 1) * kUniqueTile >= n) ctl->kept = (uint32_t)prefix + total;
        }
    }
    __syncthreads();
    if (s_stop) return;
    uint32_t p = s_base + s_wsum[wid];
#pragma unroll
    for (int r = 0; r < kUniqueItems; ++r) {
        if ((kept[r] >> lane) & 1u) {
            const uint32_t q = p + __popc(kept[r] & ((1u << lane) - 1u));
            src_out[q] = (uint32_t)(key[r] >> id_bits);
            dst_out[q] = (uint32_t)(key[r] & idm);
            if (w_out) w_out[q] = w ? (float)(uint32_t)__uint_as_float(val[r]) : 1.0f;
        }
        p += __popc(kept[r]);
    }
}

unsigned hist_grid(uint64_t n) {
    return std::max(1u, std::min<unsigned>(ceil_div(n, 256 * 4), (unsigned)num_sms() * 8));
}

int bits_for(uint32_t maxv) {
    int b = 0;
    while (b < 32 && (maxv >> b)) ++b;
    return b;
}

__global__ void fill_ones_kernel(float *w, uint32_t n) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        w[i] = 1.0f;
}

constexpr int kUniquePass = 15;  // ticket and epoch of the removal of repeats

}  // namespace

int check_sort(const SortControl &h) {
    GBX_REQUIRE(h.error == 0, GBX_ERR_DEVICE_TIMEOUT, "a sort's wait on earlier tiles ran out");
    return GBX_OK;
}

int radix_sort_pairs(uint32_t *keys, uint32_t *vals, uint32_t n, int bits, cudaStream_t s, bool iota) {
    // without a digit to sort by, a pass over an empty one numbers the values
    const int total = std::max(std::min(bits, 32), 0), db = digit_bits(total);
    const int passes = std::max((total + db - 1) / db, iota ? 1 : 0);
    if (n == 0 || passes == 0 || (n == 1 && !iota)) return GBX_OK;
    const size_t words = (size_t)ceil_div(n, kSortTile) << db;
    DevBuf<uint32_t> k2, v2, hist;
    DevBuf<uint64_t> state;
    DevBuf<SortControl> ctl;
    GBX_TRY(k2.alloc(n, s));
    GBX_TRY(v2.alloc(n, s));
    GBX_TRY(hist.alloc(4 * kMaxRadix, s));
    GBX_TRY(ctl.alloc(1, s));
    GBX_TRY(state.alloc(words, s));
    GBX_CUDA(cudaMemsetAsync(hist.p, 0, 4 * kMaxRadix * 4, s));
    GBX_CUDA(cudaMemsetAsync(ctl.p, 0, sizeof(SortControl), s));
    GBX_CUDA(cudaMemsetAsync(state.p, 0, words * 8, s));
    key_hist_kernel<<<hist_grid(n), 256, 0, s>>>(keys, n, db, passes, hist.p);
    GBX_LAUNCH_CHECK();
    digit_base_kernel<<<passes, kMaxRadix, 0, s>>>(hist.p, n, ctl.p);
    GBX_LAUNCH_CHECK();
    PassArgs<uint32_t> a{};
    a.n = n;
    a.state = state.p;
    a.error = &ctl.p->error;
    uint32_t *ka = keys, *va = vals, *kb = k2.p, *vb = v2.p;
    for (int p = 0; p < passes; ++p) {
        a.kin = ka;
        a.vin = iota && p == 0 ? nullptr : va;
        a.kout = kb;
        a.vout = vb;
        a.shift = db * p;
        a.epoch = (uint32_t)p + 1;
        a.base = hist.p + p * kMaxRadix;
        a.ticket = ctl.p->ticket + p;
        GBX_TRY((launch_pass<uint32_t, true>(a, db, s)));
        std::swap(ka, kb);
        std::swap(va, vb);
    }
    if (ka != keys) {
        GBX_CUDA(cudaMemcpyAsync(keys, ka, (size_t)n * 4, cudaMemcpyDeviceToDevice, s));
        GBX_CUDA(cudaMemcpyAsync(vals, va, (size_t)n * 4, cudaMemcpyDeviceToDevice, s));
    }
    SortControl h;
    GBX_CUDA(cudaMemcpyAsync(&h, ctl.p, sizeof(h), cudaMemcpyDeviceToHost, s));
    GBX_CUDA(cudaStreamSynchronize(s));
    return check_sort(h);
}

int sort_edges(const EdgeView &e, const float *w, bool by_dst, bool dedup, uint32_t V, uint32_t *src_out,
               uint32_t *dst_out, float *w_out, DevBuf<SortControl> *ctl, cudaStream_t s) {
    const uint32_t n = e.count();
    const bool values = w && w_out;
    DevBuf<uint32_t> hist, va, vb;
    DevBuf<uint64_t> ka, kb, state;
    const size_t words = (size_t)ceil_div(n, kSortTile) << kMaxBits;
    GBX_TRY(ctl->alloc(1, s));
    GBX_CUDA(cudaMemsetAsync(ctl->p, 0, sizeof(SortControl), s));
    if (n == 0) return GBX_OK;
    GBX_TRY(hist.alloc(kMaxPasses * kMaxRadix, s));
    GBX_TRY(state.alloc(words, s));
    GBX_CUDA(cudaMemsetAsync(state.p, 0, words * 8, s));
    // Plain ids are below V. Ids with mask bits (the sort key is the whole
    // id, the reference radix-sorts all 32 bits) show in the first count and
    // get a second one.
    SortControl h{};
    int id_bits = std::max(1, bits_for(V - 1)), lo = 0, db = 8, passes = 0;
    for (int round = 0; round < 2; ++round) {
        lo = by_dst ? 0 : id_bits;
        db = digit_bits(2 * id_bits - lo);
        passes = (2 * id_bits - lo + db - 1) / db;
        GBX_CUDA(cudaMemsetAsync(hist.p, 0, kMaxPasses * kMaxRadix * 4, s));
        edge_hist_kernel<<<hist_grid(e.E), 256, 0, s>>>(e, id_bits, lo, db, passes, hist.p, ctl->p);
        GBX_LAUNCH_CHECK();
        digit_base_kernel<<<passes, kMaxRadix, 0, s>>>(hist.p, n, ctl->p);
        GBX_LAUNCH_CHECK();
        GBX_CUDA(cudaMemcpyAsync(&h, ctl->p, sizeof(h), cudaMemcpyDeviceToHost, s));
        GBX_CUDA(cudaStreamSynchronize(s));
        GBX_REQUIRE(h.max_vertex < V, GBX_ERR_INVALID, "vertex id %u >= num_vertices %u", h.max_vertex, V);
        if (h.max_id < V || round) break;
        id_bits = bits_for(h.max_id);
        GBX_CUDA(cudaMemsetAsync(ctl->p, 0, sizeof(SortControl), s));
    }
    // The passes that move something; at least one into working memory before
    // the one that writes the outputs, which may be the inputs.
    int order[9], count = 0;
    for (int k = 0; k < passes; ++k)
        if (!((h.trivial >> k) & 1u)) order[count++] = k;
    while (count < (dedup ? 1 : 2)) order[count++] = 0 < count ? order[count - 1] : 0;
    GBX_TRY(ka.alloc(n, s));
    if (count > 2 || (dedup && count > 1)) GBX_TRY(kb.alloc(n, s));
    if (values) {
        GBX_TRY(va.alloc(n, s));
        if (kb.p) GBX_TRY(vb.alloc(n, s));
    }
    PassArgs<uint64_t> a{};
    a.edges = e;
    a.n = n;
    a.id_bits = id_bits;
    a.state = state.p;
    a.error = &ctl->p->error;
    a.vin = reinterpret_cast<const uint32_t *>(w);
    uint64_t *kout = ka.p, *kin = nullptr;
    uint32_t *vout = va.p;
    for (int p = 0; p < count; ++p) {
        const bool last = !dedup && p + 1 == count;
        a.kin = kin;
        a.kout = last ? nullptr : kout;
        a.src_out = src_out;
        a.dst_out = dst_out;
        a.vout = last ? reinterpret_cast<uint32_t *>(w_out) : vout;
        a.shift = lo + db * order[p];
        a.epoch = (uint32_t)p + 1;
        a.base = hist.p + order[p] * kMaxRadix;
        a.ticket = ctl->p->ticket + p;
        if (values)
            GBX_TRY((launch_pass<uint64_t, true>(a, db, s)));
        else
            GBX_TRY((launch_pass<uint64_t, false>(a, db, s)));
        kin = kout;
        a.vin = vout;
        kout = kout == ka.p ? kb.p : ka.p;
        vout = vout == va.p ? vb.p : va.p;
    }
    if (dedup) {
        unique_edges_kernel<<<ceil_div(n, kUniqueTile), kUniqueThreads, 0, s>>>(
            kin, values ? a.vin : nullptr, n, id_bits, kUniquePass, state.p, ctl->p->ticket + kUniquePass, ctl->p,
            src_out, dst_out, w_out);
        GBX_LAUNCH_CHECK();
    } else if (w_out && !values) {
        fill_ones_kernel<<<hist_grid(n), 256, 0, s>>>(w_out, n);
        GBX_LAUNCH_CHECK();
    }
    return GBX_OK;
}

}  // namespace gbx
