// Multi-source BFS with per-vertex source bitmasks: up to 256 BFS runs over
// one graph in one level-synchronous sweep. No reference counterpart as a
// batch; for every source the distances, processed_nodes and iteration are
// those of the reference's breadthFirstSearchGraphCSR (BFS.c:103-127) from
// that source alone (levels are unique, so the schedule does not change them).
//
// State, NW = ceil(S/32) rounded up to 1, 2, 4 or 8 words per vertex:
//   seen[v][NW]  sources that have reached v
//   F[v][NW]     sources whose frontier holds v (this level)
//   Fn[v][NW]    the next level's bits (before masking with seen)
// Each level either pushes from a compacted frontier list (atomicOr of F[u]
// into Fn of every out-neighbour; few frontier edges) or pulls over in-edges
// (OR of F[u] over v's in-edges, stopping once every bit v still misses is
// found; a source whose frontier is empty is missed by nobody any more). A group of NW lanes owns one vertex, lane k its k-th mask word, so a
// mask is one 4*NW-byte access. Pull rows above kMsLight in-edges are cut into
// kMsChunk-edge chunks worked by whole warps and OR-ed into Fn with atomics
// (OR is order-free, so the result is deterministic). An update pass then
// sets new = Fn & ~seen, seen |= new, and compacts the next frontier list;
// the new masks of each level are kept (up to kMsMaxStoredLevels of them).
//
// distances is vertex-major: distances[v * S + i] is the level of v from
// sources[i] (0 for sources[i] itself and for unreached vertices, as the
// reference reports). One final pass writes every row of distances from the
// kept level masks (a warp per vertex, whole 16-byte stores) and reduces the
// per-source results; only levels past the kept ones write their distances
// bit by bit during the traversal.
#include <algorithm>
#include <cstdint>
#include <vector>

#include "gbx_coop.cuh"

namespace gbx {

constexpr uint32_t kMsLight = 64;
constexpr uint32_t kMsChunk = 1024;
constexpr int kMsThreads = 256;

// bits of mask word k that belong to one of the S sources
__device__ __forceinline__ uint32_t ms_valid(uint32_t k, uint32_t S) {
    return 32 * k + 32 <= S ? 0xFFFFFFFFu : (S > 32 * k ? (1u << (S - 32 * k)) - 1u : 0u);
}

struct MsCounters {
    uint32_t qn;                // next frontier list length
    uint32_t pad;
    unsigned long long mf;      // out-edges of the next frontier
    uint32_t alive[8];          // sources whose next frontier holds any vertex
};

// Whether the step from the frontier *cur is a push (few out-edges) or a pull.
// Steps are enqueued before the host knows their frontiers, so the kernels of
// both kinds look here whether the step is theirs.
__host__ __device__ __forceinline__ bool ms_pushes(const MsCounters &cur, uint32_t E) {
    return cur.mf * 16 < E;
}

// ---- expansion: push ----------------------------------------------------------
template <int NW>
__global__ void __launch_bounds__(kMsThreads)
    ms_push_kernel(const uint32_t *__restrict__ off, const uint32_t *__restrict__ dest, const uint32_t *__restrict__ q,
                   const MsCounters *__restrict__ cur, uint32_t E, const uint32_t *__restrict__ F,
                   const uint32_t *__restrict__ seen, uint32_t *__restrict__ Fn) {
    const uint32_t qn = cur->qn;
    if (qn == 0 || !ms_pushes(*cur, E)) return;
    constexpr int GPW = 32 / NW;  // groups per warp
    const uint32_t lane = threadIdx.x & 31, k = lane % NW;
    const uint32_t grp = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * GPW + lane / NW;
    const uint32_t ngrp = ((gridDim.x * blockDim.x) >> 5) * GPW;
    // a short list's rows are each shared by several groups (a hub among the
    // sources: 118 us for its one group, 8 when shared)
    const uint32_t share = max(1u, min(64u, ngrp / qn));
    for (uint32_t i = grp; i < qn * share; i += ngrp) {
        const uint32_t u = q[i / share];
        const uint32_t fu = F[(size_t)u * NW + k];
        if (!fu) continue;  // lane-local: other lanes of the group may still push
        const uint32_t ee = off[u + 1];
        for (uint32_t e = off[u] + 4 * (i % share); e < ee; e += 4 * share) {
            // four out-edges per round: targets, then their seen words
            uint32_t v[4], sw[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) v[q] = e + q < ee ? __ldg(dest + e + q) : 0u;
#pragma unroll
            for (int q = 0; q < 4; ++q) sw[q] = e + q < ee ? __ldg(seen + (size_t)v[q] * NW + k) : 0xFFFFFFFFu;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint32_t add = fu & ~sw[q];
                if (add) atomicOr(Fn + (size_t)v[q] * NW + k, add);
            }
        }
    }
}

// ---- expansion: pull -----------------------------------------------------------
// Light rows: one NW-lane group per vertex; the warp's groups step through
// their rows together so the early-exit vote is warp-uniform. A level of
// RMAT-20 with 256 sources takes 233 us for light and heavy rows while every
// source is alive (283 with four edges a round and ids fetched in the round)
// and 50 to 70 once few are: bits of finished sources are not looked for.
template <int NW>
__global__ void __launch_bounds__(kMsThreads)
    ms_pull_light_kernel(const uint32_t *__restrict__ poff, const uint32_t *__restrict__ psrc, uint32_t V, uint32_t S,
                         const MsCounters *__restrict__ cnt, uint32_t E, const uint32_t *__restrict__ F,
                         const uint32_t *__restrict__ seen, uint32_t *__restrict__ Fn) {
    if (cnt->qn == 0 || ms_pushes(*cnt, E)) return;
    constexpr int GPW = 32 / NW, kIds = 8 / NW;
    const uint32_t lane = threadIdx.x & 31, k = lane % NW;
    const uint32_t alive = cnt->alive[k] & ms_valid(k, S);
    const uint32_t gmask = (NW == 32 ? 0xFFFFFFFFu : ((1u << NW) - 1u)) << (lane / NW * NW);
    const uint32_t warp0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nwarp = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t base = warp0 * GPW; base < V; base += nwarp * GPW) {
        const uint32_t v = base + lane / NW;
        uint32_t b = 0, e = 0, need = 0;
        if (v < V) {
            b = poff[v];
            e = poff[v + 1];
            need = ~seen[(size_t)v * NW + k] & alive;
            if (e - b > kMsLight) e = b;  // heavy rows are worked by the chunk kernel
        }
        uint32_t acc = 0;
        // Eight in-edges per round: their ids, spread over the group's lanes
        // and fetched a round ahead, then their mask words, all in flight
        // together (the early exit checks once per round). open: some lane of
        // the group has bits it needs and lacks.
        bool open = __ballot_sync(0xFFFFFFFFu, need != 0 && b < e) & gmask;
        uint32_t j = b;
        uint32_t ids[kIds];
#pragma unroll
        for (int i = 0; i < kIds; ++i) ids[i] = open && j + i * NW + k < e ? __ldg(psrc + j + i * NW + k) : 0u;
        while (__any_sync(0xFFFFFFFFu, open)) {
            uint32_t u[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) u[q] = __shfl_sync(0xFFFFFFFFu, ids[q / NW], q % NW, NW);
#pragma unroll
            for (int i = 0; i < kIds; ++i)
                ids[i] = open && j + 8 + i * NW + k < e ? __ldg(psrc + j + 8 + i * NW + k) : 0u;
            uint32_t m[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) m[q] = open && j + q < e ? __ldg(F + (size_t)u[q] * NW + k) : 0u;
#pragma unroll
            for (int q = 0; q < 8; ++q) acc |= m[q];
            j += 8;
            open = __ballot_sync(0xFFFFFFFFu, open && (need & ~acc) != 0 && j < e) & gmask;
        }
        if (v < V && acc) Fn[(size_t)v * NW + k] = acc;  // heavy rows leave acc 0 here
    }
}

struct MsChunk {
    uint32_t row, eb, ee, pad;
};

// Heavy rows: one warp per chunk, its groups striding the chunk's edges.
template <int NW>
__global__ void __launch_bounds__(kMsThreads)
    ms_pull_heavy_kernel(const MsChunk *__restrict__ chunks, uint32_t n_chunks, const uint32_t *__restrict__ psrc,
                         uint32_t S, const MsCounters *__restrict__ cnt, uint32_t E, const uint32_t *__restrict__ F,
                         const uint32_t *__restrict__ seen, uint32_t *__restrict__ Fn) {
    if (cnt->qn == 0 || ms_pushes(*cnt, E)) return;
    constexpr int GPW = 32 / NW;
    constexpr int kPer = 8, kEdges = kPer * GPW;             // edges per group and per warp in a round
    constexpr int kLoads = kEdges / 32 > 0 ? kEdges / 32 : 1;
    const uint32_t lane = threadIdx.x & 31, k = lane % NW, gi = lane / NW;
    const uint32_t alive = cnt->alive[k] & ms_valid(k, S);
    const uint32_t warp0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nwarp = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t c = warp0; c < n_chunks; c += nwarp) {
        const MsChunk ck = chunks[c];
        const uint32_t need = ~seen[(size_t)ck.row * NW + k] & alive;
        if (!__any_sync(0xFFFFFFFFu, need)) continue;
        uint32_t acc = 0;
        // kEdges edges per round: 32 ids per load, fetched a round ahead, then
        // each group's mask words in flight together
        uint32_t ids[kLoads];
#pragma unroll
        for (int i = 0; i < kLoads; ++i)
            ids[i] = ck.eb + 32 * i + lane < ck.ee ? __ldg(psrc + ck.eb + 32 * i + lane) : 0u;
        for (uint32_t j0 = ck.eb; j0 < ck.ee; j0 += kEdges) {
            uint32_t u[kPer];
#pragma unroll
            for (int q = 0; q < kPer; ++q)
                u[q] = __shfl_sync(0xFFFFFFFFu, ids[(q * GPW) / 32], (q * GPW) % 32 + gi);
#pragma unroll
            for (int i = 0; i < kLoads; ++i) {
                const uint32_t j = j0 + kEdges + 32 * i + lane;
                ids[i] = j < ck.ee ? __ldg(psrc + j) : 0u;
            }
            uint32_t m[kPer];
#pragma unroll
            for (int q = 0; q < kPer; ++q)
                m[q] = j0 + q * GPW + gi < ck.ee ? __ldg(F + (size_t)u[q] * NW + k) : 0u;
#pragma unroll
            for (int q = 0; q < kPer; ++q) acc |= m[q];
            // OR across the groups, then stop once every needed bit is present
            uint32_t all = acc;
#pragma unroll
            for (int o = NW; o < 32; o <<= 1) all |= __shfl_xor_sync(0xFFFFFFFFu, all, o);
            if (!__any_sync(0xFFFFFFFFu, (need & ~all) != 0)) break;
        }
#pragma unroll
        for (int o = NW; o < 32; o <<= 1) acc |= __shfl_xor_sync(0xFFFFFFFFu, acc, o);
        if (gi == 0 && (acc & need)) atomicOr(Fn + (size_t)ck.row * NW + k, acc & need);
    }
}

// ---- update ----------------------------------------------------------------------
// new = Fn & ~seen; seen |= new; F_next = new (written into Fn, which is kept
// as this level's mask while levels are stored); v appended to the next
// frontier list when any bit is new. Past the stored levels (kWriteDist) the
// distances of the new bits are written here, one by one. Fz is the mask that
// the step after this one fills, zeroed on the way (or null).
template <int NW, bool kWriteDist>
__global__ void __launch_bounds__(kMsThreads)
    ms_update_kernel(uint32_t V, uint32_t S, uint32_t level, const uint32_t *__restrict__ off,
                     uint32_t *__restrict__ seen, uint32_t *__restrict__ Fn, uint32_t *__restrict__ Fz,
                     uint32_t *__restrict__ dist, uint32_t *__restrict__ qnext, const MsCounters *cur,
                     MsCounters *cnt) {
    if (cur->qn == 0) return;  // the sweep ended before this step
    // next-frontier appends are staged per warp in shared memory; what the
    // warps hold at the end and the out-degree sum go out once per CTA, since
    // atomics on one address take about a nanosecond each, one after the other
    // (RMAT-20, 256 sources, 8 levels, one step at a time: 1,660 -> 1,570 us)
    __shared__ uint32_t s_q[kMsThreads / 32][kWarpQueueCap];
    __shared__ uint32_t s_alive[NW];
    __shared__ unsigned long long s_mf;
    if (threadIdx.x < NW) s_alive[threadIdx.x] = 0;
    if (threadIdx.x == 0) s_mf = 0;
    __syncthreads();
    uint32_t alive = 0;
    constexpr int GPW = 32 / NW;
    const uint32_t lane = threadIdx.x & 31, k = lane % NW, gi = lane / NW;
    const uint32_t warp0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nwarp = (gridDim.x * blockDim.x) >> 5;
    WarpQueue next(s_q[threadIdx.x >> 5]);
    unsigned long long mf = 0;
    for (uint32_t base = warp0 * GPW; base < V; base += nwarp * GPW) {
        const uint32_t v = base + gi;
        uint32_t nw = 0;
        if (v < V) {
            const size_t i = (size_t)v * NW + k;
            const uint32_t s0 = seen[i];
            nw = Fn[i] & ~s0;
            alive |= nw;
            Fn[i] = nw;
            if (Fz) Fz[i] = 0;
            if (nw) {
                seen[i] = s0 | nw;
                if (kWriteDist) {
                    uint32_t *row = dist + (size_t)v * S + 32 * k;
                    for (uint32_t m = nw; m; m &= m - 1) row[__ffs(m) - 1] = level;
                }
            }
        }
        // one append per vertex with any new bit: the group's lowest lane
        const uint32_t any = __ballot_sync(0xFFFFFFFFu, nw != 0);
        const uint32_t gm = (NW == 32 ? 0xFFFFFFFFu : ((1u << NW) - 1u)) << (gi * NW);
        const bool leader = k == 0 && (any & gm);
        if (leader) mf += off[v + 1] - off[v];
        next.push(v, leader, qnext, &cnt->qn);
    }
    mf = warp_sum(mf);
    if (lane == 0 && mf) atomicAdd(&s_mf, mf);
    if (alive) atomicOr(s_alive + k, alive);
    const WarpQueue none(nullptr);
    cta_flush(next, qnext, &cnt->qn, none, nullptr, nullptr);  // (waits for the CTA's warps)
    if (threadIdx.x == 0 && s_mf) atomicAdd(&cnt->mf, s_mf);
    if (threadIdx.x < NW && s_alive[threadIdx.x]) atomicOr(cnt->alive + threadIdx.x, s_alive[threadIdx.x]);
}

__global__ void ms_seed_kernel(const uint32_t *sources, uint32_t S, uint32_t NW, const uint32_t *off, uint32_t *seen,
                               uint32_t *F, uint32_t *q, MsCounters *cnt) {
    for (uint32_t i = threadIdx.x; i < S; i += blockDim.x) {
        const uint32_t s = sources[i];
        atomicOr(seen + (size_t)s * NW + i / 32, 1u << (i % 32));
        atomicOr(F + (size_t)s * NW + i / 32, 1u << (i % 32));
        q[i] = s;  // a repeated source is pushed twice: OR makes that harmless
        atomicAdd(&cnt->mf, (unsigned long long)(off[s + 1] - off[s]));
        atomicOr(cnt->alive + i / 32, 1u << (i % 32));
    }
    if (threadIdx.x == 0) cnt->qn = S;
}

// Level masks kept for the final pass: masks[L][v * NW + k] holds the
// sources (bits of word k) that reached v at level L (level 0: the seeds).
constexpr uint32_t kMsMaxStoredLevels = 32;
struct MsLevels {
    const uint32_t *m[kMsMaxStoredLevels];
    uint32_t n;
};

// The distances and the per-source results in one pass: a warp per vertex,
// lane l owning sources l*NW .. l*NW + NW-1 (NW consecutive bits of mask
// word l*NW/32). A source's level at v is the first stored level whose mask
// holds its bit; a bit that is seen but in no stored mask was reached past
// the stored levels, and its distance was written by the update kernel; the
// rest are unreached (0, as is the source's own entry at level 0). Per
// source: reached vertices (level >= 1), the out-degree sum over them, the
// deepest level.
template <int NW>
__global__ void __launch_bounds__(kMsThreads)
    ms_final_kernel(MsLevels lv, const uint32_t *__restrict__ seen, uint32_t V, uint32_t S,
                    const uint32_t *__restrict__ off, const uint32_t *__restrict__ sources, bool vec_rows,
                    uint32_t *__restrict__ dist, uint32_t *__restrict__ cnt, unsigned long long *__restrict__ edges,
                    uint32_t *__restrict__ depth) {
    __shared__ uint32_t s_cnt[32 * NW], s_depth[32 * NW];
    __shared__ unsigned long long s_edges[32 * NW];
    for (uint32_t i = threadIdx.x; i < 32 * NW; i += blockDim.x) {
        s_cnt[i] = 0;
        s_depth[i] = 0;
        s_edges[i] = 0;
    }
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t k = lane * NW / 32, sh = (lane * NW) % 32;
    const uint32_t bmask = NW == 32 ? 0xFFFFFFFFu : ((1u << NW) - 1u);
    const uint32_t s0 = lane * NW;  // this lane's first source
    uint32_t c[NW], dm[NW];
    unsigned long long ed[NW];
#pragma unroll
    for (int j = 0; j < NW; ++j) c[j] = dm[j] = 0, ed[j] = 0;
    const uint32_t warp0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nwarp = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t v = warp0; v < V; v += nwarp) {
        const size_t w = (size_t)v * NW + k;
        const uint32_t sw = (__ldg(seen + w) >> sh) & bmask;
        const uint32_t deg = __ldg(off + v + 1) - __ldg(off + v);
        uint32_t lvl[NW];
#pragma unroll
        for (int j = 0; j < NW; ++j) lvl[j] = 0;
        uint32_t found = 0;
        for (uint32_t L0 = 0; L0 < lv.n && found != sw; L0 += 8) {
            uint32_t m[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) m[q] = L0 + q < lv.n ? (__ldg(lv.m[L0 + q] + w) >> sh) & bmask : 0u;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const uint32_t nb = m[q] & ~found;
#pragma unroll
                for (int j = 0; j < NW; ++j)
                    if ((nb >> j) & 1u) lvl[j] = L0 + q;
                found |= m[q];
            }
        }
        uint32_t *row = dist + (size_t)v * S + s0;
        const uint32_t deep = sw & ~found;  // written by the update kernel past the stored levels
        if (deep) {
#pragma unroll
            for (int j = 0; j < NW; ++j)
                if ((deep >> j) & 1u) lvl[j] = row[j];
        }
        const bool full = s0 + NW <= S;
        if (NW % 4 == 0 && vec_rows && full) {
#pragma unroll
            for (int q = 0; q < NW / 4; ++q)
                reinterpret_cast<uint4 *>(row)[q] = make_uint4(lvl[4 * q], lvl[4 * q + 1], lvl[4 * q + 2], lvl[4 * q + 3]);
        } else {
#pragma unroll
            for (int j = 0; j < NW; ++j)
                if (s0 + j < S) row[j] = lvl[j];
        }
#pragma unroll
        for (int j = 0; j < NW; ++j) {
            if (lvl[j]) {  // only sources below S can hold a level
                c[j] += 1;
                ed[j] += deg;
                dm[j] = max(dm[j], lvl[j]);
            }
        }
    }
#pragma unroll
    for (int j = 0; j < NW; ++j) {
        if (s0 + j < S && c[j]) {
            atomicAdd(s_cnt + s0 + j, c[j]);
            atomicAdd(s_edges + s0 + j, ed[j]);
            atomicMax(s_depth + s0 + j, dm[j]);
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < S; i += blockDim.x) {
        // block 0 adds each source's own out-edges
        const unsigned long long own = blockIdx.x == 0 ? __ldg(off + sources[i] + 1) - __ldg(off + sources[i]) : 0u;
        if (s_cnt[i] || own) {
            atomicAdd(cnt + i, s_cnt[i]);
            atomicAdd(edges + i, s_edges[i] + own);
            atomicMax(depth + i, s_depth[i]);
        }
    }
}

// The same for a traversal of up to 2^kPlanes levels, all of them kept (the
// usual case). A lane first takes one mask word of one vertex and turns the
// levels of its 32 sources into kPlanes bit planes of the level number --
// GPW vertices per warp, loads coalesced, four instructions per level and
// word. Then the warp goes through those vertices one by one: each lane gets
// the planes' NW bits of its own sources by a shuffle, spreads them to bytes
// with a multiplication, and writes its NW levels. The deepest level of a
// source is kept as one word per level; counts as bytes that are emptied every
// 255 vertices. Bound by the 4 V S bytes written: RMAT-20, 256 sources, 1.07 GB
// in 286 us; a select per source and level, and 64-bit sums per source and
// vertex, took 730 us.
template <int NW, int kPlanes>
__global__ void __launch_bounds__(kMsThreads)
    ms_planes_kernel(MsLevels lv, uint32_t V, uint32_t S, const uint32_t *__restrict__ off,
                     const uint32_t *__restrict__ sources, bool vec_rows, uint32_t *__restrict__ dist,
                     uint32_t *__restrict__ cnt, unsigned long long *__restrict__ edges, uint32_t *__restrict__ depth) {
    constexpr int GPW = 32 / NW, kLevels = 1 << kPlanes;
    __shared__ uint32_t s_cnt[32 * NW], s_depth[32 * NW];
    __shared__ unsigned long long s_edges[32 * NW];
    for (uint32_t i = threadIdx.x; i < 32 * NW; i += blockDim.x) {
        s_cnt[i] = 0;
        s_depth[i] = 0;
        s_edges[i] = 0;
    }
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t s0 = lane * NW, word = s0 / 32, sh = s0 % 32;  // this lane's sources in the second half
    constexpr uint32_t bmask = (1u << NW) - 1u;
    uint32_t at_level[kLevels];  // first half: sources of this lane's word that reach anything at each level
#pragma unroll
    for (int L = 0; L < kLevels; ++L) at_level[L] = 0;
    uint32_t c4[(NW + 3) / 4], ed[NW];  // reached: a byte per source; out-degree sums
    unsigned long long held = 0;        // what ed may have grown to
    uint32_t since = 0;
#pragma unroll
    for (int j = 0; j < (NW + 3) / 4; ++j) c4[j] = 0;
#pragma unroll
    for (int j = 0; j < NW; ++j) ed[j] = 0;
    auto empty = [&]() {
#pragma unroll
        for (int j = 0; j < NW; ++j) {
            const uint32_t n = (c4[j / 4] >> (8 * (j % 4))) & 0xFFu;
            if (s0 + j < S && n) {
                atomicAdd(s_cnt + s0 + j, n);
                atomicAdd(s_edges + s0 + j, (unsigned long long)ed[j]);
            }
            ed[j] = 0;
        }
#pragma unroll
        for (int j = 0; j < (NW + 3) / 4; ++j) c4[j] = 0;
        since = 0;
        held = 0;
    };
    const uint32_t warp0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nwarp = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t base = warp0 * GPW; base < V; base += nwarp * GPW) {
        const uint32_t mine = base + lane / NW;
        const bool in = mine < V;
        const size_t w = (size_t)mine * NW + lane % NW;
        uint32_t deg = in ? __ldg(off + mine + 1) - __ldg(off + mine) : 0u;
        uint32_t found = 0, plane[kPlanes];
#pragma unroll
        for (int p = 0; p < kPlanes; ++p) plane[p] = 0;
#pragma unroll
        for (int L0 = 0; L0 < kLevels; L0 += 8) {
            if (L0 && (uint32_t)L0 >= lv.n) break;
            uint32_t m[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) m[q] = in && (uint32_t)(L0 + q) < lv.n ? __ldg(lv.m[L0 + q] + w) : 0u;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const uint32_t fresh = m[q] & ~found;
                found |= m[q];
                at_level[L0 + q] |= fresh;
#pragma unroll
                for (int p = 0; p < kPlanes; ++p)
                    if (((L0 + q) >> p) & 1) plane[p] |= fresh;
            }
        }
#pragma unroll
        for (int i = 0; i < GPW; ++i) {
            const uint32_t v = base + i;
            if (v >= V) break;
            const uint32_t d = __shfl_sync(0xffffffffu, deg, i * NW);
            uint32_t bits[kPlanes], reached = 0;
#pragma unroll
            for (int p = 0; p < kPlanes; ++p) {
                bits[p] = (__shfl_sync(0xffffffffu, plane[p], i * NW + word) >> sh) & bmask;
                reached |= bits[p];  // level 1 or more
            }
            if (held + d > 0xFFFFFFFFull || since == 255) empty();
            held += d;
            ++since;
            uint32_t lvl[NW];
#pragma unroll
            for (int j = 0; j < NW; j += 4) {
                // four sources' bits to the low bits of four bytes
                uint32_t bytes = 0;
#pragma unroll
                for (int p = 0; p < kPlanes; ++p)
                    bytes |= ((((bits[p] >> j) & 15u) * 0x00204081u) & 0x01010101u) << p;
                c4[j / 4] += (((reached >> j) & 15u) * 0x00204081u) & 0x01010101u;
#pragma unroll
                for (int q = 0; q < 4 && j + q < NW; ++q) lvl[j + q] = (bytes >> (8 * q)) & 0xFFu;
            }
#pragma unroll
            for (int j = 0; j < NW; ++j) ed[j] += (reached >> j) & 1u ? d : 0u;
            uint32_t *row = dist + (size_t)v * S + s0;
            if (NW % 4 == 0 && vec_rows && s0 + NW <= S) {
#pragma unroll
                for (int q = 0; q < NW / 4; ++q)
                    reinterpret_cast<uint4 *>(row)[q] =
                        make_uint4(lvl[4 * q], lvl[(4 * q + 1) % NW], lvl[(4 * q + 2) % NW], lvl[(4 * q + 3) % NW]);
            } else {
#pragma unroll
                for (int j = 0; j < NW; ++j)
                    if (s0 + j < S) row[j] = lvl[j];
            }
        }
    }
    empty();
    // the deepest level that reached anything, per source
#pragma unroll
    for (int L = 1; L < kLevels; ++L)
        for (uint32_t m = at_level[L]; m; m &= m - 1) atomicMax(s_depth + 32 * (lane % NW) + __ffs(m) - 1, (uint32_t)L);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < S; i += blockDim.x) {
        // block 0 adds each source's own out-edges
        const unsigned long long own = blockIdx.x == 0 ? __ldg(off + sources[i] + 1) - __ldg(off + sources[i]) : 0u;
        if (s_cnt[i] || own) {
            atomicAdd(cnt + i, s_cnt[i]);
            atomicAdd(edges + i, s_edges[i] + own);
            atomicMax(depth + i, s_depth[i]);
        }
    }
}

}  // namespace gbx

// Chunk list of the heavy pull rows of a graph (cached on the graph).
struct gbx_ms_plan {
    gbx::MsChunk *chunks = nullptr;
    uint32_t n_chunks = 0;
};

void gbx_free_ms_plan(gbx_ms_plan *p) {
    if (!p) return;
    cudaFree(p->chunks);
    delete p;
}

using namespace gbx;

namespace {

int ms_plan(gbx_graph *g, cudaStream_t s, gbx_ms_plan **out) {
    if (!g->ms_plan) {
        const uint32_t V = g->V;
        std::vector<uint32_t> off(V + 1);
        GBX_CUDA(cudaMemcpyAsync(off.data(), g->pull_offsets(), 4 * ((size_t)V + 1), cudaMemcpyDeviceToHost, s));
        GBX_CUDA(cudaStreamSynchronize(s));
        std::vector<MsChunk> ch;
        for (uint32_t v = 0; v < V; ++v)
            if (off[v + 1] - off[v] > kMsLight)
                for (uint32_t c = off[v]; c < off[v + 1]; c += kMsChunk)
                    ch.push_back({v, c, std::min(c + kMsChunk, off[v + 1]), 0});
        gbx_ms_plan *p = new gbx_ms_plan();
        p->n_chunks = (uint32_t)ch.size();
        if (cudaMalloc(&p->chunks, sizeof(MsChunk) * std::max<size_t>(1, ch.size())) != cudaSuccess) {
            (void)cudaGetLastError();
            delete p;
            set_error("multi-source BFS plan allocation failed");
            return GBX_ERR_NOMEM;
        }
        if (!ch.empty()) {
            const cudaError_t e =
                cudaMemcpyAsync(p->chunks, ch.data(), sizeof(MsChunk) * ch.size(), cudaMemcpyHostToDevice, s);
            if (e == cudaSuccess) cudaStreamSynchronize(s);
            if (e != cudaSuccess) {
                gbx_free_ms_plan(p);
                return cuda_fail(e, "cudaMemcpyAsync", __FILE__, __LINE__);
            }
        }
        g->ms_plan = p;
    }
    *out = g->ms_plan;
    return GBX_OK;
}

// Steps enqueued before the host looks: as many as most graphs have levels at
// first, then fewer, since those past a sweep's end are empty launches. us for
// 100 sources, one at a time / 2 / 4 / 8: R-MAT of 1,000 vertices 481 / 405 /
// 376 / 358, 250,000 613 / 543 / 515 / 495; local graph of 30,000 842 / 706 /
// 684 / 728; RMAT-20 with 256 sources 1,622 / 1,543 / 1,519 / 1,494 (the same
// inputs again and again; new inputs each time 1,605 with 8). Masks above
// kAheadBytes, or that there is no memory for, are not allocated ahead.
constexpr uint32_t kAhead = 8, kAheadLater = 4;
constexpr size_t kAheadBytes = size_t(64) << 20;

template <int NW>
int msbfs_impl(gbx_graph *g, uint32_t S, const uint32_t *src_d, uint32_t *dist, gbx_bfs_result *res_host,
               cudaStream_t s) {
    const uint32_t V = g->V;
    gbx_ms_plan *plan = nullptr;
    GBX_TRY(ms_plan(g, s, &plan));
    const size_t words = (size_t)V * NW;
    // the level masks kept for the final pass: as many levels as fit 8 GiB
    // (at least two), at most kMsMaxStoredLevels; deeper levels use the two
    // `deep` buffers in turn and write their distances bit by bit
    const uint32_t max_stored = (uint32_t)std::max<size_t>(
        2, std::min<size_t>(kMsMaxStoredLevels, (8ull << 30) / std::max<size_t>(1, words * 4)));
    std::vector<DevBuf<uint32_t>> lvbuf(max_stored);
    DevBuf<uint32_t> seen, deep[2], q0, q1;
    DevBuf<unsigned long long> per_source;  // edges, then reached vertices and depths, S of each
    // Steps go out kAhead at a time where a mask is small: a step that is short
    // against the host's round trip does not wait for one. cnt[j]: the
    // frontier of the j-th step of a batch.
    uint32_t ahead = words * 4 <= kAheadBytes ? kAhead : 1;
    DevBuf<MsCounters> cnt;
    GBX_TRY(seen.alloc(words, s));
    GBX_TRY(lvbuf[0].alloc(words, s));
    GBX_TRY(q0.alloc(std::max(V, S), s));
    GBX_TRY(q1.alloc(std::max(V, S), s));
    GBX_TRY(cnt.alloc(ahead + 1, s));
    GBX_TRY(per_source.alloc(2 * (size_t)S, s));
    GBX_CUDA(cudaMemsetAsync(seen.p, 0, words * 4, s));
    GBX_CUDA(cudaMemsetAsync(lvbuf[0].p, 0, words * 4, s));
    GBX_CUDA(cudaMemsetAsync(cnt.p, 0, (ahead + 1) * sizeof(MsCounters), s));
    ms_seed_kernel<<<1, 256, 0, s>>>(src_d, S, NW, g->offsets, seen.p, lvbuf[0].p, q0.p, cnt.p);
    GBX_LAUNCH_CHECK();
    MsCounters h[kAhead + 1] = {};
    h[0].qn = S;
    bool known = false;  // the host has read the batch's first frontier
    // the mask of a level: kept while it fits, else one of two in turn
    auto mask_of = [&](uint32_t l, uint32_t **out) -> int {
        DevBuf<uint32_t> &d = l < max_stored ? lvbuf[l] : deep[l & 1];
        if (!d.p) GBX_TRY(d.alloc(words, s));
        *out = d.p;
        return GBX_OK;
    };
    // The masks of a batch's levels before its first step. Where there is no
    // memory for them, steps go one at a time from here on and allocate what
    // each needs.
    auto reserve = [&](uint32_t level) -> int {
        uint32_t *mask = nullptr;
        int st = GBX_OK;
        for (uint32_t l = level + 1; ahead > 1 && st == GBX_OK && l <= level + 1 + ahead; ++l) st = mask_of(l, &mask);
        if (st == GBX_ERR_NOMEM) {
            clear_error();
            for (uint32_t l = level + 2; l < max_stored; ++l) lvbuf[l].release();
            ahead = 1;
            st = GBX_OK;
        }
        if (st == GBX_OK && ahead == 1 && !known) {
            GBX_CUDA(cudaMemcpyAsync(h, cnt.p, sizeof(h[0]), cudaMemcpyDeviceToHost, s));
            GBX_CUDA(cudaStreamSynchronize(s));
            known = true;
        }
        return st;
    };
    uint32_t *F = lvbuf[0].p, *Fn = nullptr, *q = q0.p, *qn = q1.p;
    GBX_TRY(reserve(0));
    if (ahead > 1) {
        GBX_TRY(mask_of(1, &Fn));
        GBX_CUDA(cudaMemsetAsync(Fn, 0, words * 4, s));
    }
    // no more CTAs than a small graph's words give work to
    const unsigned grid = (unsigned)std::min<size_t>((size_t)num_sms() * 8, std::max<size_t>(num_sms(), ceil_div(words, kMsThreads)));
    const uint32_t E = g->E;
    uint32_t level = 0, pushes = 0, pulls = 0, stored = 1;
    while (h[0].qn > 0 && level <= V) {
        for (uint32_t j = 0; j < ahead; ++j) {
            const uint32_t next = level + 1 + j;
            const bool keep = next < max_stored;
            uint32_t *Fz = nullptr;
            if (ahead > 1) {
                GBX_TRY(mask_of(next + 1, &Fz));
            } else {
                // large masks: none before it is needed
                GBX_TRY(mask_of(next, &Fn));
                GBX_CUDA(cudaMemsetAsync(Fn, 0, words * 4, s));
            }
            const MsCounters *cur = cnt.p + j;
            const bool push = !(known && j == 0) || ms_pushes(h[0], E), pull = !(known && j == 0) || !push;
            if (push) {
                ms_push_kernel<NW><<<grid, kMsThreads, 0, s>>>(g->offsets, g->dest, q, cur, E, F, seen.p, Fn);
                GBX_LAUNCH_CHECK();
            }
            if (pull) {
                ms_pull_light_kernel<NW><<<grid, kMsThreads, 0, s>>>(g->pull_offsets(), g->pull_src(), V, S, cur, E, F,
                                                                     seen.p, Fn);
                GBX_LAUNCH_CHECK();
                if (plan->n_chunks) {
                    ms_pull_heavy_kernel<NW><<<grid, kMsThreads, 0, s>>>(plan->chunks, plan->n_chunks, g->pull_src(),
                                                                         S, cur, E, F, seen.p, Fn);
                    GBX_LAUNCH_CHECK();
                }
            }
            if (keep)
                ms_update_kernel<NW, false><<<grid, kMsThreads, 0, s>>>(V, S, next, g->offsets, seen.p, Fn, Fz, dist,
                                                                        qn, cur, cnt.p + j + 1);
            else
                ms_update_kernel<NW, true><<<grid, kMsThreads, 0, s>>>(V, S, next, g->offsets, seen.p, Fn, Fz, dist,
                                                                       qn, cur, cnt.p + j + 1);
            GBX_LAUNCH_CHECK();
            F = Fn;
            Fn = Fz;
            std::swap(q, qn);
        }
        GBX_CUDA(cudaMemcpyAsync(h, cnt.p, (ahead + 1) * sizeof(MsCounters), cudaMemcpyDeviceToHost, s));
        GBX_CUDA(cudaStreamSynchronize(s));
        uint32_t j = 0;
        for (; j < ahead && h[j].qn > 0; ++j) {
            ++(ms_pushes(h[j], E) ? pushes : pulls);
            ++level;
            if (level < max_stored) stored = level + 1;
        }
        h[0] = h[j];
        if (h[0].qn > 0) {
            GBX_CUDA(cudaMemcpyAsync(cnt.p, cnt.p + ahead, sizeof(MsCounters), cudaMemcpyDeviceToDevice, s));
            GBX_CUDA(cudaMemsetAsync(cnt.p + 1, 0, ahead * sizeof(MsCounters), s));
        }
        known = true;
        ahead = std::min(ahead, kAheadLater);
        if (h[0].qn > 0) GBX_TRY(reserve(level));
    }
    GBX_REQUIRE(h[0].qn == 0, GBX_ERR_ITER_CAP, "multi-source BFS level cap reached");
    // distances of the stored levels, zeros for unreached pairs, and the
    // per-source results, in one pass
    MsLevels lv{};
    lv.n = stored;
    for (uint32_t L = 0; L < stored; ++L) lv.m[L] = lvbuf[L].p;
    GBX_CUDA(cudaMemsetAsync(per_source.p, 0, 16 * (size_t)S, s));
    unsigned long long *const re = per_source.p;
    uint32_t *const rc = reinterpret_cast<uint32_t *>(re + S), *const rd = rc + S;
    const bool vec_rows = S % 4 == 0 && (reinterpret_cast<uintptr_t>(dist) & 15u) == 0;
    const unsigned fgrid = std::min<unsigned>((unsigned)num_sms() * 6, ceil_div((uint64_t)V * NW, kMsThreads));
    if (stored == level + 1 && stored <= 8)
        ms_planes_kernel<NW, 3><<<fgrid, kMsThreads, 0, s>>>(lv, V, S, g->offsets, src_d, vec_rows, dist, rc, re, rd);
    else if (stored == level + 1 && stored <= 16)
        ms_planes_kernel<NW, 4><<<fgrid, kMsThreads, 0, s>>>(lv, V, S, g->offsets, src_d, vec_rows, dist, rc, re, rd);
    else
        ms_final_kernel<NW><<<(unsigned)num_sms() * 4, kMsThreads, 0, s>>>(lv, seen.p, V, S, g->offsets, src_d,
                                                                           vec_rows, dist, rc, re, rd);
    GBX_LAUNCH_CHECK();
    if (res_host) {
        std::vector<unsigned long long> he(2 * (size_t)S);
        GBX_CUDA(cudaMemcpyAsync(he.data(), re, 16 * (size_t)S, cudaMemcpyDeviceToHost, s));
        GBX_CUDA(cudaStreamSynchronize(s));
        const uint32_t *hc = reinterpret_cast<const uint32_t *>(he.data() + S), *hd = hc + S;
        for (uint32_t i = 0; i < S; ++i) {
            gbx_bfs_result r{};
            r.processed_nodes = hc[i] + 1;
            r.depth = hd[i];
            r.iteration = hd[i] + 2;
            r.top_down_steps = pushes;
            r.bottom_up_steps = pulls;
            r.edges_traversed = he[i];
            res_host[i] = r;
        }
    } else {
        GBX_CUDA(cudaStreamSynchronize(s));
    }
    return GBX_OK;
}

}  // namespace

extern "C" int gbx_bfs_multisource(gbx_graph *g, uint32_t num_sources, const uint32_t *sources, uint32_t *distances,
                                   gbx_bfs_result *results, void *stream) {
    clear_error();
    GBX_REQUIRE(g && sources && distances, GBX_ERR_INVALID, "graph, sources or distances is NULL");
    GBX_REQUIRE(num_sources >= 1 && num_sources <= 256, GBX_ERR_INVALID, "num_sources must be 1..256 (got %u)",
                num_sources);
    GBX_TRY(ensure_device());
    cudaStream_t s = (cudaStream_t)stream;
    std::vector<uint32_t> hs(num_sources);
    GBX_CUDA(cudaMemcpyAsync(hs.data(), sources, 4 * (size_t)num_sources, cudaMemcpyDefault, s));
    GBX_CUDA(cudaStreamSynchronize(s));
    for (uint32_t i = 0; i < num_sources; ++i)
        GBX_REQUIRE(hs[i] < g->V, GBX_ERR_INVALID, "source %u (index %u) is not below %u vertices", hs[i], i, g->V);
    DevBuf<uint32_t> src_d;
    GBX_TRY(src_d.alloc(num_sources, s));
    GBX_CUDA(cudaMemcpyAsync(src_d.p, hs.data(), 4 * (size_t)num_sources, cudaMemcpyHostToDevice, s));
    OutArray<uint32_t> dist;
    GBX_TRY(dist.bind(distances, (size_t)g->V * num_sources, s));
    std::vector<gbx_bfs_result> hr;
    if (results) hr.resize(num_sources);
    const uint32_t nw = (num_sources + 31) / 32;
    int st;
    if (nw == 1)
        st = msbfs_impl<1>(g, num_sources, src_d.p, dist.d, results ? hr.data() : nullptr, s);
    else if (nw == 2)
        st = msbfs_impl<2>(g, num_sources, src_d.p, dist.d, results ? hr.data() : nullptr, s);
    else if (nw <= 4)
        st = msbfs_impl<4>(g, num_sources, src_d.p, dist.d, results ? hr.data() : nullptr, s);
    else
        st = msbfs_impl<8>(g, num_sources, src_d.p, dist.d, results ? hr.data() : nullptr, s);
    GBX_TRY(st);
    GBX_TRY(dist.finish(s));
    GBX_CUDA(cudaStreamSynchronize(s));
    if (results) std::copy(hr.begin(), hr.end(), results);
    return GBX_OK;
}
