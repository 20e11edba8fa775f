// Persistent cooperative kernels: a grid barrier with a bounded wait and the
// launch helper that sizes the grid to what is co-resident.
//
// The barrier is one monotonic 64-bit arrival counter: at its n-th barrier
// each CTA's thread 0 adds 1 with release semantics (no reply awaited) and
// polls the counter with acquire loads until it reaches n * gridDim.x. The
// __syncthreads on either side extends the ordering to the whole CTA. Nobody
// resets or re-arms anything, so a barrier costs one arrival plus one poll
// round trip (about half the latency of a count-and-generation barrier, whose
// last arrival must reset the count and then publish the generation). The
// kernels are launched with cudaLaunchCooperativeKernel, which guarantees
// that every CTA is resident, so the wait always ends; it is still capped
// (kBarrierSpinLimit polls, about two seconds): on expiry the CTA raises the
// error word and every CTA leaves the kernel at its next barrier, so the host
// sees GBX_ERR_DEVICE_TIMEOUT instead of a hung device.
#pragma once

#include "gbx_internal.cuh"

namespace gbx {

struct GridSync {
    unsigned long long arrived;  // total arrivals since launch (zeroed by the host)
    unsigned error;              // 1 = a barrier wait expired
    unsigned pad;
};

constexpr unsigned kBarrierSpinLimit = 1u << 22;

// this CTA's arrival target for its next barrier (set by grid_barrier_init)
__shared__ unsigned long long s_grid_target;
// units of the current phase taken by this CTA's warps after their first ones (UnitDealer)
__shared__ unsigned s_units_dealt;

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

// Once at kernel start, by all threads.
__device__ __forceinline__ void grid_barrier_init() {
    if (threadIdx.x == 0) {
        s_grid_target = 0;
        s_units_dealt = 0;
    }
    __syncthreads();
}

// The CTAs that work on one thing: the whole grid, or one of several equal
// teams of a cooperative grid, each with a GridSync of its own (all CTAs are
// resident, so a team's wait ends like the grid's).
struct Team {
    uint32_t cta, ctas;
    __device__ __forceinline__ uint32_t thread() const { return cta * blockDim.x + threadIdx.x; }
    __device__ __forceinline__ uint32_t threads() const { return ctas * blockDim.x; }
    __device__ __forceinline__ bool leader() const { return cta == 0 && threadIdx.x == 0; }
};
__device__ __forceinline__ Team whole_grid() { return Team{blockIdx.x, gridDim.x}; }

// Returns false when the team must stop (a wait expired somewhere).
__device__ __forceinline__ bool grid_barrier(GridSync *gs, uint32_t ctas = gridDim.x) {
    __shared__ unsigned s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned long long target = s_grid_target + ctas;
        s_grid_target = target;
        s_units_dealt = 0;
        asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(&gs->arrived) : "memory");
        unsigned ok = 1, spins = 0;
        while (ld_acquire_u64(&gs->arrived) < target) {
            if (++spins > kBarrierSpinLimit) {
                atomicExch(&gs->error, 1u);
                break;
            }
            __nanosleep(32);
        }
        if (ld_acquire_u32(&gs->error)) ok = 0;
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// After a grid barrier: the first warp copies the step counters *src (a
// struct of 32-bit words) into the CTA's shared *dst, and the CTA waits for
// it. The other warps then read shared memory instead of sending the same
// few L2 lines thousands of requests per step. The barrier's acquire (by
// thread 0) and its closing __syncthreads order the loads after the other
// CTAs' counter updates.
template <class T>
__device__ __forceinline__ void fetch_counters(const T *src, T *dst) {
    static_assert(sizeof(T) % 4 == 0 && sizeof(T) / 4 <= 32, "counters are at most 32 words");
    if (threadIdx.x < sizeof(T) / 4)
        reinterpret_cast<uint32_t *>(dst)[threadIdx.x] = __ldcg(reinterpret_cast<const uint32_t *>(src) + threadIdx.x);
    __syncthreads();
}

// Per-warp staging of queue appends in shared memory: lanes append with
// ballot ranks into the warp's buffer, and the warp reserves space in the
// global queue with one atomic per kWarpQueueCap/2..kWarpQueueCap entries
// instead of one per ballot round (a single global length counter is
// otherwise hammered by every warp of the grid).
constexpr uint32_t kWarpQueueCap = 128;

struct WarpQueue {
    uint32_t *buf;  // kWarpQueueCap entries of shared memory owned by this warp
    uint32_t n;     // fill, identical in all lanes
    uint32_t cap;
    __device__ __forceinline__ explicit WarpQueue(uint32_t *b, uint32_t c = kWarpQueueCap) : buf(b), n(0), cap(c) {}
    __device__ __forceinline__ void flush(uint32_t *queue, unsigned *len) {
        if (n == 0) return;
        __syncwarp();
        const uint32_t lane = threadIdx.x & 31;
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(len, n);
        base = __shfl_sync(0xffffffffu, base, 0);
        for (uint32_t i = lane; i < n; i += 32) queue[base + i] = buf[i];
        __syncwarp();
        n = 0;
    }
    // all lanes call together
    __device__ __forceinline__ void push(uint32_t x, bool p, uint32_t *queue, unsigned *len) {
        const unsigned m = __ballot_sync(0xffffffffu, p);
        if (!m) return;
        const uint32_t lane = threadIdx.x & 31;
        if (p) buf[n + __popc(m & ((1u << lane) - 1u))] = x;
        n += __popc(m);
        if (n > cap - 32) flush(queue, len);
    }
};

// The warp's hubs (lanes with hub set, of `chunks` work chunks each) into a
// hub list behind one atomic: *len holds (hubs << 32) | chunks, and the list
// stays sorted by first chunk.
__device__ __forceinline__ void push_hubs(uint32_t v, uint32_t chunks, bool hub, uint32_t *hv, uint32_t *hc,
                                          unsigned long long *len) {
    const unsigned m = __ballot_sync(0xffffffffu, hub);
    if (!m) return;
    const uint32_t lane = threadIdx.x & 31, mine = hub ? chunks : 0u;
    uint32_t incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += t;
    }
    unsigned long long h = 0;
    if (lane == 31) h = atomicAdd(len, ((unsigned long long)__popc(m) << 32) | incl);
    h = __shfl_sync(0xffffffffu, h, 31);
    if (hub) {
        const uint32_t slot = (uint32_t)(h >> 32) + __popc(m & ((1u << lane) - 1u));
        hv[slot] = v;
        hc[slot] = (uint32_t)h + incl - mine;
    }
}

// End of a phase, all threads of the CTA: what its warps still hold of two
// queues goes out behind one reservation per queue and CTA. A reservation per
// warp would be 4,864 atomics on one address, which L2 takes one by one, about
// a nanosecond each.
__device__ __forceinline__ void cta_flush(const WarpQueue &a, uint32_t *qa, unsigned *la, const WarpQueue &b,
                                          uint32_t *qb, unsigned *lb) {
    __shared__ uint32_t s_fill[2][32], s_at[2][32];
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) {
        s_fill[0][wid] = a.n;
        s_fill[1][wid] = b.n;
    }
    __syncthreads();
    if (wid < 2) {
        const uint32_t n = lane < blockDim.x >> 5 ? s_fill[wid][lane] : 0u;
        uint32_t incl = n, at = 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o) incl += t;
        }
        if (lane == 31 && incl) at = atomicAdd(wid ? lb : la, incl);
        s_at[wid][lane] = __shfl_sync(0xffffffffu, at, 31) + incl - n;
    }
    __syncthreads();
    for (uint32_t i = lane; i < a.n; i += 32) qa[s_at[0][wid] + i] = a.buf[i];
    for (uint32_t i = lane; i < b.n; i += 32) qb[s_at[1][wid] + i] = b.buf[i];
}

// Work-unit dealer: unit u belongs to CTA u mod ctas. A CTA's warps take its
// units in turn -- the first by their index, later ones from a counter in
// shared memory, which grid_barrier clears, so every phase between two
// barriers deals anew. One counter for the grid would be an atomic per unit on
// one address, about a nanosecond each one after the other: 20,000 units are
// 20 us however they are spread (SSSP on RMAT-22 1,812 -> 1,525 us, on 16M
// edges 1,003 -> 763). What the CTAs lose by not helping one another is less,
// as long as a CTA has several units a warp (with the last quarter of the
// units from a common counter: 1,680 and 871).
struct UnitDealer {
    uint32_t cta, ctas, k;
    bool first;
    __device__ __forceinline__ explicit UnitDealer(Team t = whole_grid())
        : cta(t.cta), ctas(t.ctas), k(threadIdx.x >> 5), first(true) {}
    __device__ __forceinline__ uint32_t take() {
        if (!first) {
            if ((threadIdx.x & 31) == 0) k = (blockDim.x >> 5) + atomicAdd(&s_units_dealt, 1u);
            k = __shfl_sync(0xffffffffu, k, 0);
        }
        first = false;
        return k * ctas + cta;
    }
};

// Owner of work chunk c in a list whose entry h owns chunks [hc[h], hc[h+1])
// (hc strictly increasing, hc[0] = 0): the last h in [0, n) with hc[h] <= c,
// searched 32 ways at a time by the whole warp -- log32(n) rounds of one
// load per lane instead of log2(n) dependent loads. All lanes call together
// and get the same answer.
__device__ __forceinline__ uint32_t warp_chunk_owner(const uint32_t *hc, uint32_t n, uint32_t c) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t lo = 0, hi = n;  // answer in [lo, hi); hc[lo] <= c
    while (hi - lo > 1) {
        const uint32_t step = (hi - lo + 31) / 32;
        const uint32_t idx = lo + lane * step;
        const bool ok = idx < hi && __ldcg(hc + idx) <= c;
        const unsigned m = __ballot_sync(0xffffffffu, ok);  // lane 0 always holds
        lo += (31u - __clz(m)) * step;
        hi = min(lo + step, hi);
    }
    return lo;
}

// Largest co-resident grid for `kernel` with `threads` per CTA. `cache`
// (one per call site, indexed by device) keeps the answer after the first
// occupancy query.
template <class K>
inline int coop_grid(K kernel, int threads, size_t smem, int *grid, int (*cache)[64] = nullptr) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cache && dev >= 0 && dev < 64 && (*cache)[dev] > 0) {
        *grid = (*cache)[dev];
        return GBX_OK;
    }
    int per_sm = 0;
    GBX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem));
    GBX_REQUIRE(per_sm > 0, GBX_ERR_CUDA, "kernel cannot be resident");
    *grid = per_sm * num_sms();
    if (cache && dev >= 0 && dev < 64) (*cache)[dev] = *grid;
    return GBX_OK;
}

}  // namespace gbx
