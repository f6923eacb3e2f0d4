// The walk over meetings: the suffixes of reads take free prefixes of the
// run that equals them, offset after offset.  Used by the overlap stage and
// by the full match, which list which suffix meets which prefixes beforehand
// (that depends on the two lists only, not on the links made).
//
// Items are ordered by offset; inside an offset the items of one run (equal
// suffix strings: the same lo) are contiguous and in the order in which the
// reference visits them.
#pragma once
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>

#include "common.cuh"

namespace curc {

// Compaction functors: keep the list entries whose link is still free.
struct FreeLink {
    const uint32_t* ids;
    const uint32_t* link;
    __device__ bool operator()(uint32_t i) const { return link[ids[i]] == INVALID; }
};
struct MoveId {
    const uint32_t* in;
    uint32_t* out;
    __device__ void operator()(uint32_t i, uint32_t d) const { out[d] = in[i]; }
};

// Meeting of a suffix (id s) with the prefixes [lo, hi) of the list, p the
// first one's id.
struct __align__(16) Meeting {
    uint32_t s, lo, hi, p;
};

__device__ __forceinline__ uint32_t ld_l2(const uint32_t* p) { return __ldcg(p); }

// The suffixes of one run (items [i, e) with the same lo, in order) each take
// the first free prefix that is not themselves, as the reference's merge of
// the run does (its rotation puts a prefix that meets itself back in front).
// One thread.
__device__ __forceinline__ void walk_run(const Meeting* __restrict__ item, uint32_t i, uint32_t e,
                                        const uint32_t* __restrict__ pre, uint32_t q0, uint32_t hi, int off,
                                        uint32_t* next, uint32_t* prev, uint16_t* offset) {
    const uint32_t lo = item[i].lo;
    for (; i < e && item[i].lo == lo; ++i) {
        const uint32_t s = item[i].s;
        if (ld_l2(next + s) != INVALID) continue;
        bool any = false;  // a free prefix was left
        for (uint32_t q = q0; q < hi; ++q) {
            const uint32_t p = pre[q];
            if (ld_l2(prev + p) != INVALID) {
                if (!any) q0 = q + 1;
                continue;
            }
            any = true;
            if (p == s) continue;
            next[s] = p;
            prev[p] = s;
            offset[s] = uint16_t(off);
            break;
        }
        if (!any) return;
    }
}

// The same by a whole warp, for long runs: free suffixes and free prefixes
// are taken 32 at a time and paired in order; where a read would meet itself
// the rest of the run is walked by one lane.
static __device__ void walk_run_warp(const Meeting* __restrict__ item, uint32_t i, uint32_t e, const uint32_t* __restrict__ pre,
                             uint32_t q, uint32_t hi, int off, uint32_t* next, uint32_t* prev, uint16_t* offset) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t lo = item[i].lo;
    uint32_t sm = 0, pm = 0;          // free entries of the current 32 items / prefixes
    uint32_t ib = i, qb = q;          // where the next 32 start
    uint32_t s = 0, p = 0;            // this lane's entries
    bool more_s = true;
    for (;;) {
        while (sm == 0) {
            if (!more_s) return;
            const uint32_t t = ib + lane;
            const bool in = t < e && item[t].lo == lo;
            const uint32_t all = __ballot_sync(0xFFFFFFFFu, in);
            s = in ? item[t].s : 0;
            sm = __ballot_sync(0xFFFFFFFFu, in && ld_l2(next + s) == INVALID);
            ib += 32;
            more_s = all == 0xFFFFFFFFu;
        }
        while (pm == 0) {
            if (qb >= hi) return;
            const uint32_t t = qb + lane;
            const bool in = t < hi;
            p = in ? pre[t] : 0;
            pm = __ballot_sync(0xFFFFFFFFu, in && ld_l2(prev + p) == INVALID);
            qb += 32;
        }
        const int n = min(__popc(sm), __popc(pm));
        // lane k < n pairs the k-th free suffix with the k-th free prefix
        const int ks = int(lane) < n ? int(__fns(sm, 0, int(lane) + 1)) : 0;
        const int kp = int(lane) < n ? int(__fns(pm, 0, int(lane) + 1)) : 0;
        const uint32_t S = __shfl_sync(0xFFFFFFFFu, s, ks), P = __shfl_sync(0xFFFFFFFFu, p, kp);
        const uint32_t self = __ballot_sync(0xFFFFFFFFu, int(lane) < n && S == P);
        const int good = self ? __ffs(self) - 1 : n;
        if (int(lane) < good) {
            next[S] = P;
            prev[P] = S;
            offset[S] = uint16_t(off);
        }
        __syncwarp();
        if (self) {
            if (lane == 0) walk_run(item, ib - 32, e, pre, qb - 32, hi, off, next, prev, offset);
            __syncwarp();
            return;
        }
        for (int k = 0; k < n; ++k) {  // the n lowest of each are used up
            sm &= sm - 1;
            pm &= pm - 1;
        }
    }
}

constexpr int WALK_THREADS = 512;
constexpr int WALK_MAX_OFFS = 512;

// The meetings [a, e) of one offset by `threads` threads, of which this is
// number me: one thread per run, long runs by a warp.
static __device__ __forceinline__ void walk_offset(const Meeting* __restrict__ item, uint32_t a, uint32_t e,
                                                   uint32_t threads, uint32_t me, const uint32_t* __restrict__ pre,
                                                   int off, uint32_t* next, uint32_t* prev, uint16_t* offset) {
    for (uint32_t i0 = a; i0 < e; i0 += threads) {  // the same trip count for a whole warp
        const uint32_t i = i0 + me;
        bool long_run = false;
        Meeting it = {0, 0, 0, 0};
        if (i < e) {
            it = item[i];
            const bool lead = i == a || item[i - 1].lo != it.lo;
            const bool alone = i + 1 == e || item[i + 1].lo != it.lo;
            if (lead) {
                if (alone && it.hi == it.lo + 1) {
                    if (it.p != it.s) {
                        const uint32_t nx = ld_l2(next + it.s), pv = ld_l2(prev + it.p);
                        if (nx == INVALID && pv == INVALID) {
                            next[it.s] = it.p;
                            prev[it.p] = it.s;
                            offset[it.s] = uint16_t(off);
                        }
                    }
                } else {
                    // more than a few members or prefixes: by the whole warp
                    long_run = it.hi - it.lo > 8 || (i + 8 < e && item[i + 8].lo == it.lo);
                    if (!long_run) walk_run(item, i, e, pre, it.lo, it.hi, off, next, prev, offset);
                }
            }
        }
        uint32_t todo = __ballot_sync(0xFFFFFFFFu, long_run);
        while (todo) {
            const int l = __ffs(todo) - 1;
            todo &= todo - 1;
            const uint32_t ii = __shfl_sync(0xFFFFFFFFu, i, l), lo = __shfl_sync(0xFFFFFFFFu, it.lo, l),
                           hi = __shfl_sync(0xFFFFFFFFu, it.hi, l);
            walk_run_warp(item, ii, e, pre, lo, hi, off, next, prev, offset);
        }
    }
}

// One offset by a whole grid.
static __global__ void __launch_bounds__(256) walk_one_kernel(const Meeting* __restrict__ item, uint32_t a, uint32_t e,
                                                              int off, const uint32_t* __restrict__ pre, uint32_t* next,
                                                              uint32_t* prev, uint16_t* offset) {
    walk_offset(item, a, e, gridDim.x * 256, blockIdx.x * 256 + threadIdx.x, pre, off, next, prev, offset);
}

// The walk: offset after offset, one thread per run of equal suffix strings
// (long runs: a warp).  Runs of one offset share no read, so an offset's runs
// are independent; a barrier over the cluster separates the offsets.  One
// cluster suffices: an offset has few meetings (thousands at most where a
// list has 400,000 entries), and its time is the latency of two dependent
// loads and the barrier.
static __global__ void __launch_bounds__(WALK_THREADS) walk_kernel(const Meeting* __restrict__ item,
                                                                   const uint32_t* __restrict__ start_in, int off0,
                                                                   int noffs, const uint32_t* __restrict__ pre,
                                                                   const unsigned long long* __restrict__ used,
                                                                   uint32_t cap, uint32_t* next, uint32_t* prev,
                                                                   uint16_t* offset,
                                                                   unsigned long long* __restrict__ tally) {
    __shared__ uint32_t start[WALK_MAX_OFFS + 1];
    if (*used > cap) return;  // the listing is incomplete: the caller repeats it
    for (int o = threadIdx.x; o <= noffs; o += WALK_THREADS) start[o] = start_in[o];
    __syncthreads();
    const uint32_t threads = gridDim.x * WALK_THREADS, me = blockIdx.x * WALK_THREADS + threadIdx.x;
    if (tally && me == 0) {
        tally[0] += uint32_t(noffs);
        tally[1] += start[noffs];
        tally[2] += start[noffs];
    }
    for (int o = 0; o < noffs; ++o) {
        const uint32_t a = start[o], e = start[o + 1];
        if (a == e) continue;
        walk_offset(item, a, e, threads, me, pre, off0 + o, next, prev, offset);
        if (gridDim.x > 1) {
            asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        } else {
            __syncthreads();
        }
    }
}


// Walks the meetings of offsets [off0, off0 + noffs), noffs <= WALK_MAX_OFFS;
// start (device) holds the first item of each offset and the end of the last.
inline void walk_meetings(const Meeting* item, const uint32_t* start, int off0, int noffs, const uint32_t* pre,
                          const unsigned long long* used, uint32_t cap, uint32_t entries, uint32_t* next,
                          uint32_t* prev, uint16_t* offset, unsigned long long* tally, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    // short lists meet a few hundred at a time: one block, whose barrier is
    // cheaper than the cluster's
    const unsigned blocks = entries > 16384 ? 8 : 1;
    at.val.clusterDim.x = blocks;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(WALK_THREADS);
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    CURC_CHECK(cudaLaunchKernelEx(&cfg, walk_kernel, item, start, off0, noffs, pre, used, cap, next, prev, offset,
                                  tally));
    CURC_LAUNCH_CHECK();
}

// The same with the starts known to the host: an offset with many meetings is
// walked by a grid of its own (one launch each, no barrier), the others
// between them by one cluster.
constexpr uint32_t WALK_GRID = 32768;
inline void walk_stage(const Meeting* item, const uint32_t* host_start, const uint32_t* start, int off0, int noffs,
                       const uint32_t* pre, const unsigned long long* used, uint32_t cap, uint32_t* next,
                       uint32_t* prev, uint16_t* offset, cudaStream_t s) {
    for (int o = 0; o < noffs;) {
        const uint32_t n = host_start[o + 1] - host_start[o];
        if (n > WALK_GRID) {
            walk_one_kernel<<<resident_grid(walk_one_kernel, 256, n), 256, 0, s>>>(
                item, host_start[o], host_start[o + 1], off0 + o, pre, next, prev, offset);
            CURC_LAUNCH_CHECK();
            ++o;
            continue;
        }
        int e = o + 1;
        uint32_t most = n;
        while (e < noffs && host_start[e + 1] - host_start[e] <= WALK_GRID) {
            most = std::max(most, host_start[e + 1] - host_start[e]);
            ++e;
        }
        if (host_start[e] != host_start[o])
            walk_meetings(item, start + o, off0 + o, e - o, pre, used, cap, most * 8, next, prev, offset, nullptr, s);
        o = e;
    }
}

}  // namespace curc
