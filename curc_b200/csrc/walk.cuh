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
#include "primitives.cuh"

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

// What a walk did, where it is counted: links made, and the free suffixes of
// runs with a free prefix that two or more of them met.
struct Walked {
    uint32_t links = 0, contested = 0;
    __device__ __forceinline__ void met(uint32_t free_members) { contested += free_members > 1 ? free_members : 0; }
};

// The suffixes of one run (items [i, e) with the same lo, in order) each take
// the first free prefix that is not themselves, as the reference's merge of
// the run does (its rotation puts a prefix that meets itself back in front).
// One thread.  Returns the free suffixes it met from item `from` on, where that
// is counted: all of them, unless there was no free prefix to begin with.
template <bool COUNT>
__device__ __forceinline__ uint32_t walk_run(const Meeting* __restrict__ item, uint32_t i, uint32_t e,
                                             const uint32_t* __restrict__ pre, uint32_t q0, uint32_t hi, int off,
                                             uint32_t* next, uint32_t* prev, uint16_t* offset, uint32_t from,
                                             Walked& w) {
    const uint32_t lo = item[i].lo;
    uint32_t met = 0;
    bool any = true, had = false;  // a free prefix was left; there was one
    for (; i < e && item[i].lo == lo; ++i) {
        const uint32_t s = item[i].s;
        if (ld_l2(next + s) != INVALID) continue;
        if (COUNT) {
            met += i >= from;
            if (!any) continue;
        }
        any = false;
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
            if (COUNT) ++w.links;
            break;
        }
        had |= any;
        if (!any && (!COUNT || !had)) return 0;
    }
    return met;
}

// The same by a whole warp, for long runs: free suffixes and free prefixes
// are taken 32 at a time and paired in order; where a read would meet itself
// the rest of the run is walked by one lane.  Lane 0 counts.
template <bool COUNT>
static __device__ void walk_run_warp(const Meeting* __restrict__ item, uint32_t i, uint32_t e,
                                     const uint32_t* __restrict__ pre, uint32_t q, uint32_t hi, int off, uint32_t* next,
                                     uint32_t* prev, uint16_t* offset, Walked& w) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t lo = item[i].lo;
    uint32_t sm = 0, pm = 0;          // free entries of the current 32 items / prefixes
    uint32_t ib = i, qb = q;          // where the next 32 start
    uint32_t s = 0, p = 0;            // this lane's entries
    uint32_t met = 0;
    bool more_s = true, had = false;  // had: there was a free prefix
    for (;;) {
        while (sm == 0 && more_s) {
            const uint32_t t = ib + lane;
            const bool in = t < e && item[t].lo == lo;
            const uint32_t all = __ballot_sync(0xFFFFFFFFu, in);
            s = in ? item[t].s : 0;
            sm = __ballot_sync(0xFFFFFFFFu, in && ld_l2(next + s) == INVALID);
            if (COUNT) met += __popc(sm);
            ib += 32;
            more_s = all == 0xFFFFFFFFu;
        }
        if (sm == 0) break;
        while (pm == 0 && qb < hi) {
            const uint32_t t = qb + lane;
            const bool in = t < hi;
            p = in ? pre[t] : 0;
            pm = __ballot_sync(0xFFFFFFFFu, in && ld_l2(prev + p) == INVALID);
            qb += 32;
        }
        if (pm == 0) {
            if (COUNT && !had) return;
            break;
        }
        had = true;
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
        if (COUNT && lane == 0) w.links += uint32_t(good);
        if (self) {
            if (lane == 0) met += walk_run<COUNT>(item, ib - 32, e, pre, qb - 32, hi, off, next, prev, offset, ib, w);
            __syncwarp();
            more_s = false;
            break;
        }
        for (int k = 0; k < n; ++k) {  // the n lowest of each are used up
            sm &= sm - 1;
            pm &= pm - 1;
        }
    }
    if (COUNT) {
        uint32_t left = 0;  // free suffixes for which no prefix is left, eight a lane at a time
        for (; more_s; ib += 256) {
            uint32_t sv[8], in = 0;
#pragma unroll
            for (uint32_t k = 0; k < 8; ++k) {
                const uint32_t t = ib + 32 * k + lane;
                const bool is = t < e && item[t].lo == lo;
                sv[k] = is ? item[t].s : 0;
                in |= uint32_t(is) << k;
            }
#pragma unroll
            for (uint32_t k = 0; k < 8; ++k)
                if (in >> k & 1u) left += ld_l2(next + sv[k]) == INVALID;
            more_s = __all_sync(0xFFFFFFFFu, in >> 7);
        }
        met += __reduce_add_sync(0xFFFFFFFFu, left);
        if (lane == 0) w.met(met);
    }
}

constexpr int WALK_THREADS = 512;
constexpr int WALK_MAX_OFFS = 512;

// The meetings [a, e) of one offset by `threads` threads, of which this is
// number me: one thread per run, long runs by a warp.
template <bool COUNT>
static __device__ __forceinline__ void walk_offset(const Meeting* __restrict__ item, uint32_t a, uint32_t e,
                                                   uint32_t threads, uint32_t me, const uint32_t* __restrict__ pre,
                                                   int off, uint32_t* next, uint32_t* prev, uint16_t* offset,
                                                   Walked& w) {
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
                            if (COUNT) ++w.links;
                        }
                    }
                } else {
                    // more than a few members or prefixes: by the whole warp
                    long_run = it.hi - it.lo > 8 || (i + 8 < e && item[i + 8].lo == it.lo);
                    if (!long_run) {
                        const uint32_t met =
                            walk_run<COUNT>(item, i, e, pre, it.lo, it.hi, off, next, prev, offset, i, w);
                        if (COUNT) w.met(met);
                    }
                }
            }
        }
        uint32_t todo = __ballot_sync(0xFFFFFFFFu, long_run);
        while (todo) {
            const int l = __ffs(todo) - 1;
            todo &= todo - 1;
            const uint32_t ii = __shfl_sync(0xFFFFFFFFu, i, l), lo = __shfl_sync(0xFFFFFFFFu, it.lo, l),
                           hi = __shfl_sync(0xFFFFFFFFu, it.hi, l);
            walk_run_warp<COUNT>(item, ii, e, pre, lo, hi, off, next, prev, offset, w);
        }
    }
}

// A run of up to FEW suffixes and FEW prefixes, by the thread of its first
// meeting: its reads, which do not depend on the links and are loaded ahead
// of the barrier.  ns = 0: not a run's first meeting; np = 0: a longer run.
constexpr uint32_t FEW = 4;
struct Ahead {
    uint32_t s[FEW], p[FEW];
    uint32_t ns, np;
};
__device__ __forceinline__ Ahead look_ahead(const Meeting* __restrict__ item, uint32_t a, uint32_t e, uint32_t i,
                                            const uint32_t* __restrict__ pre) {
    Ahead h;
    h.ns = h.np = 0;
    if (i >= e) return h;
    const Meeting it = item[i];
    if (i > a && item[i - 1].lo == it.lo) return h;
    h.s[0] = it.s;
    h.p[0] = it.p;
    h.ns = 1;
#pragma unroll
    for (uint32_t k = 1; k <= FEW; ++k) {
        if (h.ns < k || i + k >= e) continue;
        const Meeting m = item[i + k];
        if (m.lo != it.lo) continue;
        h.ns = k + 1;
        if (k < FEW) h.s[k] = m.s;
    }
    if (h.ns > FEW || it.hi - it.lo > FEW) return h;
    h.np = it.hi - it.lo;
#pragma unroll
    for (uint32_t k = 1; k < FEW; ++k)
        if (k < h.np) h.p[k] = pre[it.lo + k];
    return h;
}

// The same with the runs read ahead (h: this thread's first): one thread per
// run of few, whose links are loaded together and paired in registers, longer
// runs by a warp.  Where the overlap stage walks thousands of meetings an
// offset, mostly of runs of one to three, a thread's chain of ten dependent
// loads was what an offset took; where an offset has few meetings, as in the
// full match, the plain form is the shorter one.
template <bool COUNT>
static __device__ __forceinline__ void walk_offset_ahead(const Meeting* __restrict__ item, uint32_t a, uint32_t e,
                                                         uint32_t threads, uint32_t me, Ahead h,
                                                         const uint32_t* __restrict__ pre, int off, uint32_t* next,
                                                         uint32_t* prev, uint16_t* offset, Walked& w) {
    for (uint32_t i0 = a;;) {  // the same trip count for a whole warp
        if (h.np) {
            uint32_t fs = 0, fp = 0;  // free suffixes and prefixes
#pragma unroll
            for (uint32_t k = 0; k < FEW; ++k) {
                if (k < h.ns && ld_l2(next + h.s[k]) == INVALID) fs |= 1u << k;
                if (k < h.np && ld_l2(prev + h.p[k]) == INVALID) fp |= 1u << k;
            }
            if (COUNT && fp) w.met(__popc(fs));
#pragma unroll
            for (uint32_t k = 0; k < FEW; ++k) {
                if (!(fs >> k & 1u)) continue;
                bool open = true;
#pragma unroll
                for (uint32_t q = 0; q < FEW; ++q)
                    if (open && (fp >> q & 1u) && h.p[q] != h.s[k]) {
                        open = false;
                        fp &= ~(1u << q);
                        next[h.s[k]] = h.p[q];
                        prev[h.p[q]] = h.s[k];
                        offset[h.s[k]] = uint16_t(off);
                        if (COUNT) ++w.links;
                    }
            }
        }
        uint32_t todo = __ballot_sync(0xFFFFFFFFu, h.ns && !h.np);
        while (todo) {
            const int l = __ffs(todo) - 1;
            todo &= todo - 1;
            const uint32_t ii = i0 + me - (threadIdx.x & 31u) + l;
            const Meeting it = item[ii];
            walk_run_warp<COUNT>(item, ii, e, pre, it.lo, it.hi, off, next, prev, offset, w);
        }
        i0 += threads;
        if (i0 >= e) return;
        h = look_ahead(item, a, e, i0 + me, pre);
    }
}

// A warp's counts to counts[0] (links) and counts[1] (contested).
__device__ __forceinline__ void add_walked(const Walked& w, unsigned long long* counts) {
    const uint32_t l = __reduce_add_sync(0xFFFFFFFFu, w.links), c = __reduce_add_sync(0xFFFFFFFFu, w.contested);
    if ((threadIdx.x & 31u) != 0) return;
    if (l) atomicAdd(counts, static_cast<unsigned long long>(l));
    if (c) atomicAdd(counts + 1, static_cast<unsigned long long>(c));
}

// One offset by a whole grid.
static __global__ void __launch_bounds__(256) walk_one_kernel(const Meeting* __restrict__ item, uint32_t a, uint32_t e,
                                                              int off, const uint32_t* __restrict__ pre, uint32_t* next,
                                                              uint32_t* prev, uint16_t* offset,
                                                              unsigned long long* __restrict__ counts) {
    const uint32_t me = blockIdx.x * 256 + threadIdx.x;
    Walked w;
    if (a < e)
        walk_offset_ahead<true>(item, a, e, gridDim.x * 256, me, look_ahead(item, a, e, a + me, pre), pre, off, next,
                                prev, offset, w);
    add_walked(w, counts);
}

// The walk: offset after offset, one thread per run of equal suffix strings
// (long runs: a warp).  Runs of one offset share no read, so an offset's runs
// are independent; a barrier over the cluster separates the offsets.  One
// cluster suffices: an offset has few meetings (thousands at most where a
// list has 400,000 entries), and its time is the latency of its dependent
// loads, the sectors that 8 or 16 SMs can ask for, and the barrier.  With
// AHEAD the next offset's runs are read between the barrier's two halves.
// Overlap stage on B200, 8 blocks plain, 16 blocks plain, 16 with AHEAD: 100k
// pairs 0.64, 0.44, 0.37 ms; 700k reads of 251 1.00, 0.90, 0.75; 8M of 250
// 3.22, 2.56, 2.09 (blocks of 256 or 1024 threads: slower, as is AHEAD in one
// block: 64 offsets of 83 meetings 0.133 -> 0.158).
// COUNT: links and contested suffixes go to counts; else counts, if given, are
// the full match's (offsets passed, and twice the meetings).
template <bool AHEAD, bool COUNT>
static __global__ void __launch_bounds__(WALK_THREADS) walk_kernel(const Meeting* __restrict__ item,
                                                                   const uint32_t* __restrict__ start_in, int off0,
                                                                   int noffs, const uint32_t* __restrict__ pre,
                                                                   const unsigned long long* __restrict__ used,
                                                                   uint32_t cap, uint32_t* next, uint32_t* prev,
                                                                   uint16_t* offset,
                                                                   unsigned long long* __restrict__ counts) {
    __shared__ uint32_t start[WALK_MAX_OFFS + 1];
    if (*used > cap) return;  // the listing is incomplete: the caller repeats it
    for (int o = threadIdx.x; o <= noffs; o += WALK_THREADS) start[o] = start_in[o];
    __syncthreads();
    const uint32_t threads = gridDim.x * WALK_THREADS, me = blockIdx.x * WALK_THREADS + threadIdx.x;
    if (!COUNT && counts && me == 0) {
        counts[0] += uint32_t(noffs);
        counts[1] += start[noffs];
        counts[2] += start[noffs];
    }
    Walked w;
    auto skip = [&](int o) {  // the next offset with meetings
        while (o < noffs && start[o] == start[o + 1]) ++o;
        return o;
    };
    int o = skip(0);
    if (o == noffs) return;
    Ahead h;
    if (AHEAD) h = look_ahead(item, start[o], start[o + 1], start[o] + me, pre);
    for (;;) {
        if (AHEAD)
            walk_offset_ahead<COUNT>(item, start[o], start[o + 1], threads, me, h, pre, off0 + o, next, prev, offset, w);
        else
            walk_offset<COUNT>(item, start[o], start[o + 1], threads, me, pre, off0 + o, next, prev, offset, w);
        o = skip(o + 1);
        if (o == noffs) break;
        if (gridDim.x > 1) cluster_arrive();
        if (AHEAD) h = look_ahead(item, start[o], start[o + 1], start[o] + me, pre);
        if (gridDim.x > 1) cluster_wait();
        else __syncthreads();
    }
    if (COUNT) add_walked(w, counts);
}

constexpr unsigned WALK_CLUSTER = 16;

// Walks the meetings of offsets [off0, off0 + noffs), noffs <= WALK_MAX_OFFS;
// start (device) holds the first item of each offset and the end of the last.
static inline void walk_meetings(const Meeting* item, const uint32_t* start, int off0, int noffs, const uint32_t* pre,
                                 const unsigned long long* used, uint32_t cap, uint32_t entries, uint32_t* next,
                                 uint32_t* prev, uint16_t* offset, unsigned long long* tally, cudaStream_t s) {
    // short lists meet a few hundred at a time: one block, whose barrier is
    // cheaper than the cluster's (50k reads, 2,048 to 4,096 ends: full match
    // 0.33 against 0.36 ms; 100k reads, more ends: 0.60 against 0.53)
    launch_cluster(walk_kernel<false, false>, entries > 4096 ? WALK_CLUSTER : 1, WALK_THREADS, s, item, start, off0, noffs, pre,
                   used, cap, next, prev, offset, tally);
}

// The same with the starts known to the host: an offset with many meetings is
// walked by a grid of its own (one launch each, no barrier), the others
// between them by one cluster.
constexpr uint32_t WALK_GRID = 32768;
static inline void walk_stage(const Meeting* item, const uint32_t* host_start, const uint32_t* start, int off0, int noffs,
                       const uint32_t* pre, const unsigned long long* used, uint32_t cap, uint32_t* next,
                       uint32_t* prev, uint16_t* offset, unsigned long long* counts, cudaStream_t s) {
    for (int o = 0; o < noffs;) {
        const uint32_t n = host_start[o + 1] - host_start[o];
        if (n > WALK_GRID) {
            walk_one_kernel<<<resident_grid(walk_one_kernel, 256, n), 256, 0, s>>>(
                item, host_start[o], host_start[o + 1], off0 + o, pre, next, prev, offset, counts);
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
        if (host_start[e] != host_start[o]) {
            const bool many = most > 2048;
            launch_cluster(many ? walk_kernel<true, true> : walk_kernel<false, true>, many ? WALK_CLUSTER : 1,
                           WALK_THREADS, s, item, start + o, off0 + o, e - o, pre, used, cap, next, prev, offset, counts);
        }
        o = e;
    }
}

}  // namespace curc
