// Decoupled look-back: the sum over the tiles before a tile, in one launch.
//
// Tiles are taken in order from a counter, so the blocks of all earlier tiles
// have started.  A tile publishes its own sum at once and the sum up to and
// with itself as soon as it knows it; the next tiles add up what they find.
//
// Waits are bounded, and none can fail: a tile that has waited LOOK_SPINS
// reads for another waits no more, and adds up the items of the tiles it has
// not heard from itself, from the kernel's input.  (It never came to that in any measurement: a block that
// has started publishes within microseconds, and a wait lasts 0.1 s.)
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

namespace curc {

// Reads of a state before its tile is not waited for any longer.
#ifndef CURC_LOOK_SPINS
#define CURC_LOOK_SPINS (1u << 22)
#endif
constexpr uint32_t LOOK_SPINS = CURC_LOOK_SPINS;

// A tile's state: a flag (0 nothing yet, 1 the tile's own sum, 2 the sum up
// to and with the tile) and the sum.  States of a single launch, zeroed before
// it; sums below 2^62.
struct LookOnce {
    __device__ __forceinline__ uint64_t make(uint32_t flag, uint64_t v) const {
        return uint64_t(flag) << 62 | (v & ((1ull << 62) - 1));
    }
    __device__ __forceinline__ uint32_t flag(uint64_t s) const { return uint32_t(s >> 62); }
    __device__ __forceinline__ uint64_t sum(uint64_t s) const { return s & ((1ull << 62) - 1); }
};

// States that carry the launch's number (never 0 in 30 bits), so that those of
// earlier launches need not be cleared; sums below 2^32.
struct LookEpoch {
    uint32_t epoch;
    __device__ __forceinline__ uint64_t make(uint32_t flag, uint64_t v) const {
        return uint64_t(epoch) << 34 | uint64_t(flag) << 32 | uint32_t(v);
    }
    __device__ __forceinline__ uint32_t flag(uint64_t s) const {
        return uint32_t(s >> 34) == epoch ? uint32_t(s >> 32) & 3u : 0u;
    }
    __device__ __forceinline__ uint64_t sum(uint64_t s) const { return uint32_t(s); }
};

// A state that is set, or an unset one once no reads are left.
template <class S>
__device__ __forceinline__ uint64_t look_wait(const S& S_, const unsigned long long* st, uint32_t& spins) {
    for (;;) {
        const uint64_t v = *reinterpret_cast<const volatile unsigned long long*>(st);
        if (S_.flag(v) || spins == 0) return v;
        --spins;
        __nanosleep(32);
    }
}

// Sum of a value over the warp's lanes.
__device__ __forceinline__ uint64_t warp_sum(uint64_t v) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, d);
    return v;
}

// The rest of a look-back without waits: the sum of the tiles up to and with
// `top`, one after another; those not heard from are counted.  Out of line, to
// keep its registers out of the kernels.
template <class S, class Count>
__device__ __noinline__ uint64_t look_on(S S_, unsigned long long* st, uint32_t top, bool in_place, Count count) {
    uint64_t before = 0;
    for (uint32_t j = top;; --j) {
        uint32_t spins = 0;
        uint64_t v = __shfl_sync(0xFFFFFFFFu, look_wait(S_, &st[j], spins), 0);
        if (!S_.flag(v)) {
            const uint64_t own = count(j);
            if (in_place) {  // it holds if the tile is silent still
                __threadfence();
                v = __shfl_sync(0xFFFFFFFFu, look_wait(S_, &st[j], spins), 0);
            }
            if (!S_.flag(v)) v = S_.make(1, own);
        }
        before += S_.sum(v);
        if (S_.flag(v) == 2 || j == 0) return before;
    }
}

// One warp, all lanes: publishes the tile's sum and returns the sum of the
// tiles before it (32 predecessors per step).  count(j), called by all lanes,
// is tile j's sum from the input.  in_place: the kernel overwrites its input
// behind this call, so what count() read only holds while the tile has not
// published, which happens before it writes.
template <class S, class Count>
__device__ __forceinline__ uint64_t look_back(const S& S_, unsigned long long* st, uint32_t tile, uint64_t sum,
                                              bool in_place, Count count) {
    const uint32_t lane = threadIdx.x & 31u;
    if (lane == 0) {
        atomicExch(&st[tile], S_.make(tile == 0 ? 2 : 1, sum));
        if (in_place) __threadfence();
    }
    if (tile == 0) return 0;
    uint64_t before = 0;
    for (int64_t top = int64_t(tile) - 1;; top -= 32) {
        const int64_t j = top - int64_t(lane);
        uint64_t v = S_.make(2, 0);  // lanes past tile 0 add nothing
        uint32_t spins = LOOK_SPINS;
        if (j >= 0) v = look_wait(S_, &st[j], spins);
        __syncwarp();
        if (__any_sync(0xFFFFFFFFu, S_.flag(v) == 0)) {
            before += look_on(S_, st, uint32_t(top), in_place, count);
            break;
        }
        // the nearest lane with an inclusive sum ends the search
        const uint32_t inc = __ballot_sync(0xFFFFFFFFu, S_.flag(v) == 2);
        const int stop = inc ? __ffs(inc) - 1 : 32;
        before += warp_sum(int(lane) <= stop ? S_.sum(v) : 0);
        if (inc) break;
    }
    if (lane == 0) atomicExch(&st[tile], S_.make(2, before + sum));
    return before;
}

}  // namespace curc
