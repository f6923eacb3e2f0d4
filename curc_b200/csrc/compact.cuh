// Stable compaction in one launch, with the item count read on the device.
//
// Tiles of CP_TILE items are taken in order from an atomic counter; each
// tile ranks its kept items with one block scan and finds its output offset
// by looking back over the tiles before it (lookback.cuh).  Because the count
// is read on the device, loops of data-dependent passes can be queued without
// a host round trip per pass.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

#include "common.cuh"
#include "lookback.cuh"
#include "primitives.cuh"

namespace curc {

constexpr int CP_THREADS = 512;
constexpr int CP_ITEMS = 8;
constexpr uint32_t CP_TILE = CP_THREADS * CP_ITEMS;

// Items kept of a tile not heard from (an earlier one is full).
template <class Keep>
__device__ __forceinline__ uint64_t kept_in_tile(const Keep& keep, uint32_t j) {
    uint64_t c = 0;
#pragma unroll 1
    for (uint32_t i = threadIdx.x; i < CP_TILE; i += 32) c += keep(j * CP_TILE + i) ? 1 : 0;  // warp 0
    return warp_sum(c);
}

// keep(i) -> bool for item i < n; move(i, dst) places kept item i at dst.
// Each thread takes CP_ITEMS consecutive items; one block scan ranks them.
// The grid covers *n_dev items; keep() gives the same for an item whenever it
// is asked.
template <class Keep, class Move>
__global__ void __launch_bounds__(CP_THREADS, 4) compact_kernel(const uint32_t* __restrict__ n_dev,
                                                             uint32_t* __restrict__ n_out, Keep keep, Move move,
                                                             unsigned long long* tiles, uint32_t* counter,
                                                             uint32_t base, uint32_t epoch) {
    __shared__ uint32_t s_tile, s_excl, s_warp[CP_THREADS / 32];
    const uint32_t n = uint32_t(min(uint64_t(*n_dev), uint64_t(gridDim.x) * CP_TILE));
    if (threadIdx.x == 0) s_tile = atomicAdd(counter, 1u) - base;
    __syncthreads();
    const uint32_t tile = s_tile;
    const uint64_t start = uint64_t(tile) * CP_TILE;
    if (start >= n && tile != 0) return;  // beyond the items; nobody looks back at it
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint64_t first = start + uint64_t(threadIdx.x) * CP_ITEMS;
    uint32_t kept = 0;  // bit r: item first + r is kept
#pragma unroll
    for (int r = 0; r < CP_ITEMS; ++r) {
        const uint64_t i = first + r;
        if (i < n && keep(uint32_t(i))) kept |= 1u << r;
    }
    // block-wide exclusive scan of the per-thread counts
    const uint32_t mine = __popc(kept);
    uint32_t incl = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, d);
        if (lane >= uint32_t(d)) incl += v;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    uint32_t before = 0, local = 0;
#pragma unroll
    for (int w = 0; w < CP_THREADS / 32; ++w) {
        const uint32_t c = s_warp[w];
        before += w < int(warp) ? c : 0;
        local += c;
    }
    const uint32_t rank = before + incl - mine;
    if (warp == 0) {
        const uint32_t excl = uint32_t(look_back(LookEpoch{epoch}, tiles, tile, local, false, [&](uint32_t j) {
            return kept_in_tile(keep, j);
        }));
        if (lane == 0) {
            s_excl = excl;
            if (start + CP_TILE >= n) *n_out = excl + local;
        }
    }
    __syncthreads();
    uint32_t d = s_excl + rank;
#pragma unroll
    for (int r = 0; r < CP_ITEMS; ++r)
        if ((kept >> r) & 1u) move(uint32_t(first + r), d++);
}

// Owns the tile states of a sequence of compactions on one stream (epoch and
// tile base kept on the host, one launch per compaction).
class Compactor {
public:
    Compactor(uint32_t max_items, Arena& a, cudaStream_t s) : s_(s) {
        max_tiles_ = uint32_t(div_up(uint64_t(max_items ? max_items : 1), uint64_t(CP_TILE)));
        tiles_ = a.zeros<unsigned long long>(max_tiles_, s);
        counter_ = a.zeros<uint32_t>(1, s);
    }
    // Compacts the first *n_dev (<= max_items) items; *n_out = number kept.
    template <class Keep, class Move>
    void run(const uint32_t* n_dev, uint32_t n_max, uint32_t* n_out, Keep keep, Move move) {
        const uint32_t grid = grid_for_items(n_max);
        ++epoch_;
        compact_kernel<Keep, Move><<<grid, CP_THREADS, 0, s_>>>(n_dev, n_out, keep, move, tiles_, counter_, base_,
                                                                  epoch_);
        CURC_LAUNCH_CHECK();
        base_ += grid;
    }

private:
    uint32_t grid_for_items(uint32_t n_max) const {
        const uint32_t grid = uint32_t(div_up(uint64_t(n_max ? n_max : 1), uint64_t(CP_TILE)));
        if (grid > max_tiles_) throw std::runtime_error("Compactor: more items than it was sized for");
        return grid;
    }
    cudaStream_t s_;
    uint32_t max_tiles_ = 0, base_ = 0, epoch_ = 0;
    unsigned long long* tiles_ = nullptr;
    uint32_t* counter_ = nullptr;
};

}  // namespace curc
