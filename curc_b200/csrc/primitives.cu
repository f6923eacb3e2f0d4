// Device-wide primitives: arena, scan, stable compaction, stable radix sort.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <stdexcept>
#include <string>

#include <mutex>

#include "lookback.cuh"
#include "primitives.cuh"

namespace curc {

namespace {
std::atomic<uint64_t> g_launches{0};
}
void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }
uint64_t launches() { return g_launches.load(); }

// ---------------------------------------------------------------- arena

Arena::~Arena() {
    for (auto& c : chunks_) cudaFree(c.base);
    if (zero_) cudaFree(zero_);
}

void Arena::clear_zeros(cudaStream_t s) {
    zero_used_ = ZERO_POOL;
    if (!zero_ && cudaMalloc(&zero_, ZERO_POOL) != cudaSuccess) {
        cudaGetLastError();  // no room: pieces are cleared one by one
        zero_ = nullptr;
        return;
    }
    CURC_CHECK(cudaMemsetAsync(zero_, 0, ZERO_POOL, s));
    zero_used_ = 0;
    zero_stream_ = s;
}

void* Arena::zero_bytes(size_t bytes, cudaStream_t s) {
    const size_t take = (bytes + 255) & ~size_t(255);
    if (take <= ZERO_PIECE && zero_used_ + take <= ZERO_POOL && s == zero_stream_) {
        void* p = zero_ + zero_used_;
        zero_used_ += take;
        return p;
    }
    void* p = alloc_bytes(bytes);
    CURC_CHECK(cudaMemsetAsync(p, 0, bytes, s));
    return p;
}

void* Arena::alloc_bytes(size_t bytes) {
    bytes = (bytes + 255) & ~size_t(255);
    if (bytes == 0) bytes = 256;
    while (cur_ < chunks_.size()) {
        Chunk& c = chunks_[cur_];
        if (c.used + bytes <= c.size) {
            void* p = c.base + c.used;
            c.used += bytes;
            high_water_ = std::max(high_water_, in_use());
            return p;
        }
        // chunks after the current one are free: take the first that is
        // large enough, moved up to follow the current one
        size_t fit = cur_ + 1;
        while (fit < chunks_.size() && chunks_[fit].size < bytes) ++fit;
        if (fit < chunks_.size()) {
            std::rotate(chunks_.begin() + cur_ + 1, chunks_.begin() + fit, chunks_.begin() + fit + 1);
            ++cur_;
            chunks_[cur_].used = 0;
            continue;
        }
        break;
    }
    size_t sz = std::max(bytes, chunk_);
    char* p = nullptr;
    if (cudaMalloc(&p, sz) != cudaSuccess) {
        // out of memory: give back the free chunks (all too small) and retry
        cudaGetLastError();
        const size_t keep = chunks_.empty() ? 0 : cur_ + 1;
        for (size_t i = keep; i < chunks_.size(); ++i) CURC_CHECK(cudaFree(chunks_[i].base));
        chunks_.resize(keep);
        if (cudaMalloc(&p, sz) != cudaSuccess) {
            cudaGetLastError();
            size_t held = 0, fr = 0, tot = 0;
            for (const auto& c : chunks_) held += c.size;
            cudaMemGetInfo(&fr, &tot);
            const std::string msg = "arena: out of device memory for " + std::to_string(sz >> 20) +
                                    " MiB (the arena holds " + std::to_string(held >> 20) + " MiB in " +
                                    std::to_string(chunks_.size()) + " chunks; " + std::to_string(fr >> 20) +
                                    " MiB free on the device)";
            throw CudaError(cudaErrorMemoryAllocation, msg.c_str());
        }
    }
    // keep chunks ordered as used: insert after the current one
    Chunk c{p, sz, bytes};
    if (chunks_.empty()) {
        chunks_.push_back(c);
        cur_ = 0;
    } else {
        chunks_.insert(chunks_.begin() + cur_ + 1, c);
        ++cur_;
        for (size_t i = cur_ + 1; i < chunks_.size(); ++i) chunks_[i].used = 0;
    }
    high_water_ = std::max(high_water_, in_use());
    return p;
}

size_t Arena::in_use() const {
    size_t u = 0;
    for (size_t i = 0; i <= cur_ && i < chunks_.size(); ++i) u += chunks_[i].used;
    return u;
}

void Arena::reset() {
    // Several chunks (blocks of changing sizes grew the arena): give them
    // back and keep one chunk that holds the largest run seen, so later runs
    // allocate nothing and chunks do not pile up.  Nothing is in use here.
    if (chunks_.size() > 1) {
        const size_t mib = size_t(1) << 20;
        const size_t need = std::max(chunk_, (high_water_ + mib - 1) / mib * mib);
        for (auto& c : chunks_) CURC_CHECK(cudaFree(c.base));
        chunks_.clear();
        char* p = nullptr;
        if (cudaMalloc(&p, need) == cudaSuccess)
            chunks_.push_back(Chunk{p, need, 0});
        else
            cudaGetLastError();  // no room for one chunk: allocate on demand again
    }
    for (auto& c : chunks_) c.used = 0;
    cur_ = 0;
}

void Arena::trim() {
    if (zero_) CURC_CHECK(cudaFree(zero_));
    zero_ = nullptr;
    zero_used_ = ZERO_POOL;
    for (auto& c : chunks_) CURC_CHECK(cudaFree(c.base));
    chunks_.clear();
    cur_ = 0;
    high_water_ = 0;
}

void Arena::release(const Mark& m) {
    if (chunks_.empty()) return;
    for (size_t i = m.chunk + 1; i < chunks_.size(); ++i) chunks_[i].used = 0;
    cur_ = m.chunk;
    if (cur_ < chunks_.size()) chunks_[cur_].used = m.used;
}

// ---------------------------------------------------------------- small reads

namespace {
constexpr size_t READ_SMALL_MAX = 4096;

__global__ void read_small_kernel(const uint8_t* __restrict__ src, size_t bytes, uint8_t* dst) {
    for (size_t i = threadIdx.x; i < bytes; i += blockDim.x) dst[i] = src[i];
}

// Mapped pinned buffer of this host thread (portable: valid on every device
// through unified addressing), allocated on first use and kept until exit.
uint8_t* thread_readback_buffer() {
    thread_local struct Buf {
        uint8_t* p = nullptr;
        ~Buf() {
            if (p) cudaFreeHost(p);
        }
    } b;
    if (!b.p)
        CURC_CHECK(cudaHostAlloc(reinterpret_cast<void**>(&b.p), READ_SMALL_MAX,
                                 cudaHostAllocMapped | cudaHostAllocPortable));
    return b.p;
}
}  // namespace

void read_small(void* host, const void* dev, size_t bytes, cudaStream_t s) {
    if (bytes == 0) return;
    if (bytes > READ_SMALL_MAX) throw std::runtime_error("read_small: more than 4 KiB");
    uint8_t* buf = thread_readback_buffer();
    read_small_kernel<<<1, 128, 0, s>>>(static_cast<const uint8_t*>(dev), bytes, buf);
    CURC_LAUNCH_CHECK();
    CURC_CHECK(cudaStreamSynchronize(s));
    std::memcpy(host, buf, bytes);
}

// ---------------------------------------------------------------- pinned arena

PinnedArena::~PinnedArena() {
    for (auto& c : chunks_) cudaFreeHost(c.base);
}

PinnedArena& PinnedArena::operator=(PinnedArena&& o) noexcept {
    if (this != &o) {
        for (auto& c : chunks_) cudaFreeHost(c.base);
        chunks_ = std::move(o.chunks_);
        cur_ = o.cur_;
        o.chunks_.clear();
        o.cur_ = 0;
    }
    return *this;
}

uint8_t* PinnedArena::alloc(size_t bytes) {
    bytes = (bytes + 63) & ~size_t(63);
    while (cur_ < chunks_.size()) {
        Chunk& c = chunks_[cur_];
        if (c.used + bytes <= c.size) {
            uint8_t* p = c.base + c.used;
            c.used += bytes;
            return p;
        }
        ++cur_;
    }
    Chunk c{nullptr, std::max(bytes, size_t(256) << 20), 0};
    CURC_CHECK(cudaHostAlloc(reinterpret_cast<void**>(&c.base), c.size, cudaHostAllocPortable));
    c.used = bytes;
    chunks_.push_back(c);
    cur_ = chunks_.size() - 1;
    return c.base;
}

void PinnedArena::reset() {
    for (auto& c : chunks_) c.used = 0;
    cur_ = 0;
}

// ---------------------------------------------------------------- stage timer

cudaEvent_t StageTimer::mark() {
    // (another thread's launches only make it record once more)
    if (!last_ || launches() != last_launches_) {
        last_launches_ = launches();
        last_ = pool_.take();
        CURC_CHECK(cudaEventRecord(last_, s_));
    }
    return last_;
}

size_t StageTimer::begin_span(const std::string& name) {
    ev_.push_back(Span{name, mark(), nullptr});
    return ev_.size() - 1;
}

void StageTimer::collect(std::map<std::string, float>& out) {
    CURC_CHECK(cudaStreamSynchronize(s_));
    for (auto& e : ev_) {
        float ms = 0;
        if (e.a != e.b) CURC_CHECK(cudaEventElapsedTime(&ms, e.a, e.b));
        out[e.name] += ms;
    }
    ev_.clear();
    open_.clear();
}

StageTimer*& active_timer() {
    thread_local StageTimer* t = nullptr;
    return t;
}

unsigned cluster_blocks(const void* kernel, unsigned most, unsigned threads) {
    if (most == 1) return 1;
    static std::mutex mu;
    static std::map<std::pair<int, const void*>, int> held;  // the largest the device can hold
    int dev = 0;
    CURC_CHECK(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> g(mu);
    int& h = held[{dev, kernel}];
    if (h == 0) {
        CURC_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(16);
        cfg.blockDim = dim3(threads);
        int n = 0;
        CURC_CHECK(cudaOccupancyMaxPotentialClusterSize(&n, kernel, &cfg));
        h = std::max(1, n);
    }
    return cluster_fit(most, unsigned(h));
}

// ---------------------------------------------------------------- scan

namespace {
constexpr int SCAN_THREADS = 256, SCAN_ITEMS = 16, SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

template <class T>
__device__ T block_exclusive_sum(T v, T* block_total) {
    __shared__ T warp_sums[SCAN_THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        T y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        T w = lane < SCAN_THREADS / 32 ? warp_sums[lane] : T(0);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            T y = __shfl_up_sync(0xFFFFFFFFu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < SCAN_THREADS / 32) warp_sums[lane] = w;
    }
    __syncthreads();
    T warp_prefix = warp ? warp_sums[warp - 1] : T(0);
    *block_total = warp_sums[SCAN_THREADS / 32 - 1];
    __syncthreads();
    return warp_prefix + x - v;
}

// Sum of a tile not heard from (lookback.cuh).  An earlier tile is full.
template <class T>
__device__ __forceinline__ uint64_t scan_tile_sum(const T* in) {
    uint64_t c = 0;
#pragma unroll 1
    for (int i = int(threadIdx.x); i < SCAN_TILE; i += 32) c += __ldcg(in + i);
    return warp_sum(c);
}

// One-pass scan (lookback.cuh).  st: one state per tile and, behind them, the
// tile counter (all zero).
template <class T>
__global__ void __launch_bounds__(SCAN_THREADS, sizeof(T) == 4 ? 6 : 5) scan_kernel(const T* in, T* out, size_t n, T* total,
                                                            unsigned long long* st, uint32_t tiles) {
    __shared__ T sm[SCAN_TILE];
    __shared__ uint32_t s_tile;
    __shared__ uint64_t s_before;
    if (threadIdx.x == 0) s_tile = tiles > 1 ? uint32_t(atomicAdd(&st[tiles], 1ull)) : 0;
    __syncthreads();
    const uint32_t tile = s_tile;
    const size_t base = size_t(tile) * SCAN_TILE;
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; ++i) {
        size_t idx = base + size_t(i) * SCAN_THREADS + threadIdx.x;
        sm[i * SCAN_THREADS + threadIdx.x] = idx < n ? in[idx] : T(0);
    }
    __syncthreads();
    T local[SCAN_ITEMS];
    T tsum = 0;
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; ++i) {
        local[i] = sm[threadIdx.x * SCAN_ITEMS + i];
        tsum += local[i];
    }
    T btotal;
    T run = block_exclusive_sum(tsum, &btotal);
    if (tiles > 1) {
        if (threadIdx.x < 32) {
            const uint64_t before = look_back(LookOnce{}, st, tile, uint64_t(btotal), in == out, [&](uint32_t j) {
                return scan_tile_sum(in + size_t(j) * SCAN_TILE);
            });
            if (threadIdx.x == 0) s_before = before;
        }
        __syncthreads();
        run += T(s_before);
    }
    if (total && tile + 1 == tiles && threadIdx.x == 0) *total = btotal + (tiles > 1 ? T(s_before) : T(0));
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; ++i) {
        T t = local[i];
        sm[threadIdx.x * SCAN_ITEMS + i] = run;
        run += t;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; ++i) {
        size_t idx = base + size_t(i) * SCAN_THREADS + threadIdx.x;
        if (idx < n) out[idx] = sm[i * SCAN_THREADS + threadIdx.x];
    }
}

// Zeroed tile states and counter of a one-pass kernel.
unsigned long long* look_states(size_t tiles, Arena& a, cudaStream_t s) {
    return a.zeros<unsigned long long>(tiles + 1, s);
}
}  // namespace

template <class T>
void exclusive_scan(const T* in, T* out, size_t n, T* total, Arena& a, cudaStream_t s) {
    if (n == 0) {
        if (total) CURC_CHECK(cudaMemsetAsync(total, 0, sizeof(T), s));
        return;
    }
    const size_t tiles = div_up(n, SCAN_TILE);
    auto m = a.mark();
    unsigned long long* st = tiles > 1 ? look_states(tiles, a, s) : nullptr;
    scan_kernel<T><<<unsigned(tiles), SCAN_THREADS, 0, s>>>(in, out, n, total, st, uint32_t(tiles));
    CURC_LAUNCH_CHECK();
    a.release(m);
}

template void exclusive_scan<uint32_t>(const uint32_t*, uint32_t*, size_t, uint32_t*, Arena&, cudaStream_t);
template void exclusive_scan<uint64_t>(const uint64_t*, uint64_t*, size_t, uint64_t*, Arena&, cudaStream_t);

// ---------------------------------------------------------------- compaction

namespace {
constexpr int SEL_THREADS = 256, SEL_ITEMS = 16, SEL_TILE = SEL_THREADS * SEL_ITEMS;
static_assert(SEL_THREADS == SCAN_THREADS, "block_exclusive_sum");

__device__ __forceinline__ uint64_t flagged_in_tile(const uint8_t* flags) {
    uint64_t c = 0;
#pragma unroll 1
    for (int i = int(threadIdx.x); i < SEL_TILE; i += 32) c += flags[i] != 0;
    return warp_sum(c);
}

// One-pass stable compaction (tile states as in scan_kernel); thread t owns
// the tile's items [16 t, 16 t + 16).
template <class T, bool kIndices>
__global__ void __launch_bounds__(SEL_THREADS, 8) select_kernel(const T* __restrict__ in, const uint8_t* __restrict__ flags,
                                                             size_t n, T* __restrict__ out, uint32_t* __restrict__ count,
                                                             unsigned long long* st, uint32_t tiles) {
    __shared__ uint32_t s_tile;
    __shared__ uint64_t s_before;
    if (threadIdx.x == 0) s_tile = tiles > 1 ? uint32_t(atomicAdd(&st[tiles], 1ull)) : 0;
    __syncthreads();
    const uint32_t tile = s_tile;
    const size_t base = size_t(tile) * SEL_TILE + size_t(threadIdx.x) * SEL_ITEMS;
    uint32_t keep = 0;  // bit i: item base + i
    if (base + SEL_ITEMS <= n && (reinterpret_cast<uintptr_t>(flags) & 15) == 0) {
        const uint4 f = *reinterpret_cast<const uint4*>(flags + base);
        const uint32_t w[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
        for (int i = 0; i < SEL_ITEMS; ++i) keep |= uint32_t(((w[i / 4] >> (8 * (i % 4))) & 0xFFu) != 0) << i;
    } else {
#pragma unroll
        for (int i = 0; i < SEL_ITEMS; ++i)
            if (base + i < n && flags[base + i]) keep |= 1u << i;
    }
    uint32_t total;
    uint64_t pos = block_exclusive_sum<uint32_t>(__popc(keep), &total);
    if (tiles > 1) {
        if (threadIdx.x < 32) {
            const uint64_t before = look_back(LookOnce{}, st, tile, total, false, [&](uint32_t j) {
                return flagged_in_tile(flags + size_t(j) * SEL_TILE);
            });
            if (threadIdx.x == 0) s_before = before;
        }
        __syncthreads();
        pos += s_before;
    }
    if (tile + 1 == tiles && threadIdx.x == 0) *count = total + (tiles > 1 ? uint32_t(s_before) : 0u);
    while (keep) {
        const int i = __ffs(keep) - 1;
        keep &= keep - 1;
        if constexpr (kIndices) out[pos] = T(base + i);
        else out[pos] = in[base + i];
        ++pos;
    }
}

template <class T, bool kIndices>
void select_impl(const T* in, const uint8_t* flags, T* out, size_t n, uint32_t* count, Arena& a, cudaStream_t s) {
    if (n == 0) {
        CURC_CHECK(cudaMemsetAsync(count, 0, sizeof(uint32_t), s));
        return;
    }
    auto m = a.mark();
    const size_t tiles = div_up(n, SEL_TILE);
    unsigned long long* st = tiles > 1 ? look_states(tiles, a, s) : nullptr;
    select_kernel<T, kIndices><<<unsigned(tiles), SEL_THREADS, 0, s>>>(in, flags, n, out, count, st, uint32_t(tiles));
    CURC_LAUNCH_CHECK();
    a.release(m);
}
}  // namespace

template <class T>
void select_flagged(const T* in, const uint8_t* flags, T* out, size_t n, uint32_t* count, Arena& a, cudaStream_t s) {
    select_impl<T, false>(in, flags, out, n, count, a, s);
}
template void select_flagged<uint32_t>(const uint32_t*, const uint8_t*, uint32_t*, size_t, uint32_t*, Arena&,
                                       cudaStream_t);
template void select_flagged<uint64_t>(const uint64_t*, const uint8_t*, uint64_t*, size_t, uint32_t*, Arena&,
                                       cudaStream_t);

void select_indices(const uint8_t* flags, uint32_t* out, size_t n, uint32_t* count, Arena& a, cudaStream_t s) {
    select_impl<uint32_t, true>(nullptr, flags, out, n, count, a, s);
}

// ---------------------------------------------------------------- radix sort

namespace {
constexpr int RS_THREADS = 256, RS_WARPS = RS_THREADS / 32;
// Items per thread of a pass, and of a pass over few items.
constexpr int RS_ROUNDS = 16, RS_ROUNDS_FEW = 4, RS_TILE = RS_THREADS * RS_ROUNDS;
// Few: less than one full tile per SM.  A tile of 4 rounds is ranked in a
// quarter of the time and the SMs are not idle; with more items its longer
// look-back and shorter runs cost more than that gives.  Sort of 50k reads
// 0.167 -> 0.11 ms, 200k 0.19 -> 0.155, 700k and more unchanged or slower.
constexpr size_t RS_FEW = size_t(SM_COUNT_B200) * RS_TILE;

template <class K>
__device__ __forceinline__ uint32_t digit_of(K k, int shift, uint32_t mask) {
    return uint32_t(k >> shift) & mask;
}

constexpr int RS_PASSES = 8;  // digits of a 64-bit key

// The digits of a sort: `passes` of them from begin_bit on, 8 bits each (the
// last one what is left).
struct RsDigits {
    int begin, end;
    __host__ __device__ int passes() const { return (end - begin + 7) / 8; }
    __host__ __device__ int shift(int p) const { return begin + 8 * p; }
    __host__ __device__ uint32_t mask(int p) const {
        const int left = end - shift(p);
        return left >= 8 ? 0xFFu : (1u << left) - 1u;
    }
};

// Counts of every digit of every pass in one read of the keys:
// hist[pass * 256 + digit].
template <class K>
__global__ void __launch_bounds__(RS_THREADS) rs_hist_kernel(const K* __restrict__ keys, size_t n, RsDigits dg,
                                                             uint32_t* __restrict__ hist) {
    __shared__ uint32_t h[RS_PASSES][256];
    const int np = dg.passes();
    for (int p = 0; p < np; ++p) h[p][threadIdx.x] = 0;
    __syncthreads();
    for (size_t i = size_t(blockIdx.x) * RS_THREADS + threadIdx.x; i < n; i += size_t(gridDim.x) * RS_THREADS) {
        const K k = keys[i];
        for (int p = 0; p < np; ++p) atomicAdd(&h[p][digit_of(k, dg.shift(p), dg.mask(p))], 1u);
    }
    __syncthreads();
    for (int p = 0; p < np; ++p)
        if (h[p][threadIdx.x]) atomicAdd(&hist[p * 256 + threadIdx.x], h[p][threadIdx.x]);
}

// Exclusive scan over the block's 256 threads.
__device__ __forceinline__ uint32_t rs_scan256(uint32_t v, uint32_t* wsum) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    __syncthreads();  // wsum may still be read from an earlier call
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    uint32_t before = 0;
    for (int w = 0; w < warp; ++w) before += wsum[w];
    return before + x - v;
}

// Items of one tile in registers, R rounds of 32 consecutive items per warp,
// each ranked among the warp's earlier items of its digit with match_any and
// warp-private digit counters (no block barrier inside).
template <class K, class V, int R>
struct RsTile {
    K k[R];
    V v[R];
    uint32_t rk[R];
    __device__ __forceinline__ void rank(uint32_t items, int shift, uint32_t mask, uint32_t* cnt) {
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        const uint32_t lt_mask = (1u << lane) - 1u;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const uint32_t t = uint32_t(warp) * (R * 32) + r * 32 + lane;
            const bool valid = t < items;
            const uint32_t d = valid ? digit_of(k[r], shift, mask) : 256u;
            const uint32_t peers = __match_any_sync(0xFFFFFFFFu, d);
            const uint32_t before = __popc(peers & lt_mask);
            uint32_t c0 = 0;
            if (valid) c0 = cnt[d];  // the warp's earlier items of digit d
            __syncwarp();
            if (valid && before == 0) cnt[d] = c0 + __popc(peers);
            __syncwarp();
            rk[r] = c0 + before;
        }
    }
};

// Items of digit d in the tiles before tile j + 1, by one thread that no longer
// waits (lookback.cuh): those of tiles not heard from are counted.  p: tile
// j's state of the digit.
template <class K>
__device__ __noinline__ uint32_t rs_look_on(const K* __restrict__ keys, uint32_t j, int items, int shift, uint32_t mask,
                                            uint32_t d, const unsigned long long* p) {
    const LookOnce look;
    uint32_t before = 0;
    for (;; p -= 256, --j) {
        uint32_t spins = 0;
        const uint64_t v = look_wait(look, p, spins);
        if (look.flag(v)) {
            before += uint32_t(look.sum(v));
        } else {
            const K* k = keys + size_t(j) * items;
            for (int i = 0; i < items; ++i) before += digit_of(k[i], shift, mask) == d;
        }
        if (look.flag(v) == 2 || j == 0) return before;
    }
}

// One pass: tiles are taken in order from a counter; each ranks its items,
// publishes its count of every digit, reorders itself by digit in shared
// memory and, thread d for digit d, looks back over the tiles before it for
// the items of its digit that precede (one state per tile and digit, as in
// look_back).  The start of a digit comes from the counts of the whole input.
// Items of one digit leave the tile as one contiguous run, so the stores
// coalesce.  One launch and one read and write of the items per pass; with a
// histogram, a scan and a scatter launch per pass a sort of a few thousand
// items took 360 us, all of it launches (B200, 64-bit keys).
template <class K, class V, int R>
__global__ void __launch_bounds__(RS_THREADS) rs_pass_kernel(const K* __restrict__ kin, const V* __restrict__ vin,
                                                             K* __restrict__ kout, V* __restrict__ vout, size_t n,
                                                             int shift, uint32_t mask,
                                                             const uint32_t* __restrict__ hist,
                                                             unsigned long long* __restrict__ st, uint32_t tiles) {
    constexpr int TILE = RS_THREADS * R;
    extern __shared__ __align__(16) uint8_t rs_smem[];
    K* sk = reinterpret_cast<K*>(rs_smem);
    V* sv = reinterpret_cast<V*>(rs_smem + sizeof(K) * TILE);
    __shared__ uint32_t gbase[256], tstart[256];
    __shared__ uint32_t wcnt[RS_WARPS][256];
    __shared__ uint32_t wsum[RS_WARPS], s_tile;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) s_tile = uint32_t(atomicAdd(&st[size_t(tiles) * 256], 1ull));
#pragma unroll
    for (int w = 0; w < RS_WARPS; ++w) wcnt[w][tid] = 0;
    const uint32_t digit_start = rs_scan256(hist[tid], wsum);
    __syncthreads();
    const uint32_t tile = s_tile;
    const size_t base = size_t(tile) * TILE;
    const uint32_t items = uint32_t(min(size_t(TILE), n - base));
    RsTile<K, V, R> T;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const uint32_t t = uint32_t(warp) * (R * 32) + r * 32 + lane;
        T.k[r] = t < items ? kin[base + t] : K{};
        T.v[r] = (t < items && vin) ? vin[base + t] : V{};
    }
    T.rank(items, shift, mask, wcnt[warp]);
    __syncthreads();
    // per digit: this tile's count, the items of earlier warps first
    uint32_t mine = 0;
#pragma unroll
    for (int w = 0; w < RS_WARPS; ++w) {
        const uint32_t c = wcnt[w][tid];
        wcnt[w][tid] = mine;
        mine += c;
    }
    unsigned long long* state = st + size_t(tile) * 256 + tid;
    const LookOnce look;
    atomicExch(state, look.make(tile == 0 ? 2 : 1, mine));
    tstart[tid] = rs_scan256(mine, wsum);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const uint32_t t = uint32_t(warp) * (R * 32) + r * 32 + lane;
        if (t < items) {
            const uint32_t d = digit_of(T.k[r], shift, mask);
            const uint32_t lp = tstart[d] + wcnt[warp][d] + T.rk[r];
            sk[lp] = T.k[r];
            if (vin) sv[lp] = T.v[r];
        }
    }
    // items of digit tid in the tiles before this one
    uint32_t before = 0;
    if (tile > 0) {
        const unsigned long long* p = state;
        uint32_t j = tile;
        uint64_t v;
        do {  // as far as tile 0, whose sum is inclusive
            p -= 256;
            --j;
            uint32_t spins = LOOK_SPINS;
            v = look_wait(look, p, spins);
            before += uint32_t(look.sum(v));
        } while (look.flag(v) == 1);
        if (look.flag(v) == 0) before += rs_look_on(kin, j, TILE, shift, mask, uint32_t(tid), p);
        atomicExch(state, look.make(2, before + mine));
    }
    gbase[tid] = digit_start + before - tstart[tid];
    __syncthreads();
    // the tile in digit order: runs of one digit go to consecutive places
    for (uint32_t p = tid; p < items; p += RS_THREADS) {
        const K kk = sk[p];
        const uint32_t gpos = gbase[digit_of(kk, shift, mask)] + p;
        kout[gpos] = kk;
        if (vout) vout[gpos] = sv[p];
    }
}

// Every pass of a sort of at most one tile, in place, by one block.
template <class K, class V>
__global__ void __launch_bounds__(RS_THREADS) rs_single_kernel(K* __restrict__ keys, V* __restrict__ vals, uint32_t n,
                                                               RsDigits dg) {
    extern __shared__ __align__(16) uint8_t rs_smem[];
    K* sk = reinterpret_cast<K*>(rs_smem);
    V* sv = reinterpret_cast<V*>(rs_smem + sizeof(K) * RS_TILE);
    __shared__ uint32_t tstart[256];
    __shared__ uint32_t wcnt[RS_WARPS][256];
    __shared__ uint32_t wsum[RS_WARPS];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr int R = RS_ROUNDS;
    RsTile<K, V, R> T;
    const int np = dg.passes();
    for (int p = 0; p < np; ++p) {
        const int shift = dg.shift(p);
        const uint32_t mask = dg.mask(p);
#pragma unroll
        for (int w = 0; w < RS_WARPS; ++w) wcnt[w][tid] = 0;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const uint32_t t = uint32_t(warp) * (R * 32) + r * 32 + lane;
            T.k[r] = t < n ? (p ? sk[t] : keys[t]) : K{};
            T.v[r] = (t < n && vals) ? (p ? sv[t] : vals[t]) : V{};
        }
        __syncthreads();
        T.rank(n, shift, mask, wcnt[warp]);
        __syncthreads();
        uint32_t mine = 0;
#pragma unroll
        for (int w = 0; w < RS_WARPS; ++w) {
            const uint32_t c = wcnt[w][tid];
            wcnt[w][tid] = mine;
            mine += c;
        }
        tstart[tid] = rs_scan256(mine, wsum);
        __syncthreads();
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const uint32_t t = uint32_t(warp) * (R * 32) + r * 32 + lane;
            if (t < n) {
                const uint32_t d = digit_of(T.k[r], shift, mask);
                const uint32_t lp = tstart[d] + wcnt[warp][d] + T.rk[r];
                sk[lp] = T.k[r];
                if (vals) sv[lp] = T.v[r];
            }
        }
        __syncthreads();
    }
    for (uint32_t t = tid; t < n; t += RS_THREADS) {
        keys[t] = sk[t];
        if (vals) vals[t] = sv[t];
    }
}

template <class K, class V>
constexpr size_t rs_smem_bytes() {
    return (sizeof(K) + sizeof(V)) * size_t(RS_TILE);
}

// The kernels' dynamic shared-memory limit, raised once per device.
template <class K, class V>
void rs_prepare() {
    static std::mutex mu;
    static bool done[64] = {};
    int dev = 0;
    CURC_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) throw std::runtime_error("device ordinal out of range");
    std::lock_guard<std::mutex> g(mu);
    if (!done[dev]) {
        CURC_CHECK(cudaFuncSetAttribute(rs_pass_kernel<K, V, RS_ROUNDS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        int(rs_smem_bytes<K, V>())));
        CURC_CHECK(cudaFuncSetAttribute(rs_single_kernel<K, V>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        int(rs_smem_bytes<K, V>())));
        done[dev] = true;
    }
}
}  // namespace

template <class K, class V>
void radix_sort_pairs(K* keys, V* vals, size_t n, int begin_bit, int end_bit, Arena& a, cudaStream_t s) {
    if (n <= 1 || end_bit <= begin_bit) return;
    if (n > 0xFFFFFFFFull) throw std::runtime_error("radix_sort_pairs: more than 2^32 items");
    rs_prepare<K, V>();
    const RsDigits dg{begin_bit, end_bit};
    if (n <= size_t(RS_TILE)) {
        rs_single_kernel<K, V><<<1, RS_THREADS, rs_smem_bytes<K, V>(), s>>>(keys, vals, uint32_t(n), dg);
        CURC_LAUNCH_CHECK();
        return;
    }
    auto m = a.mark();
    K* kalt = a.alloc<K>(n);
    V* valt = vals ? a.alloc<V>(n) : nullptr;
    const bool few = n < RS_FEW;
    const uint32_t tile = few ? RS_THREADS * RS_ROUNDS_FEW : RS_TILE;
    const uint32_t tiles = uint32_t(div_up(n, tile));
    const int np = dg.passes();
    // per pass: 256 states per tile and the tile counter; then the counts
    const size_t pass_words = size_t(tiles) * 256 + 1;
    unsigned long long* st = a.zeros<unsigned long long>(pass_words * np + size_t(np) * 128, s);
    uint32_t* hist = reinterpret_cast<uint32_t*>(st + pass_words * np);
    rs_hist_kernel<K><<<unsigned(std::min<size_t>(div_up(n, RS_THREADS * 8), size_t(SM_COUNT_B200) * 8)), RS_THREADS, 0,
                        s>>>(keys, n, dg, hist);
    CURC_LAUNCH_CHECK();
    K* kc = keys;
    V* vc = vals;
    for (int p = 0; p < np; ++p) {
        K* ko = (kc == keys) ? kalt : keys;
        V* vo = vals ? ((vc == vals) ? valt : vals) : nullptr;
        auto pass = few ? rs_pass_kernel<K, V, RS_ROUNDS_FEW> : rs_pass_kernel<K, V, RS_ROUNDS>;
        pass<<<tiles, RS_THREADS, (sizeof(K) + sizeof(V)) * size_t(tile), s>>>(
            kc, vc, ko, vo, n, dg.shift(p), dg.mask(p), hist + p * 256, st + pass_words * p, tiles);
        CURC_LAUNCH_CHECK();
        kc = ko;
        vc = vo;
    }
    if (kc != keys) {
        CURC_CHECK(cudaMemcpyAsync(keys, kc, n * sizeof(K), cudaMemcpyDeviceToDevice, s));
        if (vals) CURC_CHECK(cudaMemcpyAsync(vals, vc, n * sizeof(V), cudaMemcpyDeviceToDevice, s));
    }
    a.release(m);
}

template void radix_sort_pairs<uint64_t, uint32_t>(uint64_t*, uint32_t*, size_t, int, int, Arena&, cudaStream_t);
template void radix_sort_pairs<uint32_t, uint32_t>(uint32_t*, uint32_t*, size_t, int, int, Arena&, cudaStream_t);
template void radix_sort_pairs<uint64_t, uint64_t>(uint64_t*, uint64_t*, size_t, int, int, Arena&, cudaStream_t);

// ---------------------------------------------------------------- misc

namespace {
__global__ void gather_words_kernel(const uint64_t* __restrict__ src, const uint32_t* __restrict__ idx, size_t n,
                                    int stride, int word, uint64_t* __restrict__ out) {
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x)
        out[i] = src[size_t(idx[i]) * stride + word];
}

template <class T>
__global__ void fill_kernel(T* p, T v, size_t n) {
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x)
        p[i] = v;
}

__global__ void iota_kernel(uint32_t* p, size_t n) {
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x)
        p[i] = uint32_t(i);
}

__global__ void unlinked_kernel(uint32_t* next, uint32_t* prev, uint16_t* offset, size_t n, uint32_t* ids0,
                                uint32_t* ids1, uint32_t* ids2) {
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x) {
        next[i] = INVALID;
        prev[i] = INVALID;
        offset[i] = INVALOFF;
        if (ids0) ids0[i] = uint32_t(i);
        if (ids1) ids1[i] = uint32_t(i);
        if (ids2) ids2[i] = uint32_t(i);
    }
}

int persistent_grid(size_t n) {
    size_t g = div_up(n, 256);
    return int(std::max<size_t>(1, std::min<size_t>(g, size_t(SM_COUNT_B200) * 16)));
}
}  // namespace

void gather_words(const uint64_t* src, const uint32_t* idx, size_t n, int stride, int word, uint64_t* out,
                  cudaStream_t s) {
    if (!n) return;
    gather_words_kernel<<<persistent_grid(n), 256, 0, s>>>(src, idx, n, stride, word, out);
    CURC_LAUNCH_CHECK();
}

template <class T>
void fill(T* p, T v, size_t n, cudaStream_t s) {
    if (!n) return;
    fill_kernel<T><<<persistent_grid(n), 256, 0, s>>>(p, v, n);
    CURC_LAUNCH_CHECK();
}
void unlinked(uint32_t* next, uint32_t* prev, uint16_t* offset, size_t n, cudaStream_t s, uint32_t* ids0,
              uint32_t* ids1, uint32_t* ids2) {
    if (n == 0) return;
    unlinked_kernel<<<persistent_grid(n), 256, 0, s>>>(next, prev, offset, n, ids0, ids1, ids2);
    CURC_LAUNCH_CHECK();
}

template void fill<uint8_t>(uint8_t*, uint8_t, size_t, cudaStream_t);
template void fill<uint16_t>(uint16_t*, uint16_t, size_t, cudaStream_t);
template void fill<uint32_t>(uint32_t*, uint32_t, size_t, cudaStream_t);
template void fill<uint64_t>(uint64_t*, uint64_t, size_t, cudaStream_t);

void iota(uint32_t* p, size_t n, cudaStream_t s) {
    if (!n) return;
    iota_kernel<<<persistent_grid(n), 256, 0, s>>>(p, n);
    CURC_LAUNCH_CHECK();
}

namespace {
// 1 where a tie element starts a new run (its predecessor in the tie list
// is not its neighbour or has another first word).
__global__ void run_starts_kernel(const uint32_t* __restrict__ pos, const uint64_t* __restrict__ k0, uint32_t m,
                                  uint32_t* __restrict__ start) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= m) return;
    start[t] = t == 0 || pos[t - 1] + 1 != pos[t] || k0[pos[t - 1]] != k0[pos[t]];
}

// inclusive count of run starts: equal for all elements of one run
__global__ void run_number_kernel(const uint32_t* __restrict__ excl, const uint32_t* __restrict__ start, uint32_t m,
                                  uint64_t* __restrict__ out) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < m) out[t] = uint64_t(excl[t]) + start[t];
}

// Runs of rows that share their first word (k0, sorted), ordered in place by
// their remaining words, ties by position (stable).  The thread at a run's
// start orders runs of up to RUN_THREAD rows by insertion; a warp orders
// runs of up to 32, each lane ranking its row against the others' words by
// shuffles (rows of up to 16 words) or loads; the rows of longer runs are
// flagged for the radix path, each by its own thread, and *any_large counts
// them.  Most runs have two or three rows (reads that start at one place), so
// a warp per run left most lanes idle; and a run may be the whole list (reads
// behind one primer), which one warp took 8 ms a million rows to flag, 32 rows
// a step (sort of 4M such reads of 64 bp 33.1 -> 1.69 ms, B200).
constexpr uint32_t RUN_THREAD = 4, RUN_WARP = 32;

// Whether row i lies in a run of more than RUN_WARP rows.  Most rows of
// such a run have RUN_WARP equal ones to one side, the others half as many.
__device__ __forceinline__ bool in_long_run(const uint64_t* __restrict__ k0, uint32_t i, uint32_t n, uint64_t v) {
    constexpr uint32_t H = RUN_WARP / 2;
    if ((i >= RUN_WARP && k0[i - RUN_WARP] == v) || (n - i > RUN_WARP && k0[i + RUN_WARP] == v)) return true;
    if (!(i >= H && k0[i - H] == v) && !(n - i > H && k0[i + H] == v)) return false;
    // equal rows before and behind, fewer than RUN_WARP of each, by bisection
    uint32_t b = 0, f = 0;
#pragma unroll
    for (uint32_t d = H; d > 0; d >>= 1) {
        if (i >= b + d && k0[i - b - d] == v) b += d;
        if (n - i > f + d && k0[i + f + d] == v) f += d;
    }
    return b + f + 1 > RUN_WARP;
}
__global__ void __launch_bounds__(256) order_runs_kernel(const uint64_t* __restrict__ db, int W,
                                                         uint32_t* __restrict__ ids,
                                                         const uint64_t* __restrict__ k0, uint32_t n,
                                                         uint8_t* __restrict__ large, uint32_t* __restrict__ any_large) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31u;
    uint32_t len = 0;  // of the run that starts here, if a thread or warp orders it
    bool flag = false;
    if (i < n) {
        const uint64_t v = k0[i];
        const bool behind = i + 1 < n && k0[i + 1] == v, before = i > 0 && k0[i - 1] == v;
        flag = (behind || before) && in_long_run(k0, i, n, v);
        large[i] = flag;
        if (!flag && behind && !before) {
            len = 2;
            while (len < RUN_WARP && i + len < n && k0[i + len] == v) ++len;
        }
    }
    const uint32_t flagged = __popc(__ballot_sync(0xFFFFFFFFu, flag));
    if (flagged && lane == 0) atomicAdd(any_large, flagged);
    if (len >= 2 && len <= RUN_THREAD) {
        uint32_t id[RUN_THREAD];
#pragma unroll
        for (uint32_t t = 0; t < RUN_THREAD; ++t) id[t] = t < len ? ids[i + t] : 0;
        auto before = [&](uint32_t x, uint32_t y) {  // row x strictly before row y
            for (int w = 1; w < W; ++w) {
                const uint64_t p = db[uint64_t(x) * W + w], q = db[uint64_t(y) * W + w];
                if (p != q) return p < q;
            }
            return false;
        };
#pragma unroll
        for (uint32_t t = 1; t < RUN_THREAD; ++t) {
            if (t < len) {
                bool go = true;
#pragma unroll
                for (uint32_t u = t; u > 0; --u) {
                    if (go && before(id[u], id[u - 1])) {
                        const uint32_t x = id[u];
                        id[u] = id[u - 1];
                        id[u - 1] = x;
                    } else {
                        go = false;
                    }
                }
            }
        }
#pragma unroll
        for (uint32_t t = 0; t < RUN_THREAD; ++t)
            if (t < len) ids[i + t] = id[t];
    }
    uint32_t todo = __ballot_sync(0xFFFFFFFFu, len > RUN_THREAD);
    while (todo) {
        const int l = __ffs(todo) - 1;
        todo &= todo - 1;
        const uint32_t p0 = __shfl_sync(0xFFFFFFFFu, i, l), m = __shfl_sync(0xFFFFFFFFu, len, l);
        const uint32_t id = lane < m ? ids[p0 + lane] : 0;
        uint32_t rank = 0;
        if (W <= 16) {
            uint64_t w[15];
#pragma unroll
            for (int k = 0; k < 15; ++k) w[k] = (lane < m && k + 1 < W) ? db[uint64_t(id) * W + k + 1] : 0;
            for (uint32_t j = 0; j < m; ++j) {
                int c = 0;  // lane j's row against mine
#pragma unroll
                for (int k = 0; k < 15; ++k) {
                    if (k + 1 < W) {
                        const uint64_t o = __shfl_sync(0xFFFFFFFFu, w[k], int(j));
                        if (c == 0 && o != w[k]) c = o < w[k] ? -1 : 1;
                    }
                }
                rank += (c < 0 || (c == 0 && j < lane)) ? 1u : 0u;
            }
        } else {
            for (uint32_t j = 0; j < m; ++j) {
                const uint32_t o = __shfl_sync(0xFFFFFFFFu, id, int(j));
                int c = 0;
                if (lane < m)
                    for (int k = 1; k < W && c == 0; ++k) {
                        const uint64_t x = db[uint64_t(o) * W + k], y = db[uint64_t(id) * W + k];
                        if (x != y) c = x < y ? -1 : 1;
                    }
                rank += (c < 0 || (c == 0 && j < lane)) ? 1u : 0u;
            }
        }
        __syncwarp();
        if (lane < m) ids[p0 + rank] = id;
        __syncwarp();
    }
}

// Up to ROWS_SMALL rows in one launch: eight lanes rank a row against all, by
// the first word (every block holds all of them in shared memory) and, where
// that is equal, by the others, ties by position.  out[rank] = id.
constexpr uint32_t ROWS_SMALL = 4096;
__global__ void __launch_bounds__(256) sort_rows_small_kernel(const uint64_t* __restrict__ db, int W,
                                                              const uint32_t* __restrict__ ids, uint32_t n,
                                                              uint32_t* __restrict__ out) {
    __shared__ uint64_t k0[ROWS_SMALL];
    for (uint32_t t = threadIdx.x; t < n; t += blockDim.x) k0[t] = db[uint64_t(ids[t]) * W];
    __syncthreads();
    const uint32_t t = blockIdx.x * 32 + (threadIdx.x >> 3), sub = threadIdx.x & 7u;
    const uint64_t mine = t < n ? k0[t] : 0;
    uint32_t rank = 0, equal = 0;
    if (t < n) {
#pragma unroll 8
        for (uint32_t j = sub; j < n; j += 8) {
            const uint64_t o = k0[j];
            rank += o < mine;
            equal += o == mine;
        }
    }
#pragma unroll
    for (int d = 1; d < 8; d <<= 1) equal += __shfl_xor_sync(0xFFFFFFFFu, equal, d);
    if (t < n && equal > 1) {
        const uint64_t* me = db + uint64_t(ids[t]) * W;
        for (uint32_t j = sub; j < n; j += 8) {
            if (k0[j] != mine || j == t) continue;
            const uint64_t* other = db + uint64_t(ids[j]) * W;
            int w = 1;
            uint64_t x = 0, y = 0;
            for (; w < W; ++w) {
                x = other[w];
                y = me[w];
                if (x != y) break;
            }
            rank += w < W ? x < y : j < t;
        }
    }
#pragma unroll
    for (int d = 1; d < 8; d <<= 1) rank += __shfl_xor_sync(0xFFFFFFFFu, rank, d);
    if (t < n && sub == 0) out[rank] = ids[t];
}

__global__ void gather_ids_kernel(const uint32_t* __restrict__ ids, const uint32_t* __restrict__ pos, uint32_t m,
                                  uint32_t* __restrict__ out) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < m) out[t] = ids[pos[t]];
}

__global__ void scatter_ids_kernel(const uint32_t* __restrict__ vals, const uint32_t* __restrict__ pos, uint32_t m,
                                   uint32_t* __restrict__ ids) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < m) ids[pos[t]] = vals[t];
}
}  // namespace

void sort_rows(const uint64_t* db, int W, int last_bits, uint32_t* ids, size_t n, Arena& a, cudaStream_t s,
               int first_bits) {
    // Stable lexicographic order of the rows (compress.cu:1400-1407 under a
    // stable comparison sort; ties keep input order).  First by the first
    // word; then only the runs of rows that share it are ordered by the
    // remaining words: runs of up to 32 rows by a thread or a warp each,
    // longer runs by radix passes over the remaining words, least significant
    // first, and finally by run so that every run returns to its place.
    if (n <= 1) return;
    auto mk = a.mark();
    if (n <= ROWS_SMALL) {
        // two launches and no read back (the general path takes a dozen and one)
        uint32_t* out = a.alloc<uint32_t>(n);
        sort_rows_small_kernel<<<grid_for(n, 32), 256, 0, s>>>(db, W, ids, uint32_t(n), out);
        CURC_LAUNCH_CHECK();
        CURC_CHECK(cudaMemcpyAsync(ids, out, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, s));
        a.release(mk);
        return;
    }
    uint64_t* k0 = a.alloc<uint64_t>(n);
    {
        // the first-word sort alone (the tie runs below read a count back to the host)
        SubStage sp("sort_dedupe.first_word");
        gather_words(db, ids, n, W, 0, k0, s);
        radix_sort_pairs<uint64_t, uint32_t>(k0, ids, n, W == 1 ? 64 - last_bits : 0, first_bits, a, s);
    }
    if (W > 1) {
        uint8_t* large = a.alloc<uint8_t>(n);
        uint32_t* cnt = a.zeros<uint32_t>(2, s);
        order_runs_kernel<<<grid_for(n, 256), 256, 0, s>>>(db, W, ids, k0, uint32_t(n), large, cnt);
        CURC_LAUNCH_CHECK();
        const uint32_t m = read_scalar(cnt, s);
        uint32_t* pos = nullptr;
        if (m) {
            pos = a.alloc<uint32_t>(m);
            select_indices(large, pos, n, cnt + 1, a, s);
        }
        if (m) {
            uint32_t* sub = a.alloc<uint32_t>(m);
            uint64_t* key = a.alloc<uint64_t>(m);
            uint64_t* run = a.alloc<uint64_t>(m);
            gather_ids_kernel<<<grid_for(m, 256), 256, 0, s>>>(ids, pos, m, sub);
            CURC_LAUNCH_CHECK();
            {
                // run number = number of run starts before the element
                uint32_t* st = a.alloc<uint32_t>(m);
                uint32_t* ex = a.alloc<uint32_t>(m);
                run_starts_kernel<<<grid_for(m, 256), 256, 0, s>>>(pos, k0, m, st);
                CURC_LAUNCH_CHECK();
                exclusive_scan<uint32_t>(st, ex, m, nullptr, a, s);
                run_number_kernel<<<grid_for(m, 256), 256, 0, s>>>(ex, st, m, run);
                CURC_LAUNCH_CHECK();
            }
            // the run numbers ride along as the sort moves the ids: sort pairs
            // of (key, index into sub) and permute both at the end
            uint32_t* perm = a.alloc<uint32_t>(m);
            iota(perm, m, s);
            uint32_t* tmp = a.alloc<uint32_t>(m);
            for (int w = W - 1; w >= 1; --w) {
                gather_ids_kernel<<<grid_for(m, 256), 256, 0, s>>>(sub, perm, m, tmp);  // current order's ids
                CURC_LAUNCH_CHECK();
                gather_words(db, tmp, m, W, w, key, s);
                const int lo = w == W - 1 ? 64 - last_bits : 0;
                radix_sort_pairs<uint64_t, uint32_t>(key, perm, m, lo, 64, a, s);
            }
            // stable by run number (ascending with position)
            uint64_t* rk = a.alloc<uint64_t>(m);
            gather_words(run, perm, m, 1, 0, rk, s);
            int bits = 1;
            while (bits < 64 && (1ull << bits) <= uint64_t(m) + 1) ++bits;
            radix_sort_pairs<uint64_t, uint32_t>(rk, perm, m, 0, bits, a, s);
            gather_ids_kernel<<<grid_for(m, 256), 256, 0, s>>>(sub, perm, m, tmp);
            CURC_LAUNCH_CHECK();
            scatter_ids_kernel<<<grid_for(m, 256), 256, 0, s>>>(tmp, pos, m, ids);
            CURC_LAUNCH_CHECK();
        }
    }
    a.release(mk);
}

void sort_ids_by_reads(const uint64_t* db, int W, int L, uint32_t* ids, size_t n, Arena& a, cudaStream_t s) {
    sort_rows(db, W, 2 * (L - 32 * (W - 1)), ids, n, a, s);
}

}  // namespace curc
