// Device-wide primitives used by every stage: a bump arena over device
// memory, exclusive scan, stable compaction, and a stable LSD radix sort.
// All are deterministic: results never depend on thread scheduling.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <map>
#include <string>
#include <vector>

#include "common.cuh"

namespace curc {

uint64_t launches();

// Bump allocator over large device chunks.  reset() keeps the memory, so a
// pipeline that runs block after block allocates device memory only while
// it grows; when a run needed more than one chunk, reset() replaces them by
// one chunk of the largest run's size.  Alignment 256 bytes (TMA and vector
// loads need 16).
class Arena {
public:
    explicit Arena(size_t chunk = size_t(1) << 30) : chunk_(chunk) {}
    ~Arena();
    Arena(const Arena&) = delete;
    Arena& operator=(const Arena&) = delete;

    void* alloc_bytes(size_t bytes);
    template <class T>
    T* alloc(size_t n) { return static_cast<T*>(alloc_bytes(n * sizeof(T))); }
    void reset();
    // Frees every chunk (nothing may be in use: the stream work that used
    // them must have completed; cudaFree waits for the device).
    void trim();
    // Zeroed scratch of a run.  clear_zeros() clears a pool once, at the
    // start of a run; zeros() takes pieces of it, each handed out once per
    // clearing.  What does not fit there, or is asked for on another stream,
    // is allocated and cleared by itself: a small memset costs 6 us between
    // two kernels (2 us and the gaps around it), and a block of 100k pairs
    // had 119 of them in 7 ms.
    void clear_zeros(cudaStream_t s);
    void* zero_bytes(size_t bytes, cudaStream_t s);
    template <class T>
    T* zeros(size_t n, cudaStream_t s) { return static_cast<T*>(zero_bytes(n * sizeof(T), s)); }
    size_t high_water() const { return high_water_; }
    size_t in_use() const;

    // Marks let a stage release its scratch once it is done.
    struct Mark { size_t chunk, used; };
    Mark mark() const { return {cur_, cur_ < chunks_.size() ? chunks_[cur_].used : 0}; }
    void release(const Mark& m);

private:
    struct Chunk { char* base; size_t size, used; };
    std::vector<Chunk> chunks_;
    size_t cur_ = 0;
    size_t chunk_;
    size_t high_water_ = 0;
    // 16 MiB clear in 3 us and hold the tile states of every sort of a block
    // of some 100k reads; a piece of 4 MiB or more is long enough to be
    // cleared by itself
    static constexpr size_t ZERO_POOL = size_t(16) << 20, ZERO_PIECE = size_t(4) << 20;
    char* zero_ = nullptr;
    size_t zero_used_ = ZERO_POOL;  // nothing clear yet
    cudaStream_t zero_stream_ = nullptr;
};

// Growable pinned host memory, bump allocated, reset per block; results are
// copied into it asynchronously and returned as views.
class PinnedArena {
public:
    PinnedArena() = default;
    ~PinnedArena();
    PinnedArena(const PinnedArena&) = delete;
    PinnedArena& operator=(const PinnedArena&) = delete;
    // moving hands the chunks over (views into them stay valid)
    PinnedArena(PinnedArena&& o) noexcept : chunks_(std::move(o.chunks_)), cur_(o.cur_) {
        o.chunks_.clear();
        o.cur_ = 0;
    }
    PinnedArena& operator=(PinnedArena&& o) noexcept;
    uint8_t* alloc(size_t bytes);
    void reset();
    // Marks let a call give back what it took.
    struct Mark { size_t chunk, used; };
    Mark mark() const { return {cur_, cur_ < chunks_.size() ? chunks_[cur_].used : 0}; }
    void release(const Mark& m) {
        for (size_t i = m.chunk + 1; i < chunks_.size(); ++i) chunks_[i].used = 0;
        cur_ = m.chunk;
        if (cur_ < chunks_.size()) chunks_[cur_].used = m.used;
    }

private:
    struct Chunk { uint8_t* base; size_t size, used; };
    std::vector<Chunk> chunks_;
    size_t cur_ = 0;
};

// Timing events, kept from run to run.
class EventPool {
public:
    EventPool() = default;
    ~EventPool() {
        for (auto e : all_) cudaEventDestroy(e);
    }
    EventPool(const EventPool&) = delete;
    EventPool& operator=(const EventPool&) = delete;
    cudaEvent_t take() {
        if (used_ == all_.size()) {
            cudaEvent_t e = nullptr;
            CURC_CHECK(cudaEventCreate(&e));
            all_.push_back(e);
        }
        return all_[used_++];
    }
    void reset() { used_ = 0; }

private:
    std::vector<cudaEvent_t> all_;
    size_t used_ = 0;
};

// CUDA events around the stages of one block run (nested names allowed,
// e.g. "refmatch" and "refmatch.probe"); collect() adds each span's time.
// Spans that meet with no launch between them share the event: a recorded
// event takes 3.4 us between two kernels, and a block of 2,000 reads had 62.
class StageTimer {
public:
    StageTimer(cudaStream_t s, EventPool& pool) : s_(s), pool_(pool) { pool_.reset(); }
    size_t begin_span(const std::string& name);
    void end_span(size_t i) { ev_[i].b = mark(); }
    void begin(const std::string& name) { open_.push_back(begin_span(name)); }
    void end() {
        end_span(open_.back());
        open_.pop_back();
    }
    // The stream's work so far.
    cudaEvent_t mark();
    // Work without a launch (a memset) lies between: the next mark is its own.
    void part() { last_ = nullptr; }
    void collect(std::map<std::string, float>& out);

private:
    struct Span { std::string name; cudaEvent_t a, b; };
    cudaStream_t s_;
    EventPool& pool_;
    std::vector<Span> ev_;
    std::vector<size_t> open_;
    cudaEvent_t last_ = nullptr;
    uint64_t last_launches_ = 0;  // when it was recorded
};

// The timer of the block run in progress on this thread (or null).
StageTimer*& active_timer();

// Times a scope as a sub-stage of the running block, if any.
struct SubStage {
    StageTimer* t;
    size_t i = 0;
    explicit SubStage(const char* name) : t(active_timer()) {
        if (t) i = t->begin_span(name);
    }
    void stop() {
        if (t) t->end_span(i);
        t = nullptr;
    }
    ~SubStage() {
        try {
            stop();
        } catch (...) {  // leaving a scope on an error: that one is reported
        }
    }
};

// Blocks of a cluster of `kernel` on the current device: `most` (a power of
// two, at most 16), or the largest half of it that the device can hold (more
// than 8 are not portable; a partition of a device may have no group of SMs
// for 16).
unsigned cluster_blocks(const void* kernel, unsigned most, unsigned threads);

// Launches one cluster of at most `most` blocks; the kernel reads how many
// there are.
template <class... P, class... Q>
void launch_cluster(void (*kernel)(P...), unsigned most, unsigned threads, cudaStream_t s, Q... args) {
    const unsigned blocks = cluster_blocks(reinterpret_cast<const void*>(kernel), most, threads);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = blocks;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(threads);
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    CURC_CHECK(cudaLaunchKernelEx(&cfg, kernel, P(args)...));
    CURC_LAUNCH_CHECK();
}

// out[i] = sum(in[0..i)); optionally *total = sum(in[0..n)) (device pointer).
// In-place (out == in) is allowed.
template <class T>
void exclusive_scan(const T* in, T* out, size_t n, T* total, Arena& a, cudaStream_t s);

// Stable compaction: out = [in[i] for i if flags[i]], *count = number kept.
template <class T>
void select_flagged(const T* in, const uint8_t* flags, T* out, size_t n, uint32_t* count, Arena& a,
                    cudaStream_t s);

// Same, writing the indices i with flags[i] set.
void select_indices(const uint8_t* flags, uint32_t* out, size_t n, uint32_t* count, Arena& a, cudaStream_t s);

// Stable LSD radix sort of (key, value) pairs on key bits [begin_bit,
// end_bit).  keys/vals are overwritten with the sorted sequence.  vals may be
// null (keys only).
template <class K, class V>
void radix_sort_pairs(K* keys, V* vals, size_t n, int begin_bit, int end_bit, Arena& a, cudaStream_t s);

// Stable sort of ids by packed read content (W words per read, lexicographic
// over all words): ids is permuted in place.
void sort_ids_by_reads(const uint64_t* db, int W, int L, uint32_t* ids, size_t n, Arena& a, cudaStream_t s);

// The same for rows of W words of which the last one's top last_bits count;
// the first words are below 2^first_bits (fewer passes).
void sort_rows(const uint64_t* rows, int W, int last_bits, uint32_t* ids, size_t n, Arena& a, cudaStream_t s,
               int first_bits = 64);

// Gather 64-bit words: out[i] = src[idx[i] * stride + word].
void gather_words(const uint64_t* src, const uint32_t* idx, size_t n, int stride, int word, uint64_t* out,
                  cudaStream_t s);

template <class T>
void fill(T* p, T v, size_t n, cudaStream_t s);

// The links of n unlinked reads (next, prev, offset), and up to three lists
// of their numbers (null: none).
void unlinked(uint32_t* next, uint32_t* prev, uint16_t* offset, size_t n, cudaStream_t s, uint32_t* ids0 = nullptr,
              uint32_t* ids1 = nullptr, uint32_t* ids2 = nullptr);

void iota(uint32_t* p, size_t n, cudaStream_t s);

// Reads back `bytes` (at most 4 KiB) of device memory after the stream's
// work so far, and synchronises the stream.  A one-block kernel stores them
// into mapped pinned host memory (one buffer per host thread), so the read
// never waits on a copy engine: another pipeline's multi-gigabyte input copy
// on the same device cannot hold it back.
void read_small(void* host, const void* dev, size_t bytes, cudaStream_t s);

// Reads back one device value (synchronises the stream).
template <class T>
T read_scalar(const T* dev, cudaStream_t s) {
    T v;
    read_small(&v, dev, sizeof(T), s);
    return v;
}

}  // namespace curc
