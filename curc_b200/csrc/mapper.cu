// a9: map leftover reads onto the pseudogenome.
//
// Reference: ReadMapper compress.cu:268-595 with util.cuh:233-270.
// A sampled index of 28-mers every 5 positions (forward, then reverse
// complemented for the second strand), buckets capped at 12 entries; each
// read probes its 28-mers at every 2nd offset and keeps the first candidate
// that strictly improves its mismatch count, stopping at <= 1 mismatch.
//
// Canonical index.  The reference fills buckets with non-atomic uint8
// counters; here a bucket holds the first 12 sampled positions in ascending
// order, visited from the last to the first (the sequential outcome of
// compress.cu:368-406).  It is built with a stable radix sort of (hash,
// sample) pairs, in which a bucket's samples are neighbours.
#include "stages.cuh"

namespace curc {

namespace {

__global__ void sample_hash_kernel(const uint64_t* __restrict__ ref, uint64_t start, uint64_t count, int k, int step,
                                   bool rc, uint32_t mask, uint32_t* __restrict__ hv, uint32_t* __restrict__ idx) {
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < count; i += uint64_t(gridDim.x) * blockDim.x) {
        uint64_t km = word_unaligned(ref, start + i * step, k);
        if (rc) km = revcomp_kmer(km, k);
        hv[i] = uint32_t(murmur64(km) & mask);
        idx[i] = uint32_t(i);
    }
}

// One bucket: its only entry and that sample's first FP bases (count 1), or
// where its entries lie in the sorted list (count 2..12).  Eight bytes, so a
// probe of a bucket with one entry is one load, and most entries are rejected
// without a look at the pseudogenome.
constexpr int FP = 14;
struct __align__(8) MapSlot {
    uint32_t at;       // sample, or first entry
    uint32_t fp_cnt;   // FP bases << 4 | entries
};
// A sample and its first bases, beside the others of its bucket.
struct __align__(8) MapEntry {
    uint32_t idx, fp;
};

// Samples sorted by (hash, index): each bucket's first sample fills its slot;
// entries are written for buckets with more than one.
__global__ void bucket_slots_kernel(const uint64_t* __restrict__ ref, uint64_t start, int step,
                                    const uint32_t* __restrict__ hv, const uint32_t* __restrict__ idx, uint64_t count,
                                    MapSlot* __restrict__ slot, MapEntry* __restrict__ ent) {
    for (uint64_t j = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; j < count; j += uint64_t(gridDim.x) * blockDim.x) {
        const uint32_t h = hv[j], id = idx[j];
        const bool first = j == 0 || hv[j - 1] != h, more = j + 1 < count && hv[j + 1] == h;
        const uint32_t fp = uint32_t(word_unaligned(ref, start + uint64_t(id) * step, FP));
        if (first && !more) {
            slot[h] = MapSlot{id, fp << 4 | 1u};
            continue;
        }
        ent[j] = MapEntry{id, fp};
        if (first) {
            uint32_t c = 2;
            while (c < BlockParams::bucket_limit && j + c < count && hv[j + c] == h) ++c;
            slot[h] = MapSlot{uint32_t(j), c};
        }
    }
}

struct MapIndex {
    uint32_t mask;
    const MapSlot* slot;
    const MapEntry* ent;
    uint64_t start;
};

// ASCII reads packed as the other reads are, and their symbols other than
// A, C, G and T as 01 groups: those differ from every base on either strand.
__global__ void pack_ascii_rows_kernel(const uint8_t* __restrict__ ndb, uint32_t NN, int L, int W,
                                       uint64_t* __restrict__ rows, uint64_t* __restrict__ other) {
    const uint64_t t = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= uint64_t(NN) * W) return;
    const uint32_t i = uint32_t(t / W), w = uint32_t(t - uint64_t(i) * W);
    const uint8_t* p = ndb + uint64_t(i) * L;
    uint64_t v = 0, o = 0;
    for (int b = 0; b < 32; ++b) {
        const int at = int(w) * 32 + b;
        const uint8_t c = at < L ? p[at] : uint8_t('A');
        v = (v << 2) | uint64_t(ascii_code(c));
        o = (o << 2) | uint64_t(c != 'A' && c != 'C' && c != 'G' && c != 'T');
    }
    rows[t] = v;
    other[t] = o;
}

// Chunk q (bases 32q .. 32q + nb - 1) of the read as compared with the
// pseudogenome: the read's own word, or for the reverse-complement strand
// the reverse complement of the matching bases from the read's end.
template <bool RC>
__device__ __forceinline__ uint64_t read_chunk(const uint64_t* __restrict__ rd, int L, int q) {
    const int i = 32 * q, nb = L - i < 32 ? L - i : 32;
    return RC ? revcomp_kmer(word_at(rd, L - i - nb, nb), nb) : word_at(rd, i, nb);
}

// Chunk q of an ASCII read's other-symbol groups, in the same order.
template <bool RC>
__device__ __forceinline__ uint64_t other_chunk(const uint64_t* __restrict__ other, int L, int q) {
    const int i = 32 * q, nb = L - i < 32 ? L - i : 32;
    return RC ? reverse_bases(word_at(other, L - i - nb, nb)) >> (64 - 2 * nb) : word_at(other, i, nb);
}

// util.cuh:233-270: 32-base chunks, early exit once the bound is reached.
// rw: the read's chunks, computed once per read (read_chunk), and for an
// ASCII read its other symbols behind them (null else).  The window's words
// are loaded once each.
__device__ __forceinline__ int window_mismatches(const uint64_t* __restrict__ ref, uint64_t mp, const uint64_t* rw,
                                                 const uint64_t* other, int L, int bound) {
    const uint64_t* r = ref + (mp >> 5);
    const uint32_t sh = uint32_t(mp & 31u) * 2u;
    uint64_t cur = r[0];
    int c = 0;
    for (int i = 0, q = 0; i < L && c < bound; i += 32, ++q) {
        const int nb = L - i < 32 ? L - i : 32;
        const uint64_t nxt = r[q + 1];
        const uint64_t g = (sh ? (cur << sh) | (nxt >> (64u - sh)) : cur) >> (64 - 2 * nb);
        const uint64_t x = g ^ rw[q];
        uint64_t y = ((x >> 1) | x) & 0x5555555555555555ULL;
        if (other) y |= other[q];
        c += __popcll(y);
        cur = nxt;
    }
    return c;
}

// One warp per read.  The reference's loop visits the candidates of the
// read's probes in order (probe offset, then bucket slot), takes each that
// strictly improves the mismatch count, and stops at the first count
// <= target.  So its result is the first candidate with count <= target,
// or else the first candidate with the smallest count (when that improves
// on the read's count so far).  The warp lists the candidates of 32 probes
// at a time and looks at them 32 at a time in that order, one per lane.
//
// About half of a probe's candidates share its bucket only.  Such a candidate
// has a count like any other, so it is not dropped for its k-mer; but its
// first FP bases are in the index, and once they alone hold as many
// mismatches as the best count so far the candidate cannot matter.  The
// candidates whose FP bases are the read's are compared first, so that the
// best count is low when the others are looked at.  One of those may come
// before the one that set the count, and then ties with it, so the limit is
// one above that count (and above target).  A count is exact below the limit,
// which is all that is needed.
//
// A window is met through many probes of the read, and a place of the genome
// may lie in several contigs.  A window that has been compared has a count of
// at least the best one and cannot matter again: a small table of the windows
// compared (seen) keeps the warp from comparing them at every probe.
constexpr uint32_t SEEN = 64;
template <bool RC>
__device__ __forceinline__ void map_read(const MapIndex& ix, const uint64_t* __restrict__ ref, uint64_t ref_len,
                                         const uint64_t* __restrict__ rd, const uint64_t* __restrict__ other, int L,
                                         int W, int k, int step, uint8_t* __restrict__ mm,
                                         uint8_t* __restrict__ strand, uint64_t* __restrict__ pos, uint32_t i,
                                         uint32_t lane, int init, uint32_t& listed, uint32_t& compared, uint64_t* rw,
                                         uint64_t* seen) {
    // the read's words, and its comparison words, once for all its candidates
    uint64_t* row = rw + 32;
    uint64_t* ow = other ? rw + 16 : nullptr;
    const uint32_t ksh = 4u * (lane & 15u);
    if (int(lane) <= W) row[lane] = int(lane) < W ? rd[lane] : 0;
    if (int(lane) < W) {
        rw[lane] = read_chunk<RC>(rd, L, int(lane));
        if (other) ow[lane] = other_chunk<RC>(other, L, int(lane));
    }
    for (uint32_t t = lane; t < SEEN; t += 32) seen[t] = ~0ull;
    __syncwarp();
    const int probes = L < k ? 0 : (L - k) / BlockParams::read_step + 1;
    int best = init;  // smallest count met so far (the same in every lane)
    uint64_t best_pos = 0;
    bool done = false;
    for (int p0 = 0; p0 < probes && !done; p0 += 32) {
        // this lane's probe: its bucket, and the read's bases where a
        // sample's first FP lie
        const int pj = p0 + int(lane);
        MapSlot sl = {0, 0};
        uint32_t rfp = 0;
        if (pj < probes) {
            // probes lie two bases apart, so a lane's shift is the same in
            // every chunk, and its words advance by two
            const uint64_t* kw = row + 2 * (p0 >> 5) + (lane >> 4);
            const uint64_t w0 = kw[0], w1 = kw[1];
            const uint64_t key = (ksh ? (w0 << ksh) | (w1 >> (64u - ksh)) : w0) >> (64 - 2 * BlockParams::k1);
            sl = ix.slot[uint32_t(murmur64(key)) & ix.mask];
            // forward: the k-mer's first FP bases; else the reverse
            // complement of its last FP
            rfp = RC ? uint32_t(reverse_bases(~key & ((1ull << (2 * FP)) - 1)) >> (64 - 2 * FP))
                     : uint32_t(key >> (2 * (BlockParams::k1 - FP)));
        }
        uint32_t cnt = sl.fp_cnt & 15u;
        if (cnt == 1) {  // rejected here, it takes no place in the list
            const uint32_t x = (sl.fp_cnt >> 4) ^ rfp;
            if (__popc(((x >> 1) | x) & 0x55555555u) >= best) cnt = 0;
        }
        // inclusive scan of the candidate counts over the lanes
        uint32_t incl = cnt;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, d);
            if (lane >= uint32_t(d)) incl += v;
        }
        const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
        listed += uint32_t(min(32, probes - p0));
        for (uint32_t cs = 0; cs < total; cs += 32) {
            compared += min(32u, total - cs);
            const uint32_t ci = cs + lane;
            // owner lane: the first lane whose inclusive count exceeds ci
            uint32_t owner = 0;
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) {
                const uint32_t v = __shfl_sync(0xFFFFFFFFu, incl, owner + d - 1);
                if (v <= ci) owner += d;
            }
            const uint32_t oat = __shfl_sync(0xFFFFFFFFu, sl.at, owner);
            const uint32_t ofc = __shfl_sync(0xFFFFFFFFu, sl.fp_cnt, owner);
            const uint32_t oin = __shfl_sync(0xFFFFFFFFu, incl, owner);
            const uint32_t orf = __shfl_sync(0xFFFFFFFFu, rfp, owner);
            uint64_t mp = 0;
            int fm = 0x7FFF;
            if (ci < total) {
                MapEntry e = {oat, ofc >> 4};
                // the bucket's entries from the last to the first
                if ((ofc & 15u) > 1) e = ix.ent[oat + (oin - ci) - 1];
                const int oj = (p0 + int(owner)) * BlockParams::read_step;
                const uint64_t refpos = ix.start + uint64_t(e.idx) * step;
                const uint64_t shift = RC ? uint64_t(L - k - oj) : uint64_t(oj);
                mp = refpos - shift;
                const uint32_t x = e.fp ^ orf;
                if (refpos >= shift && mp + L <= ref_len && seen[mp & (SEEN - 1)] != mp)
                    fm = __popc(((x >> 1) | x) & 0x55555555u);
            }
            int c = 0x7FFF;
            int low = 0x7FFE;  // smallest count of these candidates so far
            uint32_t todo = __ballot_sync(0xFFFFFFFFu, fm < best);
            if (!todo) continue;
            const uint32_t same = __ballot_sync(0xFFFFFFFFu, fm == 0);
            uint32_t left = same;
            // mostly one window that several probes met: the lanes compare a
            // word each
            for (int t = 0; t < 3 && left; ++t) {
                const uint64_t m = __shfl_sync(0xFFFFFFFFu, mp, __ffs(left) - 1);
                uint32_t v = 0;
                if (int(lane) < W) {
                    const int nb = L - 32 * int(lane) < 32 ? L - 32 * int(lane) : 32;
                    const uint64_t x = word_unaligned(ref, m + 32 * lane, nb) ^ rw[lane];
                    uint64_t y = ((x >> 1) | x) & 0x5555555555555555ULL;
                    if (ow) y |= ow[lane];
                    v = __popcll(y);
                }
                v = __reduce_add_sync(0xFFFFFFFFu, v);
                const bool it = fm == 0 && mp == m;
                if (it) c = int(v);
                left &= ~__ballot_sync(0xFFFFFFFFu, it);
                low = min(low, int(v));
                if (lane == 0) seen[m & (SEEN - 1)] = m;
            }
            if (left) {
                if ((left >> lane) & 1u) {
                    c = window_mismatches(ref, mp, rw, ow, L, best);
                    seen[mp & (SEEN - 1)] = mp;
                }
                low = min(low, __reduce_min_sync(0xFFFFFFFFu, c));
            }
            if (todo & ~same) {
                const int limit = min(best, max(low, int(BlockParams::target_mm)) + 1);
                if (fm != 0 && fm < limit) {
                    c = window_mismatches(ref, mp, rw, ow, L, limit);
                    seen[mp & (SEEN - 1)] = mp;
                }
                low = min(low, __reduce_min_sync(0xFFFFFFFFu, c));
            }
            __syncwarp();
            if (low >= best) continue;
            // the loop stops at the first count <= target; otherwise the
            // earliest candidate with the smallest count is kept
            const uint32_t stop = __ballot_sync(0xFFFFFFFFu, c <= BlockParams::target_mm);
            const uint32_t who = stop ? stop : __ballot_sync(0xFFFFFFFFu, c == low);
            const int first = __ffs(who) - 1;
            best = __shfl_sync(0xFFFFFFFFu, c, first);
            best_pos = __shfl_sync(0xFFFFFFFFu, mp, first);
            if (stop) {
                done = true;
                break;
            }
        }
    }
    if (lane == 0 && best < init) {
        mm[i] = uint8_t(best);
        strand[i] = RC ? 1 : 0;
        pos[i] = best_pos;
    }
}

// Warps take reads in turn (a resident grid, so that no warp waits for its
// block's slowest read).  What bounds it: random sectors (2M pairs of 150 bp:
// 3.3 TB/s of DRAM traffic forward, 2.5 reverse complement), and behind them
// issue slots.  The bound of 42 registers (it takes 40, and spills 12 bytes in
// the reverse-complement form) holds 1536 threads a SM, 12 blocks of the
// default 128; that hides more of the loads than 1280 threads without it, and
// 2048 spill.
// Measured on B200, forward and reverse complement together, against a bucket
// range, a position and a window load per candidate: 8M reads of 250 bp
// 60 -> 35.8 ms, 10M pairs of 150 bp 15.5 -> 9.6 ms with the index.  Tried and
// slower: a lane walking its own probe's candidates (the warp waits for the
// fullest of 32 buckets, 55 ms), and a thread per read (4 of 32 lanes active,
// 105 ms).
template <bool RC>
__global__ void __launch_bounds__(256, 6) map_kernel(MapIndex ix, const uint64_t* __restrict__ ref, uint64_t ref_len,
                                                  const uint64_t* __restrict__ udb, uint32_t U,
                                                  const uint64_t* __restrict__ npk,
                                                  const uint64_t* __restrict__ nother, uint32_t NN, int L, int W, int k,
                                                  int step, uint8_t* __restrict__ mm, uint8_t* __restrict__ strand,
                                                  uint64_t* __restrict__ pos, unsigned long long* __restrict__ tally) {
    __shared__ uint64_t s_rw[256 / 32][52];  // per warp: the read's words, comparison words, other symbols
    __shared__ uint64_t s_seen[256 / 32][SEEN];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    uint32_t searched = 0, listed = 0, compared = 0;
    for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < U + NN; i += warps) {  // whole warp
        const int init = mm[i];
        if (init <= BlockParams::target_mm) continue;
        ++searched;
        const bool isn = i >= U;
        const uint64_t at = uint64_t(isn ? i - U : i) * W;
        map_read<RC>(ix, ref, ref_len, (isn ? npk : udb) + at, isn ? nother + at : nullptr, L, W, k, step, mm, strand,
                     pos, i, lane, init, listed, compared, s_rw[warp], s_seen[warp]);
        __syncwarp();
    }
    if (tally) {  // lane 0 carries its warp's counts
        block_tally<unsigned long long>(lane == 0 ? searched : 0u, &tally[0]);
        block_tally<unsigned long long>(lane == 0 ? listed : 0u, &tally[1]);
        block_tally<unsigned long long>(lane == 0 ? compared : 0u, &tally[2]);
    }
}

inline int log2_exact(uint32_t x) {
    int b = 0;
    while ((1u << b) < x) ++b;
    return b;
}

// Every read unmapped: one mismatch more than allowed.
__global__ void unmapped_kernel(uint8_t* __restrict__ mm, uint8_t* __restrict__ strand, uint64_t* __restrict__ pos,
                                uint32_t n, uint8_t beyond) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    mm[i] = beyond;
    strand[i] = 0;
    pos[i] = 0;
}

}  // namespace

void map_reads(const BlockParams& p, const uint64_t* ref, uint64_t ref_len, const uint64_t* udb, uint32_t U,
               const uint8_t* ndb, uint32_t NN, MapOut& out, Arena& a, cudaStream_t s) {
    const uint32_t total = U + NN;
    if (total) {
        unmapped_kernel<<<grid_for(total, 256), 256, 0, s>>>(out.mm, out.strand, out.pos, total, uint8_t(p.max_mm + 1));
        CURC_LAUNCH_CHECK();
    }
    const int k = BlockParams::k1, step = BlockParams::ref_step;
    if (total == 0 || ref_len < uint64_t(k)) return;
    const uint64_t index_count = (ref_len - k + 1 + step - 1) / step;
    struct Part { uint64_t start, count; };
    Part parts[2];
    int np = 1;
    if (index_count > (1ull << 30)) {  // compress.cu:342-353
        const uint64_t h = index_count / 2;
        parts[0] = {0, h};
        parts[1] = {h * step, index_count - h};
        np = 2;
    } else {
        parts[0] = {0, index_count};
    }
    uint64_t* npk = a.alloc<uint64_t>(size_t(NN) * p.W + 1);
    uint64_t* nother = a.alloc<uint64_t>(size_t(NN) * p.W + 1);
    if (NN) {
        pack_ascii_rows_kernel<<<grid_for(uint64_t(NN) * p.W, 256), 256, 0, s>>>(ndb, NN, p.L, p.W, npk, nother);
        CURC_LAUNCH_CHECK();
    }
    for (int rc = 0; rc < 2; ++rc) {
        for (int q = 0; q < np; ++q) {
            auto mk = a.mark();
            SubStage sp_index(rc ? "mapping.index_rc" : "mapping.index_fwd");
            const uint64_t count = parts[q].count;
            const uint32_t hs = hash_size_for(count);
            uint32_t* hv = a.alloc<uint32_t>(count);
            uint32_t* idx = a.alloc<uint32_t>(count);
            sample_hash_kernel<<<grid_for(count, 256, 4), 256, 0, s>>>(ref, parts[q].start, count, k, step, rc != 0,
                                                                       hs - 1, hv, idx);
            CURC_LAUNCH_CHECK();
            radix_sort_pairs<uint32_t, uint32_t>(hv, idx, count, 0, log2_exact(hs), a, s);
            MapSlot* slot = a.alloc<MapSlot>(hs);
            MapEntry* ent = a.alloc<MapEntry>(count);
            CURC_CHECK(cudaMemsetAsync(slot, 0, size_t(hs) * sizeof(MapSlot), s));
            bucket_slots_kernel<<<grid_for(count, 256, 4), 256, 0, s>>>(ref, parts[q].start, step, hv, idx, count, slot,
                                                                        ent);
            CURC_LAUNCH_CHECK();
            sp_index.stop();
            SubStage sp_map(rc ? "mapping.map_rc" : "mapping.map_fwd");
            MapIndex ix{hs - 1, slot, ent, parts[q].start};
            const int mt = p.tune.map_threads;
            const int g = rc ? resident_grid(map_kernel<true>, mt, uint64_t(total) * 32)
                             : resident_grid(map_kernel<false>, mt, uint64_t(total) * 32);
            unsigned long long* t = out.tally ? out.tally + 3 * rc : nullptr;
            if (rc)
                map_kernel<true><<<g, mt, 0, s>>>(ix, ref, ref_len, udb, U, npk, nother, NN, p.L, p.W, k, step, out.mm,
                                                  out.strand, out.pos, t);
            else
                map_kernel<false><<<g, mt, 0, s>>>(ix, ref, ref_len, udb, U, npk, nother, NN, p.L, p.W, k, step, out.mm,
                                                   out.strand, out.pos, t);
            CURC_LAUNCH_CHECK();
            a.release(mk);
        }
    }
}

}  // namespace curc
