// a2-a5: duplicate links, k-mer index over prefix reads, error-free overlap
// linking over offsets 1..max_off-1, chain filter.
//
// Reference: compress.cu:1409-1420 (dedupe), 1427-1471 (index), 1473-1532
// (overlap passes, atomicCAS linking), 1539-1585 (filter and partition).
//
// Determinism.  The reference links with atomicCAS, so which suffix wins a
// contested prefix depends on scheduling.  Here the result is defined as the
// sequential loop over suffixes in list order, and computed in parallel
// exactly.  Which suffix meets which prefixes at which offset does not depend
// on the links, so the meetings of several offsets are listed at once; then
// they are walked offset by offset, one thread per run of equal prefixes
// (runs of different strings are disjoint), its suffixes in list order.
#include <algorithm>

#include "compact.cuh"
#include "stages.cuh"
#include "walk.cuh"

namespace curc {

namespace {

__global__ void dedupe_kernel(const uint64_t* __restrict__ db, int W, const uint32_t* __restrict__ sorted, uint32_t m,
                              uint32_t* __restrict__ next, uint32_t* __restrict__ prev, uint16_t* __restrict__ offset) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i + 1 >= m) return;
    const uint32_t a = sorted[i], b = sorted[i + 1];
    const uint64_t* ra = db + uint64_t(a) * W;
    const uint64_t* rb = db + uint64_t(b) * W;
    for (int w = 0; w < W; ++w)
        if (ra[w] != rb[w]) return;
    next[a] = b;
    prev[b] = a;
    offset[a] = 0;
}

__global__ void link_flags_kernel(const uint32_t* __restrict__ sorted, uint32_t m, const uint32_t* __restrict__ next,
                                  const uint32_t* __restrict__ prev, uint8_t* __restrict__ pre_f,
                                  uint8_t* __restrict__ suf_f) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    const uint32_t id = sorted[i];
    pre_f[i] = prev[id] == INVALID;
    suf_f[i] = next[id] == INVALID;
}

// The k-mer index of the prefixes of a stage.  A prefix that a suffix meets
// holds the suffix's k-mer at kmer_index_pos, and its other k-mers too; the
// further k-mers (positions qpos, lengths qlen, as far as the overlap
// reaches) only filter.
constexpr int OV_MAX_Q = 16;
struct OverlapIndex {
    const uint64_t* db;
    int W, L, k, kip;
    uint32_t mask;            // buckets - 1
    uint32_t* present;        // bitmap of the prefixes' k-mer hashes (high 32 bits)
    uint32_t bmask;
    uint32_t* extra;          // one bitmap per further k-mer
    uint32_t xmask;
    int nq;
    int16_t qpos[OV_MAX_Q], qlen[OV_MAX_Q];
    const uint32_t* va;       // prefix ids sorted by (bucket, read)
    const uint32_t* kr;       // bucket ranges
};

__device__ __forceinline__ uint32_t extra_bit(const OverlapIndex& c, const uint64_t* row, int at, int q) {
    return uint32_t(murmur64(word_at(row, uint32_t(at + c.qpos[q]), c.qlen[q]))) & c.xmask;
}

__global__ void __launch_bounds__(256) prefix_index_kernel(OverlapIndex c, const uint32_t* __restrict__ pre, uint32_t m,
                                                           uint32_t* __restrict__ keys, uint32_t* __restrict__ va) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    const uint32_t id = pre[i];
    const uint64_t* row = c.db + uint64_t(id) * c.W;
    const uint64_t hv = murmur64(word_at(row, c.kip, c.k));
    const uint32_t h = uint32_t(hv) & c.mask;
    keys[i] = h;
    va[i] = id;
    const uint32_t bit = uint32_t(hv >> 32) & c.bmask;
    atomicOr(&c.present[bit >> 5], 1u << (bit & 31));
    for (int q = 0; q < c.nq; ++q) {
        const uint32_t x = extra_bit(c, row, 0, q);
        atomicOr(&c.extra[uint64_t(q) * (uint64_t(c.xmask) + 1) / 32 + (x >> 5)], 1u << (x & 31));
    }
}

// (Keys sorted: neighbours count in the same sectors.)
__global__ void bucket_count_kernel(const uint32_t* __restrict__ keys, uint32_t m, uint32_t* __restrict__ kr) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < m) atomicAdd(&kr[keys[i]], 1u);
}

// compress.cu:1476-1501: the prefixes of the suffix's bucket that equal
// suffix[off, L) in [0, L - off): [lo, hi), false when there is none.
__device__ __forceinline__ bool overlap_run(const OverlapIndex& c, const uint64_t* sr, int off, uint32_t& lo_out,
                                            uint32_t& hi_out, uint32_t& compares) {
    const int cl = c.L - off;
    const uint32_t h = uint32_t(murmur64(word_at(sr, c.kip + off, c.k))) & c.mask;
    uint32_t lo = c.kr[h];
    const uint32_t e = c.kr[h + 1];
    uint32_t count = e - lo;
    auto cmp = [&](uint32_t it) {
        ++compares;
        return cmp_span(c.db + uint64_t(c.va[it]) * c.W, 0, sr, off, cl);
    };
    // lower bound; the entry it ends on (if below e) is the last one that
    // compared >= 0, so its comparison decides equality without a re-read
    int at_lo = 1;
    while (count > 0) {
        const uint32_t step = count / 2, it = lo + step;
        const int r = cmp(it);
        if (r < 0) {
            lo = it + 1;
            count -= step + 1;
        } else {
            count = step;
            at_lo = r;
        }
    }
    if (lo >= e || at_lo != 0) return false;
    uint32_t hi = lo + 1;
    if (hi < e && cmp(hi) == 0) {
        uint32_t n = e - ++hi;
        while (n > 0) {
            const uint32_t step = n / 2, it = hi + step;
            if (cmp(it) <= 0) {
                hi = it + 1;
                n -= step + 1;
            } else {
                n = step;
            }
        }
    }
    lo_out = lo;
    hi_out = hi;
    return true;
}

// Lists the meetings of the suffixes at offsets [off0, off0 + noffs).  One
// thread takes one suffix and 32 offsets at a time (words_each times): the 32
// k-mers are looked up in the presence bitmap with their loads in flight
// together.  Every lane's lookup is a cache line of its own, which is what
// bounds the kernel (a line a clock and SM), so the read itself lies in shared
// memory: with two loads of the read per k-mer it ran at a third of the rate
// (8M reads of 250 bp, 1.2e9 k-mers: 13.3 ms).  The k-mers
// found are tested against the further k-mers' bitmaps (a read pair with an
// error in the overlap fails there: of the 250 bp reads with rising errors
// 4 in 100 of the first lookup's finds are meetings), and what is left is
// searched in its bucket.  Room for the runs is reserved per warp; *used
// counts the room asked for, and past cap the caller repeats with fewer
// offsets.  Word w of suffix j has its meeting offsets in em[w * ms + j] and
// the first of its runs at ub[w * ms + j].  tally: [0] k-mers found, [1]
// buckets searched, [2] prefix rows compared.
__global__ void __launch_bounds__(256) meet_kernel(OverlapIndex c, const uint32_t* __restrict__ suf, uint32_t ms,
                                                   int off0, int noffs, int words_each, uint2* __restrict__ hits,
                                                   uint32_t cap, unsigned long long* __restrict__ used,
                                                   uint32_t* __restrict__ em, uint32_t* __restrict__ ub,
                                                   unsigned long long* __restrict__ tally) {
    extern __shared__ uint64_t s_rows[];
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31u;
    uint64_t* sr = s_rows + threadIdx.x * (c.W | 1);  // odd stride: few bank conflicts
    if (j < ms) {
        const uint64_t* row = c.db + uint64_t(suf[j]) * c.W;
        for (int w = 0; w < c.W; ++w) sr[w] = row[w];
    }
    uint32_t found = 0, wanted = 0, compares = 0;
    for (int w = blockIdx.y * words_each; w < int(blockIdx.y + 1) * words_each && w * 32 < noffs; ++w) {
        const int o0 = off0 + w * 32, no = min(32, noffs - w * 32);
        uint32_t maybe = 0;
        if (j < ms) {
            const BaseWindow win(sr, c.W, c.kip + o0);
#pragma unroll
            for (int b = 0; b < 32; ++b) {
                if (b < no) {
                    const uint32_t bit = uint32_t(murmur64(win.at(b, c.k)) >> 32) & c.bmask;
                    maybe |= ((c.present[bit >> 5] >> (bit & 31)) & 1u) << b;
                }
            }
            found += __popc(maybe);
            for (uint32_t rest = maybe; rest; rest &= rest - 1) {
                const int b = __ffs(rest) - 1, off = o0 + b;
                for (int q = 0; q < c.nq; ++q) {
                    if (c.qpos[q] + c.qlen[q] > c.L - off) break;
                    const uint32_t x = extra_bit(c, sr, off, q);
                    if (!((c.extra[uint64_t(q) * (uint64_t(c.xmask) + 1) / 32 + (x >> 5)] >> (x & 31)) & 1u)) {
                        maybe &= ~(1u << b);
                        break;
                    }
                }
            }
        }
        const uint32_t want = __popc(maybe);
        wanted += want;
        uint32_t incl = want;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, d);
            if (lane >= uint32_t(d)) incl += v;
        }
        unsigned long long base = 0;
        if (lane == 31 && incl) base = atomicAdd(used, static_cast<unsigned long long>(incl));
        base = __shfl_sync(0xFFFFFFFFu, base, 31) + (incl - want);
        if (j < ms) {
            uint32_t exact = 0, n = 0;
            if (base + want <= cap) {
                while (maybe) {
                    const int b = __ffs(maybe) - 1;
                    maybe &= maybe - 1;
                    uint32_t lo, hi;
                    if (overlap_run(c, sr, o0 + b, lo, hi, compares)) {
                        hits[base + n++] = make_uint2(lo, hi);
                        exact |= 1u << b;
                    }
                }
            }
            em[uint64_t(w) * ms + j] = exact;
            ub[uint64_t(w) * ms + j] = uint32_t(base);
        }
    }
    block_tally<unsigned long long>(found, &tally[0]);
    block_tally<unsigned long long>(wanted, &tally[1]);
    block_tally<unsigned long long>(compares, &tally[2]);
}

// Meetings per suffix and per offset.
__global__ void __launch_bounds__(256) meet_count_kernel(const uint32_t* __restrict__ em, uint32_t ms, int words,
                                                         uint32_t* __restrict__ per_suffix,
                                                         uint32_t* __restrict__ per_off) {
    __shared__ uint32_t h[WALK_MAX_OFFS];
    for (int o = threadIdx.x; o < words * 32; o += 256) h[o] = 0;
    __syncthreads();
    for (uint32_t j = blockIdx.x * 256 + threadIdx.x; j < ms; j += gridDim.x * 256) {
        uint32_t c = 0;
        for (int w = 0; w < words; ++w) {
            uint32_t m = em[uint64_t(w) * ms + j];
            c += __popc(m);
            for (; m; m &= m - 1) atomicAdd(&h[w * 32 + __ffs(m) - 1], 1u);
        }
        per_suffix[j] = c;
    }
    __syncthreads();
    for (int o = threadIdx.x; o < words * 32; o += 256)
        if (h[o]) atomicAdd(&per_off[o], h[o]);
}

// start[o] = meetings of the offsets before o (one block; noffs <= 512).
__global__ void __launch_bounds__(512) meet_starts_kernel(const uint32_t* __restrict__ per_off, int noffs,
                                                          uint32_t* __restrict__ start) {
    __shared__ uint32_t s[512];
    const int t = threadIdx.x;
    s[t] = t < noffs ? per_off[t] : 0;
    __syncthreads();
    for (int d = 1; d < 512; d <<= 1) {
        const uint32_t v = t >= d ? s[t - d] : 0;
        __syncthreads();
        s[t] += v;
        __syncthreads();
    }
    if (t < noffs) start[t + 1] = s[t];
    if (t == 0) start[0] = 0;
}

// Meetings in suffix order with their sort keys (offset, run).
template <class K>
__global__ void __launch_bounds__(256) meet_place_kernel(const uint32_t* __restrict__ suf, uint32_t ms, int words,
                                                         const uint32_t* __restrict__ em,
                                                         const uint32_t* __restrict__ ub,
                                                         const uint2* __restrict__ hits,
                                                         const uint32_t* __restrict__ first,
                                                         const uint32_t* __restrict__ va, int run_bits,
                                                         Meeting* __restrict__ item, K* __restrict__ key,
                                                         uint32_t* __restrict__ idx) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= ms) return;
    uint32_t at = first[j];
    const uint32_t s = suf[j];
    for (int w = 0; w < words; ++w) {
        uint32_t m = em[uint64_t(w) * ms + j];
        if (!m) continue;
        uint32_t u = ub[uint64_t(w) * ms + j];
        for (; m; m &= m - 1) {
            const uint2 h = hits[u++];
            item[at] = Meeting{s, h.x, h.y, va[h.x]};
            key[at] = K(w * 32 + __ffs(m) - 1) << run_bits | h.x;
            idx[at] = at;
            ++at;
        }
    }
}

__global__ void gather_meetings_kernel(const Meeting* __restrict__ in, const uint32_t* __restrict__ idx, uint32_t n,
                                       Meeting* __restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = in[idx[i]];
}

__global__ void chain_res_kernel(uint32_t n, const uint32_t* __restrict__ next, const uint32_t* __restrict__ prev,
                                 const uint16_t* __restrict__ offset, uint8_t* __restrict__ res) {
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    const uint32_t nx = next[r], pv = prev[r];
    uint8_t keep = 0;
    if (nx != INVALID && pv != INVALID) keep = 1;
    else if (nx != INVALID && offset[r] == 0) keep = 1;
    else if (pv != INVALID && offset[pv] == 0) keep = 1;
    res[r] = keep;
}

// A link is dropped iff one of its ends is filtered out; concurrent writers
// only ever store INVALID, so the result is schedule independent.
__global__ void chain_unlink_kernel(uint32_t n, uint32_t* next, uint32_t* prev, const uint8_t* __restrict__ res) {
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n || res[r]) return;
    const uint32_t nx = next[r];
    if (nx != INVALID) {
        prev[nx] = INVALID;
        next[r] = INVALID;
    }
    const uint32_t pv = prev[r];
    if (pv != INVALID) {
        next[pv] = INVALID;
        prev[r] = INVALID;
    }
}

__global__ void gather_flags_kernel(const uint32_t* __restrict__ ids, uint32_t m, const uint8_t* __restrict__ res,
                                    uint8_t* __restrict__ f, uint8_t* __restrict__ nf) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    const uint8_t v = res[ids[i]];
    f[i] = v;
    nf[i] = !v;
}

}  // namespace

void dedupe_links(const uint64_t* db, int W, const uint32_t* sorted, uint32_t m, uint32_t* next, uint32_t* prev,
                  uint16_t* offset, cudaStream_t s) {
    if (m < 2) return;
    dedupe_kernel<<<grid_for(m, 256), 256, 0, s>>>(db, W, sorted, m, next, prev, offset);
    CURC_LAUNCH_CHECK();
}

namespace {
// Meetings sorted by (offset, run); inside a run in list order.
template <class K>
Meeting* sorted_meetings(const uint32_t* suf, uint32_t ms, int words, const uint32_t* em, const uint32_t* ub,
                         const uint2* hits, const uint32_t* first, const uint32_t* va, int run_bits, int bits,
                         uint32_t n, Arena& a, cudaStream_t s) {
    Meeting* item = a.alloc<Meeting>(n);
    Meeting* out = a.alloc<Meeting>(n);
    K* key = a.alloc<K>(n);
    uint32_t* idx = a.alloc<uint32_t>(n);
    meet_place_kernel<K><<<grid_for(ms, 256), 256, 0, s>>>(suf, ms, words, em, ub, hits, first, va, run_bits, item, key,
                                                           idx);
    CURC_LAUNCH_CHECK();
    radix_sort_pairs<K, uint32_t>(key, idx, n, 0, bits, a, s);
    gather_meetings_kernel<<<grid_for(n, 256), 256, 0, s>>>(item, idx, n, out);
    CURC_LAUNCH_CHECK();
    return out;
}
}  // namespace

// Links the suffixes offset after offset (compress.cu:1473-1532), in stages
// of several offsets: index the free prefixes, list every meeting of the
// unlinked suffixes with them, sort the meetings and walk them.  A list of up
// to OV_ALL suffixes takes all offsets in one stage: its time was that of
// three launches per offset (39 us an offset, 3.2 ms for 2,000 reads).
// Longer lists take tune.check_every offsets first and twice as many in each
// next stage, since most suffixes link in the first offsets and what has
// linked is not listed again.
constexpr uint32_t OV_ALL = 1u << 19;
constexpr uint64_t OV_BITMAPS = 80ull << 20;  // bytes, of 126 MB of L2
void overlap_link(const BlockParams& p, const uint64_t* db, const uint32_t* sorted, uint32_t m, uint32_t* next,
                  uint32_t* prev, uint16_t* offset, Arena& a, cudaStream_t s, OverlapStats* st) {
    if (m == 0) return;
    auto mk = a.mark();
    uint8_t* pre_f = a.alloc<uint8_t>(m);
    uint8_t* suf_f = a.alloc<uint8_t>(m);
    link_flags_kernel<<<grid_for(m, 256), 256, 0, s>>>(sorted, m, next, prev, pre_f, suf_f);
    CURC_LAUNCH_CHECK();
    uint32_t* pre = a.alloc<uint32_t>(m);
    uint32_t* suf = a.alloc<uint32_t>(m);
    // what the host reads back: list lengths, the room asked for, and the
    // meetings' starts per offset
    struct State {
        uint32_t mp, ms, mp_out, ms_out;
        unsigned long long used, tally[3], walked[2];
        uint32_t start[WALK_MAX_OFFS + 1];
    };
    State* d = a.zeros<State>(1, s);
    State h{};
    select_flagged(sorted, pre_f, pre, m, &d->mp, a, s);
    select_flagged(sorted, suf_f, suf, m, &d->ms, a, s);
    read_small(&h, d, 8, s);
    uint32_t mp = h.mp, ms = h.ms;
    const uint32_t ms0 = ms;
    uint64_t active_sum = 0, met = 0;
    uint64_t listed[3] = {0, 0, 0}, voided[3] = {0, 0, 0};  // the tally so far, and of listings that were repeated
    uint32_t passes = 0;
    const int step0 = ms <= OV_ALL ? p.max_off : p.tune.check_every;
    int step = step0;
    if (mp && ms && p.max_off > 1) {
        uint32_t* pre2 = a.alloc<uint32_t>(mp);
        uint32_t* suf2 = a.alloc<uint32_t>(ms);
        Compactor cp(std::max(mp, ms), a, s);
        const uint32_t cap = uint32_t(std::min<uint64_t>(0xF0000000ull, std::max<uint64_t>(uint64_t(4) << 20, uint64_t(ms) * 2)));
        uint2* hits = a.alloc<uint2>(cap);
        OverlapIndex c = {};
        uint32_t *bits = nullptr, *keys = nullptr, *va = nullptr, *kr = nullptr;
        uint32_t indexed = 0;  // prefixes in the index (0: none yet)
        uint64_t bits_cap = 0;
        auto build_index = [&](int off) {
            SubStage sp_index("overlap.index");
            // Buckets: the table's size does not change which prefixes a
            // suffix meets (equal strings share a bucket whatever its size);
            // presence bitmaps: 16 bits per prefix for the indexed k-mer, 8
            // for each further one, fewer where all together would not stay
            // in L2.
            int hbits = 10, bbits = 16, xbits = 15;
            while (hbits < 31 && (4ull << hbits) < uint64_t(mp) * uint64_t(p.tune.table_factor)) ++hbits;
            while (bbits < 32 && (1ull << bbits) < uint64_t(mp) * uint64_t(p.tune.bitmap_bits)) ++bbits;
            while (xbits < 31 && (1ull << xbits) < uint64_t(mp) * 8) ++xbits;
            c = OverlapIndex{};
            c.db = db;
            c.W = p.W;
            c.L = p.L;
            c.k = p.k;
            c.kip = p.kip;
            c.mask = uint32_t((1ull << hbits) - 1);
            auto further = [&](int pos, int len) {
                if (len < 12 || c.nq == OV_MAX_Q || pos + len > p.L - off) return;
                c.qpos[c.nq] = int16_t(pos);
                c.qlen[c.nq++] = int16_t(len);
            };
            further(0, std::min(32, p.kip));
            for (int q = p.kip + p.k; q + 32 <= p.L - off; q += 32) further(q, 32);
            auto bitmap_bytes = [&] { return ((1ull << bbits) + (1ull << xbits) * uint64_t(c.nq)) / 8; };
            while (bitmap_bytes() > OV_BITMAPS && xbits > 20) {
                --xbits;
                if (bitmap_bytes() > OV_BITMAPS && (1ull << bbits) > uint64_t(mp) * 8) --bbits;
            }
            c.bmask = uint32_t((1ull << bbits) - 1);
            c.xmask = uint32_t((1ull << xbits) - 1);
            const uint64_t bwords = (1ull << bbits) / 32, xwords = (1ull << xbits) / 32 * uint64_t(c.nq);
            // (fewer further k-mers can leave a later index more bits)
            if (bwords + xwords > bits_cap) bits = a.alloc<uint32_t>(bits_cap = bwords + xwords);
            if (!indexed) {  // the first index has the most prefixes
                keys = a.alloc<uint32_t>(mp);
                va = a.alloc<uint32_t>(mp);
                kr = a.alloc<uint32_t>((size_t(1) << hbits) + 2);
            }
            indexed = mp;
            c.present = bits;
            c.extra = bits + bwords;
            CURC_CHECK(cudaMemsetAsync(bits, 0, (bwords + xwords) * 4, s));
            CURC_CHECK(cudaMemsetAsync(kr, 0, ((size_t(1) << hbits) + 2) * 4, s));
            prefix_index_kernel<<<grid_for(mp, 256), 256, 0, s>>>(c, pre, mp, keys, va);
            CURC_LAUNCH_CHECK();
            radix_sort_pairs<uint32_t, uint32_t>(keys, va, mp, 0, hbits, a, s);
            bucket_count_kernel<<<grid_for(mp, 256), 256, 0, s>>>(keys, mp, kr);
            CURC_LAUNCH_CHECK();
            exclusive_scan<uint32_t>(kr, kr, (size_t(1) << hbits) + 2, nullptr, a, s);
            c.va = va;
            c.kr = kr;
        };
        double asked = 0;  // the room that the last listing asked for, per suffix and offset
        for (int off = 1; off < p.max_off && mp && ms;) {
            int noffs = std::min({step, p.max_off - off, WALK_MAX_OFFS});
            if (asked * ms * noffs > 0.9 * cap) noffs = std::max(1, int(0.9 * cap / (asked * ms)));
            const int words = (noffs + 31) / 32;
            // an index of prefixes of which most are still free serves on: the
            // walk passes over the others
            if (!indexed || uint64_t(mp) * 4 < uint64_t(indexed) * 3) build_index(off);
            auto mk2 = a.mark();
            SubStage sp_meet("overlap.probe");
            uint32_t* em = a.alloc<uint32_t>(size_t(words) * ms);
            uint32_t* ub = a.alloc<uint32_t>(size_t(words) * ms);
            uint32_t* per = a.alloc<uint32_t>(ms);
            uint32_t* per_off = a.zeros<uint32_t>(WALK_MAX_OFFS, s);
            if (h.used) CURC_CHECK(cudaMemsetAsync(&d->used, 0, 8, s));
            // long lists fill the device with a thread per suffix
            const int each = ms > (1u << 18) ? words : 1;
            meet_kernel<<<dim3(unsigned(div_up(ms, 256)), unsigned(div_up(words, each))), 256,
                          size_t(256) * (p.W | 1) * 8, s>>>(c, suf, ms, off, noffs, each, hits, cap, &d->used, em, ub,
                                                            d->tally);
            CURC_LAUNCH_CHECK();
            meet_count_kernel<<<resident_grid(meet_count_kernel, 256, ms), 256, 0, s>>>(em, ms, words, per, per_off);
            CURC_LAUNCH_CHECK();
            meet_starts_kernel<<<1, 512, 0, s>>>(per_off, noffs, d->start);
            CURC_LAUNCH_CHECK();
            exclusive_scan<uint32_t>(per, per, ms, nullptr, a, s);
            read_small(&h, d, sizeof(State), s);
            sp_meet.stop();
            asked = double(h.used) / (double(ms) * noffs);
            if (h.used > cap) {  // too many for the room: fewer offsets
                a.release(mk2);
                step = std::max(1, noffs / 2);
                for (int q = 0; q < 3; ++q) voided[q] += h.tally[q] - listed[q];
                std::copy(h.tally, h.tally + 3, listed);
                continue;
            }
            std::copy(h.tally, h.tally + 3, listed);
            const uint32_t n = h.start[noffs];
            active_sum += uint64_t(ms) * noffs;
            met += n;
            passes += uint32_t(noffs);
            SubStage sp_walk("overlap.resolve");
            if (n) {
                int run_bits = 1, off_bits = 1;
                while ((1ull << run_bits) < indexed) ++run_bits;
                while ((1 << off_bits) < noffs) ++off_bits;
                const int kb = run_bits + off_bits;
                const Meeting* item =
                    kb <= 32 ? sorted_meetings<uint32_t>(suf, ms, words, em, ub, hits, per, va, run_bits, kb, n, a, s)
                             : sorted_meetings<uint64_t>(suf, ms, words, em, ub, hits, per, va, run_bits, kb, n, a, s);
                walk_stage(item, h.start, d->start, off, noffs, va, &d->used, cap, next, prev, offset, d->walked, s);
            }
            sp_walk.stop();
            off += noffs;
            if (off < p.max_off) {  // what is left for the next stage
                SubStage sp_comp("overlap.compact");
                cp.run(&d->mp, mp, &d->mp_out, FreeLink{pre, prev}, MoveId{pre, pre2});
                cp.run(&d->ms, ms, &d->ms_out, FreeLink{suf, next}, MoveId{suf, suf2});
                CURC_CHECK(cudaMemcpyAsync(&d->mp, &d->mp_out, 8, cudaMemcpyDeviceToDevice, s));
                std::swap(pre, pre2);
                std::swap(suf, suf2);
                read_small(&h, d, 8, s);
                // where few link, more offsets together waste little
                const uint64_t linked = ms - h.ms;
                step *= linked * 16 < ms ? 8 : linked * 4 < ms ? 4 : 2;
                mp = h.mp;
                ms = h.ms;
                if (ms <= OV_ALL) step = p.max_off;
                sp_comp.stop();
            }
            a.release(mk2);
        }
    }
    if (st) {
        read_small(&h, d, sizeof(State), s);
        st->passes = passes;
        st->links = h.walked[0];
        st->contested = h.walked[1];
        st->suffixes = ms0;
        st->active_sum = active_sum;
        st->probes = h.tally[0] - voided[0];
        st->hits = met;
        st->searched = h.tally[1] - voided[1];
        st->compares = h.tally[2] - voided[2];
    }
    a.release(mk);
}

void chain_filter(uint32_t n, const uint32_t* sorted, uint32_t m, uint32_t* next, uint32_t* prev,
                  const uint16_t* offset, uint32_t* ref_ids, uint32_t* unmatch_ids, uint32_t* counts, Arena& a,
                  cudaStream_t s) {
    // compress.cu:1539-1572
    auto mk = a.mark();
    uint8_t* res = a.alloc<uint8_t>(n ? n : 1);
    if (n) {
        chain_res_kernel<<<grid_for(n, 256), 256, 0, s>>>(n, next, prev, offset, res);
        CURC_LAUNCH_CHECK();
        chain_unlink_kernel<<<grid_for(n, 256), 256, 0, s>>>(n, next, prev, res);
        CURC_LAUNCH_CHECK();
    }
    uint8_t* f = a.alloc<uint8_t>(m ? m : 1);
    uint8_t* nf = a.alloc<uint8_t>(m ? m : 1);
    if (m) {
        gather_flags_kernel<<<grid_for(m, 256), 256, 0, s>>>(sorted, m, res, f, nf);
        CURC_LAUNCH_CHECK();
    }
    select_flagged(sorted, f, ref_ids, m, counts + 0, a, s);
    select_flagged(sorted, nf, unmatch_ids, m, counts + 1, a, s);
    a.release(mk);
}

}  // namespace curc
