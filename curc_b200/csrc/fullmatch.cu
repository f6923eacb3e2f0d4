// a6/a7: exact suffix-prefix merge of chain ends over every offset.
//
// Reference: full_match_gpu compress.cu:1003-1174 (packed reads) and
// full_match_cpu compress.cu:1176-1347 (ASCII N reads, alphabet ACGNT).
//
// Per offset the reference (1) re-sorts the suffix list by read[off, L) with
// a split on base off-1 and stable merges, (2) buckets both lists by a
// 10-base (3-symbol for ASCII) prefix with 4^10 binary searches, and (3)
// runs one sequential two-pointer merge per bucket.  Inside a bucket the
// merge pairs, in order, the suffixes and prefixes of each run of equal
// strings (with a rotation when a read meets itself), so here the work is
// organised per run of equal suffix strings instead.
//
// Which suffix meets which prefixes does not depend on the links made: only
// on the two lists.  So the meetings are listed first, for many offsets at
// once, and then only they are walked, offset by offset
// (full_match_events).  The walk needs the suffixes of a run in the
// reference's order.  Its stable merges order suffixes that share
// read[off, L) by the symbols before off, read backwards: by off-1, then
// off-2, and so on.  Since the shared part is a common prefix of the reversed
// reads, that order is at every offset the order of the whole reversed
// reads.  One sort of the suffix list by reversed reads therefore makes each
// run contiguous and ordered at every offset.
//
// Other letters.  The ASCII buckets are of A, C, G, N and T, so a string with
// another letter among its first three meets nothing; further on, other
// letters are symbols like any.  In byte order the listed form needs nothing
// more for them than that rule.
//
// The launch-per-kernel form that re-sorts at every offset
// (full_match_passes) remains as tune.fm_loop 0 for reads of those five
// letters.  There (1) is a tree of parallel stable pairwise merges of the
// per-symbol runs (merge path), whose last class would hold T and every other
// letter unsorted.
#include <algorithm>

#include "compact.cuh"
#include "stages.cuh"
#include "walk.cuh"

namespace curc {

namespace {

struct PackedAcc {
    const uint64_t* db;
    int W, L;
    static constexpr int ALPHA = 4;
    __device__ __forceinline__ int cmp(uint32_t a, int aoff, uint32_t b, int boff, int len) const {
        return cmp_span(db + uint64_t(a) * W, aoff, db + uint64_t(b) * W, boff, len);
    }
    __device__ __forceinline__ int sym(uint32_t a, int pos) const { return code_at(db + uint64_t(a) * W, pos); }
    // key: the first KS symbols of read a from pos, left-aligned, zero padded
    static constexpr int KS = 32, SB = 2;
    __device__ __forceinline__ uint64_t key(uint32_t a, int pos) const {
        const int nb = L - pos < KS ? L - pos : KS;
        return word_at(db + uint64_t(a) * W, uint32_t(pos), nb) << (64 - SB * nb);
    }
    // word k of the reversed read: 32 symbols backwards from L-1 - 32 k,
    // left-aligned, zero padded
    __device__ __forceinline__ uint64_t rword(uint32_t a, int k) const {
        const int end = L - KS * k, nb = end < KS ? end : KS;
        return reverse_bases(word_at(db + uint64_t(a) * W, uint32_t(end - nb), nb));
    }
    __device__ __forceinline__ int rwords() const { return W; }
    // whether the string from pos on can be met
    __device__ __forceinline__ bool bucketed(uint32_t, int) const { return true; }
    // hash of the FK <= FK_MAX symbols from pos
    static constexpr int FK_MAX = 32;
    __device__ __forceinline__ uint64_t fhash(uint32_t a, int pos, int fk) const {
        return murmur64(word_at(db + uint64_t(a) * W, uint32_t(pos), fk));
    }
    // the same for 32 consecutive positions
    struct Hasher {
        BaseWindow w;
        __device__ __forceinline__ Hasher(const PackedAcc& acc, uint32_t a, int pos)
            : w(acc.db + uint64_t(a) * acc.W, acc.W, pos) {}
        __device__ __forceinline__ uint64_t at(int b, int fk) const { return murmur64(w.at(b, fk)); }
    };
};

__device__ __forceinline__ bool other_letter(uint8_t c) {
    return c != 'A' && c != 'C' && c != 'G' && c != 'N' && c != 'T';
}

struct AsciiAcc {
    const uint8_t* r;
    int W, L;  // W unused
    bool other;  // the reads hold letters beyond A, C, G, N and T
    static constexpr int ALPHA = 5;
    __device__ __forceinline__ bool bucketed(uint32_t a, int pos) const {
        if (!other) return true;
        const uint8_t* x = r + uint64_t(a) * L;
        for (int i = pos; i < pos + 3 && i < L; ++i)
            if (other_letter(x[i])) return false;
        return true;
    }
    __device__ __forceinline__ int cmp(uint32_t a, int aoff, uint32_t b, int boff, int len) const {
        const uint8_t* x = r + uint64_t(a) * L + aoff;
        const uint8_t* y = r + uint64_t(b) * L + boff;
        for (int i = 0; i < len; ++i)
            if (x[i] != y[i]) return x[i] < y[i] ? -1 : 1;
        return 0;
    }
    // partition symbols of compress.cu:1238-1249: A, C, G, N, T
    __device__ __forceinline__ int sym(uint32_t a, int pos) const {
        switch (r[uint64_t(a) * L + pos]) {
            case 'A': return 0;
            case 'C': return 1;
            case 'G': return 2;
            case 'N': return 3;
            default: return 4;
        }
    }
    static constexpr int KS = 8, SB = 8;
    __device__ __forceinline__ uint64_t key(uint32_t a, int pos) const {
        const uint8_t* x = r + uint64_t(a) * L;
        uint64_t v = 0;
        for (int b = 0; b < KS; ++b) v = (v << 8) | (pos + b < L ? x[pos + b] : 0);
        return v;
    }
    __device__ __forceinline__ uint64_t rword(uint32_t a, int k) const {
        const uint8_t* x = r + uint64_t(a) * L;
        uint64_t v = 0;
        for (int b = 0; b < KS; ++b) {
            const int pos = L - 1 - KS * k - b;
            v = (v << 8) | (pos >= 0 ? x[pos] : 0);
        }
        return v;
    }
    __device__ __forceinline__ int rwords() const { return (L + KS - 1) / KS; }
    static constexpr int FK_MAX = 16;
    __device__ __forceinline__ uint64_t fhash(uint32_t a, int pos, int fk) const {
        const uint64_t k0 = key(a, pos);
        if (fk <= KS) return murmur64(k0 >> (64 - SB * fk));
        return murmur64(murmur64(k0) ^ (key(a, pos + KS) >> (64 - SB * (fk - KS))));
    }
    struct Hasher {
        const AsciiAcc& acc;
        uint32_t a;
        int pos;
        __device__ __forceinline__ Hasher(const AsciiAcc& acc_, uint32_t a_, int pos_) : acc(acc_), a(a_), pos(pos_) {}
        __device__ __forceinline__ uint64_t at(int b, int fk) const { return acc.fhash(a, pos + b, fk); }
    };
};

// Comparison of read a from aoff with read b from boff over len symbols,
// given their keys at those offsets (the key comparison decides unless the
// first KS symbols are equal and more follow).
template <class Acc>
__device__ __forceinline__ int cmp_keyed(const Acc& acc, uint64_t ka, uint32_t a, int aoff, uint64_t kb, uint32_t b,
                                         int boff, int len) {
    if (len < Acc::KS) {
        const uint64_t mask = ~0ull << (64 - Acc::SB * len);
        ka &= mask;
        kb &= mask;
    }
    if (ka != kb) return ka < kb ? -1 : 1;
    if (len <= Acc::KS) return 0;
    return acc.cmp(a, aoff + Acc::KS, b, boff + Acc::KS, len - Acc::KS);
}

// Keys of the list entries at offset off.  With sym_count (2-bit reads only),
// also how many entries have each base at off-1: the list is sorted by
// read[off-1, L), so these counts give the base runs' bounds.  Each thread
// counts in four 16-bit fields (a resident grid leaves it far fewer than 65536
// entries), then one atomic per block and base.  With tally: one thread adds
// the pass to the counters (passes with both lists non-empty, their suffix and
// prefix entries; mp_dev is the prefix list's length).
template <class Acc>
__global__ void list_keys_kernel(Acc acc, const uint32_t* __restrict__ ids, const uint32_t* __restrict__ m_dev,
                                 int off, uint64_t* __restrict__ key, uint32_t* __restrict__ sym_count,
                                 const uint32_t* __restrict__ mp_dev, unsigned long long* __restrict__ tally) {
    const uint32_t m = *m_dev;
    if (tally && blockIdx.x == 0 && threadIdx.x == 0) {
        const uint32_t mp = *mp_dev;
        if (m && mp) {
            tally[0] += 1;
            tally[1] += m;
            tally[2] += mp;
        }
    }
    uint64_t c = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
        const uint32_t id = ids[i];
        key[i] = acc.key(id, off);
        if constexpr (Acc::ALPHA == 4)
            if (sym_count) c += 1ull << (16 * acc.sym(id, off - 1));
    }
    if constexpr (Acc::ALPHA == 4)
        if (sym_count)
            for (int b = 0; b < 4; ++b) block_tally<uint32_t>(uint32_t(c >> (16 * b)) & 0xFFFFu, sym_count + b);
}

// bounds[c] = first index whose symbol at off-1 is >= c (the list is
// sorted by read[off-1, L), so symbols are nondecreasing).  One block
// narrows all boundaries at once, 64 threads each: every round samples 64
// evenly spaced positions of the boundary's interval, so a few rounds of
// independent loads replace a chain of ~log2(m) dependent ones.
template <class Acc>
__global__ void __launch_bounds__(256) run_bounds_kernel(Acc acc, const uint32_t* __restrict__ suf,
                                                         const uint32_t* __restrict__ m_dev, int off,
                                                         uint32_t* __restrict__ bounds) {
    const uint32_t m = *m_dev;
    constexpr int NB = Acc::ALPHA - 1;  // boundaries to find: symbols 1 .. ALPHA-1 (at most 4)
    constexpr uint32_t S = 64;          // samples per boundary and round
    __shared__ uint32_t lo_s[4], hi_s[4];
    __shared__ uint8_t sym_s[4][S];
    const int b = int(threadIdx.x / S);
    const uint32_t t = threadIdx.x % S;
    // invariant for boundary b: indices < lo have symbol < b+1, indices >= hi
    // have symbol >= b+1
    if (threadIdx.x < 4) {
        lo_s[threadIdx.x] = 0;
        hi_s[threadIdx.x] = m;
    }
    __syncthreads();
    for (;;) {
        bool open = false;
#pragma unroll
        for (int q = 0; q < NB; ++q) open |= lo_s[q] < hi_s[q];
        if (!open) break;
        const uint32_t lo = b < NB ? lo_s[b] : 0, hi = b < NB ? hi_s[b] : 0;
        const uint32_t span = hi - lo, k = span < S ? span : S;
        if (b < NB && t < k) sym_s[b][t] = uint8_t(acc.sym(suf[lo + uint32_t((uint64_t(span) * t) / k)], off - 1));
        __syncthreads();
        if (b < NB && t == 0 && lo < hi) {
            uint32_t f = 0;  // first sample with symbol >= b+1
            while (f < k && sym_s[b][f] < uint32_t(b + 1)) ++f;
            const uint32_t pf = f < k ? lo + uint32_t((uint64_t(span) * f) / k) : hi;
            const uint32_t pp = f > 0 ? lo + uint32_t((uint64_t(span) * (f - 1)) / k) + 1 : lo;
            lo_s[b] = k == span ? pf : pp;  // all positions sampled: exact
            hi_s[b] = pf;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        bounds[0] = 0;
#pragma unroll
        for (int q = 0; q < NB; ++q) bounds[q + 1] = lo_s[q];
        bounds[Acc::ALPHA] = m;
    }
}

// Stable merge of the symbol runs by read[off, L), as a tree of pairwise
// merges of adjacent runs (level l merges groups of 2^l runs; ties go to the
// lower run, as in the reference's stable merges), each
// output element placed by merge path: a thread takes MP_ITEMS consecutive
// outputs, finds by bisection how many of them precede in each of the two
// inputs, and then merges sequentially.  About log2(n) / MP_ITEMS + 1
// comparisons per output and level, instead of a binary search per run.
// The entries' keys at off travel with them, so a comparison reads the
// reads themselves only when the first key symbols are equal.
constexpr int MP_ITEMS = 8;

// bounds: the run bounds (ALPHA + 1 entries), or with `counts` the number of
// entries per symbol, from which the bounds are summed.
template <class Acc>
__global__ void merge_level_kernel(Acc acc, int off, const uint32_t* __restrict__ in, const uint64_t* __restrict__ ink,
                                   uint32_t* __restrict__ out, uint64_t* __restrict__ outk,
                                   const uint32_t* __restrict__ bounds, bool counts, const uint32_t* __restrict__ m_dev,
                                   int width) {
    const uint32_t m = *m_dev;
    uint32_t bd[Acc::ALPHA + 1];
    if (counts) {
        bd[0] = 0;
#pragma unroll
        for (int c = 0; c < Acc::ALPHA - 1; ++c) bd[c + 1] = bd[c] + bounds[c];
        bd[Acc::ALPHA] = m;
    } else {
#pragma unroll
        for (int c = 0; c <= Acc::ALPHA; ++c) bd[c] = bounds[c];
    }
    const int len = acc.L - off;
    auto run_at = [&](int r) { return bd[r < Acc::ALPHA ? r : Acc::ALPHA]; };
    // entry x against entry y (positions in the input)
    auto cmp_at = [&](uint32_t x, uint32_t y) {
        return cmp_keyed(acc, ink[x], in[x], off, ink[y], in[y], off, len);
    };
    const uint64_t stride = uint64_t(gridDim.x) * blockDim.x * MP_ITEMS;
    for (uint64_t d0 = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) * MP_ITEMS; d0 < m; d0 += stride) {
        const uint32_t dend = uint32_t(min(uint64_t(m), d0 + MP_ITEMS));
        uint32_t d = uint32_t(d0);
        int k = 0;
        while (d < dend) {
            // the pair of run groups that holds output d
            uint32_t a0 = run_at(2 * k * width), a1 = run_at((2 * k + 1) * width), a2 = run_at((2 * k + 2) * width);
            while (d >= a2) {
                ++k;
                a0 = run_at(2 * k * width);
                a1 = run_at((2 * k + 1) * width);
                a2 = run_at((2 * k + 2) * width);
            }
            const uint32_t na = a1 - a0, nb = a2 - a1, dd = d - a0;
            uint32_t lo = dd > nb ? dd - nb : 0, hi = dd < na ? dd : na;
            while (lo < hi) {
                const uint32_t mid = (lo + hi) / 2;
                if (cmp_at(a0 + mid, a1 + dd - mid - 1) <= 0)
                    lo = mid + 1;
                else
                    hi = mid;
            }
            uint32_t i = lo, j = dd - lo;
            const uint32_t stop = dend < a2 ? dend : a2;
            for (; d < stop; ++d) {
                const bool take_a = j >= nb || (i < na && cmp_at(a0 + i, a1 + j) <= 0);
                const uint32_t x = take_a ? a0 + i++ : a1 + j++;
                out[d] = in[x];
                outk[d] = ink[x];
            }
        }
    }
}

// One thread per run of equal suffix strings: the reference's bucket merge
// restricted to that run (compress.cu:1089-1160 / 1297-1336).  Prefix keys
// (at offset 0) and suffix keys (at off) decide most comparisons.
template <class Acc>
__device__ __forceinline__ void group_one(const Acc& acc, uint32_t* pre, uint64_t* pk, uint32_t mp,
                                          const uint32_t* __restrict__ suf, const uint64_t* __restrict__ sk,
                                          uint32_t ms, int off, uint32_t j, uint32_t* next, uint32_t* prev,
                                          uint16_t* offset) {
    const int len = acc.L - off;
    const uint32_t s0 = suf[j];
    const uint64_t k0 = sk[j];
    if (j > 0 && cmp_keyed(acc, sk[j - 1], suf[j - 1], off, k0, s0, off, len) == 0) return;
    // prefixes P with P[0, len) == s0[off, L)
    auto pcmp = [&](uint32_t i) { return cmp_keyed(acc, pk[i], pre[i], 0, k0, s0, off, len); };
    uint32_t lo = 0, count = mp;
    while (count > 0) {
        uint32_t step = count / 2, it = lo + step;
        if (pcmp(it) < 0) {
            lo = it + 1;
            count -= step + 1;
        } else {
            count = step;
        }
    }
    uint32_t hi = lo;
    while (hi < mp && pcmp(hi) == 0) ++hi;
    if (hi == lo) return;
    uint32_t se = j + 1;
    while (se < ms && cmp_keyed(acc, sk[se], suf[se], off, k0, s0, off, len) == 0) ++se;
    uint32_t pi = lo, si = j;
    while (pi < hi && si < se) {
        uint32_t P = pre[pi];
        const uint32_t S = suf[si];
        if (P == S) {
            const uint32_t cur = pi;
            bool found = false;
            while (pi + 1 < hi) {
                ++pi;
                if (pre[pi] != S) {
                    found = true;
                    break;
                }
            }
            if (!found) {
                pi = cur;
                ++si;
                continue;
            }
            // rotate P to the front of [cur, pi], keys alongside
            P = pre[pi];
            const uint64_t K = pk[pi];
            while (pi > cur) {
                pre[pi] = pre[pi - 1];
                pk[pi] = pk[pi - 1];
                --pi;
            }
            pre[pi] = P;
            pk[pi] = K;
        }
        next[S] = P;
        prev[P] = S;
        offset[S] = uint16_t(off);
        ++pi;
        ++si;
    }
}

template <class Acc>
__global__ void merge_groups_kernel(Acc acc, uint32_t* pre, uint64_t* pk, const uint32_t* __restrict__ mp_dev,
                                    const uint32_t* __restrict__ suf, const uint64_t* __restrict__ sk,
                                    const uint32_t* __restrict__ ms_dev, int off, uint32_t* next, uint32_t* prev,
                                    uint16_t* offset) {
    const uint32_t mp = *mp_dev, ms = *ms_dev;
    if (mp == 0) return;
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < ms; j += gridDim.x * blockDim.x)
        group_one(acc, pre, pk, mp, suf, sk, ms, off, j, next, prev, offset);
}

// Compaction functor: ids with their keys.
struct MoveIdKey {
    const uint32_t* in;
    const uint64_t* ink;
    uint32_t* out;
    uint64_t* outk;
    __device__ void operator()(uint32_t i, uint32_t d) const {
        out[d] = in[i];
        outk[d] = ink[i];
    }
};


// ---------------------------------------------------------------- pass form
//
// One launch per kernel and offset, queued by the host: list lengths stay on
// the device (two slots per list, read by one pass and written by its
// compaction), kernels walk the lists with resident grids, and the host looks
// at the lengths every few passes to stop early.
template <class Acc>
void full_match_passes(const Acc& acc, uint32_t* pre, uint32_t* suf, uint32_t cnt, uint32_t* next, uint32_t* prev,
                       uint16_t* offset, unsigned long long* tally, Arena& a, cudaStream_t s) {
    auto mk = a.mark();
    uint32_t* suf2 = a.alloc<uint32_t>(cnt);
    uint32_t* tmp = a.alloc<uint32_t>(cnt);
    uint32_t* mtmp = a.alloc<uint32_t>(cnt);
    // keys: prefixes at offset 0 (kept with the prefix list), suffixes at
    // the pass's offset (taken at the start of each pass)
    uint64_t* pk = a.alloc<uint64_t>(cnt);
    uint64_t* tk = a.alloc<uint64_t>(cnt);
    uint64_t* sk = a.alloc<uint64_t>(cnt);
    uint64_t* sk2 = a.alloc<uint64_t>(cnt);
    uint64_t* mk2 = a.alloc<uint64_t>(cnt);
    uint32_t* bounds = a.alloc<uint32_t>(8);
    uint32_t* len = a.alloc<uint32_t>(4);  // mp, ms for even passes, then for odd passes
    const uint32_t init[4] = {cnt, cnt, 0, 0};
    CURC_CHECK(cudaMemcpyAsync(len, init, sizeof(init), cudaMemcpyHostToDevice, s));
    Compactor cp(cnt, a, s);
    const int gk = resident_grid(list_keys_kernel<Acc>, 256, cnt);
    const int gm = resident_grid(merge_level_kernel<Acc>, 256, div_up(cnt, MP_ITEMS));
    const int gg = resident_grid(merge_groups_kernel<Acc>, 128, cnt);
    list_keys_kernel<Acc><<<gk, 256, 0, s>>>(acc, pre, len, 0, pk, nullptr, nullptr, nullptr);
    CURC_LAUNCH_CHECK();
    // 2-bit reads: the base runs' bounds come from counts taken with the keys
    constexpr bool by_count = Acc::ALPHA == 4;
    constexpr int CHECK_EVERY = 8;
    int par = 0;
    for (int off = 1; off < acc.L; ++off, par ^= 1) {
        uint32_t* mp_in = len + 2 * par;
        uint32_t* ms_in = mp_in + 1;
        uint32_t* mp_out = len + 2 * (par ^ 1);
        uint32_t* ms_out = mp_out + 1;
        if (by_count) {
            CURC_CHECK(cudaMemsetAsync(bounds, 0, 4 * sizeof(uint32_t), s));
        } else {
            run_bounds_kernel<Acc><<<1, 256, 0, s>>>(acc, suf, ms_in, off, bounds);
            CURC_LAUNCH_CHECK();
        }
        list_keys_kernel<Acc><<<gk, 256, 0, s>>>(acc, suf, ms_in, off, sk, by_count ? bounds : nullptr, mp_in, tally);
        CURC_LAUNCH_CHECK();
        {
            // levels: runs merged in pairs, then pairs of pairs, ...; the last
            // level writes suf2/sk2 (suf/sk are free after the first level)
            int levels = 0;
            while ((1 << levels) < Acc::ALPHA) ++levels;
            const uint32_t* src = suf;
            const uint64_t* srck = sk;
            for (int l = 0; l < levels; ++l) {
                const bool last = l + 1 == levels;
                uint32_t* dst = last ? suf2 : (l % 2 == 0 ? mtmp : suf);
                uint64_t* dstk = last ? sk2 : (l % 2 == 0 ? mk2 : sk);
                merge_level_kernel<Acc><<<gm, 256, 0, s>>>(acc, off, src, srck, dst, dstk, bounds, by_count, ms_in,
                                                            1 << l);
                CURC_LAUNCH_CHECK();
                src = dst;
                srck = dstk;
            }
        }
        merge_groups_kernel<Acc><<<gg, 128, 0, s>>>(acc, pre, pk, mp_in, suf2, sk2, ms_in, off, next, prev, offset);
        CURC_LAUNCH_CHECK();
        cp.run(mp_in, cnt, mp_out, FreeLink{pre, prev}, MoveIdKey{pre, pk, tmp, tk});
        cp.run(ms_in, cnt, ms_out, FreeLink{suf2, next}, MoveId{suf2, suf});
        std::swap(pre, tmp);
        std::swap(pk, tk);
        if (off % CHECK_EVERY == 0) {
            uint32_t h[2];
            read_small(h, len + 2 * (par ^ 1), 8, s);
            if (h[0] == 0 || h[1] == 0) break;
        }
    }
    a.release(mk);
}

// ---------------------------------------------------------------- event form

template <class Acc>
__global__ void fm_prefix_kernel(Acc acc, const uint32_t* __restrict__ pre, uint32_t m, uint64_t* __restrict__ pk,
                                 int fk, uint32_t* __restrict__ bits, uint32_t bmask) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    const uint32_t id = pre[i];
    pk[i] = acc.key(id, 0);
    const uint32_t h = uint32_t(acc.fhash(id, 0, fk)) & bmask;
    atomicOr(&bits[h >> 5], 1u << (h & 31));
}

// The prefixes of the list that start with s[off, L): [lo, hi), by binary
// search; false when there is none.
template <class Acc>
__device__ __forceinline__ bool fm_run(const Acc& acc, const uint32_t* pre, const uint64_t* pk, uint32_t mp,
                                       uint32_t s, int off, uint32_t& lo_out, uint32_t& hi_out) {
    if (!acc.bucketed(s, off)) return false;
    const int len = acc.L - off;
    const uint64_t k = acc.key(s, off);
    auto pcmp = [&](uint32_t i) { return cmp_keyed(acc, pk[i], pre[i], 0, k, s, off, len); };
    uint32_t lo = 0, count = mp;
    int at_lo = 1;  // the comparison of the entry the search ends on
    while (count > 0) {
        const uint32_t step = count / 2, it = lo + step;
        const int r = pcmp(it);
        if (r < 0) {
            lo = it + 1;
            count -= step + 1;
        } else {
            count = step;
            at_lo = r;
        }
    }
    if (lo >= mp || at_lo != 0) return false;
    uint32_t hi = lo + 1;
    if (hi < mp && pcmp(hi) == 0) {
        uint32_t c = mp - hi;
        while (c > 0) {
            const uint32_t step = c / 2, it = hi + step;
            if (pcmp(it) <= 0) {
                hi = it + 1;
                c -= step + 1;
            } else {
                c = step;
            }
        }
    }
    lo_out = lo;
    hi_out = hi;
    return true;
}

// Lists the meetings of the suffixes at offsets [off0, off0 + noffs): one
// thread takes one suffix and 32 offsets (blockIdx.y), tests the 32 strings
// in the prefixes' presence bitmap (loads in flight together), reserves room
// for those that pass and searches the prefix list for each.  hits holds the
// runs found, in no order; word w of suffix j has its meeting offsets in
// em[w * ms + j] and the first of its runs at ub[w * ms + j].  *used counts
// the room asked for; when it passes cap the caller repeats with fewer
// offsets.
template <class Acc>
__global__ void __launch_bounds__(256) fm_meet_kernel(Acc acc, const uint32_t* __restrict__ suf, uint32_t ms,
                                                      const uint32_t* __restrict__ pre,
                                                      const uint64_t* __restrict__ pk, uint32_t mp,
                                                      const uint32_t* __restrict__ bits, uint32_t bmask, int fk,
                                                      int off0, int noffs, uint2* __restrict__ hits, uint32_t cap,
                                                      unsigned long long* __restrict__ used,
                                                      uint32_t* __restrict__ em, uint32_t* __restrict__ ub) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    const int w = blockIdx.y;
    const uint32_t s = j < ms ? suf[j] : 0;
    uint32_t maybe = 0;
    if (j < ms) {
        const typename Acc::Hasher hash(acc, s, off0 + w * 32);
#pragma unroll
        for (int b = 0; b < 32; ++b) {
            if (w * 32 + b < noffs) {
                const uint32_t h = uint32_t(hash.at(b, fk)) & bmask;
                maybe |= ((bits[h >> 5] >> (h & 31)) & 1u) << b;
            }
        }
    }
    const uint32_t lane = threadIdx.x & 31u, want = __popc(maybe);
    uint32_t incl = want;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, d);
        if (lane >= uint32_t(d)) incl += v;
    }
    unsigned long long base = 0;
    if (lane == 31 && incl) base = atomicAdd(used, static_cast<unsigned long long>(incl));
    base = __shfl_sync(0xFFFFFFFFu, base, 31) + (incl - want);
    if (j >= ms) return;
    uint32_t exact = 0, n = 0;
    if (base + want <= cap) {
        while (maybe) {
            const int b = __ffs(maybe) - 1;
            maybe &= maybe - 1;
            uint32_t lo, hi;
            if (fm_run(acc, pre, pk, mp, s, off0 + w * 32 + b, lo, hi)) {
                hits[base + n++] = make_uint2(lo, hi);
                exact |= 1u << b;
            }
        }
    }
    em[uint64_t(w) * ms + j] = exact;
    ub[uint64_t(w) * ms + j] = uint32_t(base);
}

// Meetings per offset and warp of 32 suffixes: count[o * nw + warp].
__global__ void __launch_bounds__(256) fm_count_kernel(const uint32_t* __restrict__ em, uint32_t ms, uint32_t nw,
                                                       uint32_t* __restrict__ count) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x, warp = j >> 5, lane = threadIdx.x & 31u;
    const uint32_t m = j < ms ? em[uint64_t(blockIdx.y) * ms + j] : 0;
    uint32_t mine = 0;
#pragma unroll
    for (int b = 0; b < 32; ++b) {
        const uint32_t bal = __ballot_sync(0xFFFFFFFFu, (m >> b) & 1u);
        if (lane == uint32_t(b)) mine = __popc(bal);
    }
    if (warp < nw) count[(uint64_t(blockIdx.y) * 32 + lane) * nw + warp] = mine;
}

// Meetings in order of (offset, suffix): first = the exclusive scan of the
// counts.
__global__ void __launch_bounds__(256) fm_place_kernel(const uint32_t* __restrict__ suf, uint32_t ms, uint32_t nw,
                                                       const uint32_t* __restrict__ pre,
                                                       const uint2* __restrict__ hits,
                                                       const uint32_t* __restrict__ em,
                                                       const uint32_t* __restrict__ ub,
                                                       const uint32_t* __restrict__ first, Meeting* __restrict__ item) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x, warp = j >> 5, lane = threadIdx.x & 31u;
    const bool on = j < ms;
    const uint32_t m = on ? em[uint64_t(blockIdx.y) * ms + j] : 0;
    const uint32_t s = on ? suf[j] : 0;
    uint32_t u = on ? ub[uint64_t(blockIdx.y) * ms + j] : 0;
    if (!__any_sync(0xFFFFFFFFu, m != 0)) return;
    const uint32_t at = first[(uint64_t(blockIdx.y) * 32 + lane) * nw + warp];  // of offset `lane` of this word
    const uint32_t lt = (1u << lane) - 1u;
    for (int b = 0; b < 32; ++b) {
        const uint32_t bal = __ballot_sync(0xFFFFFFFFu, (m >> b) & 1u);
        const uint32_t base = __shfl_sync(0xFFFFFFFFu, at, b);
        if ((m >> b) & 1u) {
            const uint2 h = hits[u++];
            item[base + __popc(bal & lt)] = Meeting{s, h.x, h.y, pre[h.x]};
        }
    }
}

// First meeting of each offset, and the end of the last.
__global__ void fm_starts_kernel(const uint32_t* __restrict__ first, uint32_t nw, const uint32_t* __restrict__ total,
                                 int noffs, uint32_t* __restrict__ start) {
    for (int o = threadIdx.x; o <= noffs; o += blockDim.x)
        start[o] = o < noffs ? first[uint64_t(o) * nw] : *total;
}

// Every offset from off0 on of two short lists, by one block: keys, runs and
// link states in shared memory, two barriers per offset.  suf in the order
// of the reversed reads when `ordered`, else it is ordered here (each thread
// ranks its suffix against all).  Most suffixes meet nothing at an offset: a
// bitmap of the prefixes' first symbols (128 bits a prefix, so that most warps
// find no lane to search for) spares them the bisection, which was most of an
// offset's 2,500 cycles.  Full match of 2,000 reads 0.16 -> 0.13 ms; unmapped
// reads of 100k reads 0.74 -> 0.63 ms, of 100k pairs 0.67 -> 0.57.
constexpr uint32_t FM_SMALL = 1024, FM_BITS = 17;
template <class Acc>
__device__ __forceinline__ uint32_t fm_small_bit(uint64_t key) {
    constexpr int FS = Acc::KS < 12 ? Acc::KS : 12;  // symbols hashed
    return uint32_t(((key >> (64 - Acc::SB * FS)) * 0x9E3779B97F4A7C15ull) >> (64 - FM_BITS));
}
template <class Acc>
__global__ void __launch_bounds__(FM_SMALL) fm_small_kernel(Acc acc, const uint32_t* __restrict__ pre_in,
                                                            const uint32_t* __restrict__ suf_in, uint32_t n, int off0,
                                                            bool ordered, uint32_t* next, uint32_t* prev,
                                                            uint16_t* offset, unsigned long long* __restrict__ tally) {
    __shared__ uint64_t pk[FM_SMALL], rk[FM_SMALL];
    __shared__ uint32_t pre[FM_SMALL], suf[FM_SMALL], run[FM_SMALL];
    __shared__ uint8_t sdone[FM_SMALL], pdone[FM_SMALL];
    __shared__ uint32_t bits[(1u << FM_BITS) / 32];
    __shared__ uint32_t s_left;
    constexpr int FS = Acc::KS < 12 ? Acc::KS : 12;
    const uint32_t t = threadIdx.x;
    if (t == 0) s_left = n;
    for (uint32_t w = t; w < (1u << FM_BITS) / 32; w += blockDim.x) bits[w] = 0;
    uint32_t me = 0;
    if (t < n) {
        pre[t] = pre_in[t];
        pk[t] = acc.key(pre[t], 0);
        me = suf_in[t];
        suf[t] = me;
        rk[t] = acc.rword(me, 0);
        sdone[t] = pdone[t] = 0;
    }
    __syncthreads();
    if (t < n) {
        const uint32_t h = fm_small_bit<Acc>(pk[t]);
        atomicOr(&bits[h >> 5], 1u << (h & 31));
    }
    __syncthreads();
    if (!ordered) {
        uint32_t rank = 0;
        if (t < n) {
            const uint64_t mine = rk[t];
            uint32_t equal = 0;
#pragma unroll 8
            for (uint32_t j = 0; j < n; ++j) {
                const uint64_t o = rk[j];
                rank += o < mine;
                equal += o == mine;
            }
            if (equal > 1) {
                const int nw = acc.rwords();
                for (uint32_t j = 0; j < n; ++j) {
                    if (rk[j] != mine || j == t) continue;
                    int k = 1;
                    uint64_t x = 0, y = 0;
                    for (; k < nw; ++k) {
                        x = acc.rword(suf[j], k);
                        y = acc.rword(me, k);
                        if (x != y) break;
                    }
                    rank += k < nw ? x < y : j < t;
                }
            }
        }
        __syncthreads();
        if (t < n) suf[rank] = me;
        __syncthreads();
        if (t < n) me = suf[t];
    }
    int passes = 0;
    uint32_t met = 0;
    for (int off = off0; off < acc.L; ++off) {
        ++passes;
        uint32_t lo = INVALID;
        if (t < n) {
            // (the upper end of the run is found as it is walked)
            const int len = acc.L - off;
            const uint64_t k = acc.key(me, off);
            const uint32_t h = fm_small_bit<Acc>(k);
            const bool maybe = (len < FS || (bits[h >> 5] >> (h & 31) & 1u)) && acc.bucketed(me, off);
            uint32_t b = 0, c = maybe ? n : 0;
            int at = 1;
            while (c > 0) {
                const uint32_t step = c / 2, it = b + step;
                const int r = cmp_keyed(acc, pk[it], pre[it], 0, k, me, off, len);
                if (r < 0) {
                    b = it + 1;
                    c -= step + 1;
                } else {
                    c = step;
                    at = r;
                }
            }
            if (b < n && at == 0) lo = b;
            run[t] = lo;
        }
        const int here = __syncthreads_count(lo != INVALID && !sdone[t]);
        if (here == 0) continue;
        met += uint32_t(here);
        if (t < n && lo != INVALID && (t == 0 || run[t - 1] != lo)) {
            const int len = acc.L - off;
            const uint64_t k = acc.key(me, off);
            uint32_t q0 = lo;
            bool left = true;
            for (uint32_t i = t; left && i < n && run[i] == lo; ++i) {
                if (sdone[i]) continue;
                const uint32_t S = suf[i];
                left = false;
                for (uint32_t q = q0; q < n; ++q) {
                    if (q > lo && cmp_keyed(acc, pk[q], pre[q], 0, k, me, off, len) != 0) break;
                    if (pdone[q]) {
                        if (!left) q0 = q + 1;
                        continue;
                    }
                    left = true;
                    const uint32_t P = pre[q];
                    if (P == S) continue;
                    next[S] = P;
                    prev[P] = S;
                    offset[S] = uint16_t(off);
                    sdone[i] = pdone[q] = 1;
                    atomicSub(&s_left, 1u);
                    break;
                }
            }
        }
        __syncthreads();
        if (s_left == 0) break;
    }
    if (tally && t == 0) {
        tally[0] += uint32_t(passes);
        tally[1] += met;
        tally[2] += met;
    }
}

// Reversed reads of a list as rows for the read sort, with their positions.
template <class Acc>
__global__ void fm_reversed_kernel(Acc acc, const uint32_t* __restrict__ suf, uint32_t m, int W,
                                   uint64_t* __restrict__ rows, uint32_t* __restrict__ idx) {
    const uint64_t t = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= uint64_t(m) * W) return;
    const uint32_t i = uint32_t(t / W), w = uint32_t(t - uint64_t(i) * W);
    rows[t] = acc.rword(suf[i], int(w));
    if (w == 0) idx[i] = i;
}
__global__ void fm_permute_kernel(const uint32_t* __restrict__ suf, const uint32_t* __restrict__ idx, uint32_t m,
                                  uint32_t* __restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < m) out[i] = suf[idx[i]];
}

// out = suf in the order of the reversed reads (ties in list order).
template <class Acc>
void fm_reverse_order(const Acc& acc, const uint32_t* suf, uint32_t m, uint32_t* out, Arena& a, cudaStream_t s) {
    auto mk = a.mark();
    const int W = int(div_up(uint64_t(acc.L), Acc::KS));
    uint64_t* rows = a.alloc<uint64_t>(size_t(m) * W);
    uint32_t* idx = a.alloc<uint32_t>(m);
    fm_reversed_kernel<Acc><<<grid_for(uint64_t(m) * W, 256), 256, 0, s>>>(acc, suf, m, W, rows, idx);
    CURC_LAUNCH_CHECK();
    sort_rows(rows, W, Acc::SB * (acc.L - Acc::KS * (W - 1)), idx, m, a, s);
    fm_permute_kernel<<<grid_for(m, 256), 256, 0, s>>>(suf, idx, m, out);
    CURC_LAUNCH_CHECK();
    a.release(mk);
}

// The lowest string length of the next stage, whose highest is hi: long
// strings (16 and more) are met rarely and are all listed at once; below, a
// random list of m entries meets almost every string of ceil(log4 m) symbols,
// so a stage stops where its runs would hold 32 entries on average and the
// lists are compacted before the next one.
int fm_stage_low(int hi, uint32_t m) {
    int base = 1;
    while (base < 16 && (uint64_t(32) << (2 * base)) < m) ++base;
    return std::min(hi, hi > 16 ? std::max(16, base) : base);
}

// What bounds the match is the serial chain of offsets, not bytes: as a
// conditional graph of ten small launches an offset cost 33 us whatever the
// lists held.  Listed at once, the offsets share a handful of launches, and
// the walk costs a barrier and two dependent loads per offset that has a
// meeting.  Measured on B200, the full match of the pseudogenome: 2,000 reads
// of 100 bp (113 ends) 3.3 -> 0.19 ms, 8M reads of 250 bp (371,000 ends)
// 18.5 -> 3.7 ms, 10M pairs of 150 bp (436,000 ends) 10.5 -> 3.5 ms.  Lists
// of up to FM_SMALL ends take the one-block form: below that the launches of
// a stage (12, and a read back) cost more than the block's two barriers per
// offset.
template <class Acc>
void full_match_events(const Acc& acc, uint32_t* pre, uint32_t* suf, uint32_t cnt, uint32_t* next, uint32_t* prev,
                       uint16_t* offset, unsigned long long* tally, Arena& a, cudaStream_t s) {
    auto small = [&](const uint32_t* pl, const uint32_t* sl, uint32_t n, int off, bool ordered) {
        const uint32_t threads = std::max(64u, uint32_t(div_up(n, 32)) * 32);
        fm_small_kernel<Acc><<<1, threads, 0, s>>>(acc, pl, sl, n, off, ordered, next, prev, offset, tally);
        CURC_LAUNCH_CHECK();
    };
    if (cnt <= FM_SMALL) {
        small(pre, suf, cnt, 1, false);
        return;
    }
    auto mk = a.mark();
    uint32_t* suf_o = a.alloc<uint32_t>(cnt);
    fm_reverse_order(acc, suf, cnt, suf_o, a, s);
    uint32_t* pl = pre;
    uint32_t* sl = suf_o;
    uint32_t* pl2 = a.alloc<uint32_t>(cnt);
    uint32_t* sl2 = suf;
    uint64_t* pk = a.alloc<uint64_t>(cnt);
    // room for the runs of one stage's meetings, and false ones
    const uint32_t cap = uint32_t(std::min<uint64_t>(0xF0000000ull, std::max<uint64_t>(uint64_t(4) << 20, uint64_t(cnt) * 6)));
    uint2* hits = a.alloc<uint2>(cap);
    Meeting* item = a.alloc<Meeting>(cap);
    struct State {
        unsigned long long used;
        uint32_t total, len_in, len_out[2];
    };
    State* st = a.alloc<State>(1);
    uint32_t* start = a.alloc<uint32_t>(WALK_MAX_OFFS + 1);
    Compactor cp(cnt, a, s);
    uint32_t m = cnt;
    int hi = acc.L - 1;
    int fewer = acc.L;  // at most this many offsets per stage (lowered when a listing ran out of room)
    while (hi >= 1 && m > FM_SMALL) {
        auto mk2 = a.mark();
        const int low = std::max(fm_stage_low(hi, m), hi - std::min(fewer, WALK_MAX_OFFS) + 1);
        const int noffs = hi - low + 1, off0 = acc.L - hi, words = (noffs + 31) / 32;
        const int fk = std::min(low, int(Acc::FK_MAX));
        // presence bitmap of the prefixes' first fk symbols: 32 bits per
        // prefix, so that 3% of the strings that meet none pass
        int bbits = 15;
        while (bbits < 32 && (1ull << bbits) < uint64_t(m) * 32) ++bbits;
        uint32_t* bits = a.zeros<uint32_t>((1ull << bbits) / 32, s);
        const uint32_t bmask = uint32_t((1ull << bbits) - 1);
        const uint32_t nw = uint32_t(div_up(m, 32));
        uint32_t* em = a.alloc<uint32_t>(size_t(words) * m);
        uint32_t* ub = a.alloc<uint32_t>(size_t(words) * m);
        uint32_t* count = a.alloc<uint32_t>(size_t(words) * 32 * nw);
        const State init{0, 0, m, {0, 0}};
        CURC_CHECK(cudaMemcpyAsync(st, &init, sizeof(init), cudaMemcpyHostToDevice, s));
        fm_prefix_kernel<Acc><<<grid_for(m, 256), 256, 0, s>>>(acc, pl, m, pk, fk, bits, bmask);
        CURC_LAUNCH_CHECK();
        const dim3 grid(unsigned(div_up(m, 256)), unsigned(words));
        fm_meet_kernel<Acc><<<grid, 256, 0, s>>>(acc, sl, m, pl, pk, m, bits, bmask, fk, off0, noffs, hits, cap,
                                                  &st->used, em, ub);
        CURC_LAUNCH_CHECK();
        fm_count_kernel<<<grid, 256, 0, s>>>(em, m, nw, count);
        CURC_LAUNCH_CHECK();
        exclusive_scan<uint32_t>(count, count, size_t(words) * 32 * nw, &st->total, a, s);
        fm_place_kernel<<<grid, 256, 0, s>>>(sl, m, nw, pl, hits, em, ub, count, item);
        CURC_LAUNCH_CHECK();
        fm_starts_kernel<<<1, 256, 0, s>>>(count, nw, &st->total, noffs, start);
        CURC_LAUNCH_CHECK();
        walk_meetings(item, start, off0, noffs, pl, &st->used, cap, m, next, prev, offset, tally, s);
        cp.run(&st->len_in, m, &st->len_out[0], FreeLink{pl, prev}, MoveId{pl, pl2});
        cp.run(&st->len_in, m, &st->len_out[1], FreeLink{sl, next}, MoveId{sl, sl2});
        State h;
        read_small(&h, st, sizeof(h), s);
        a.release(mk2);
        if (h.used > cap) {
            fewer = std::max(1, noffs / 2);
            continue;  // nothing was linked; the lists are as they were
        }
        std::swap(pl, pl2);
        std::swap(sl, sl2);
        m = h.len_out[0];
        hi = low - 1;
    }
    if (hi >= 1 && m > 0) small(pl, sl, m, acc.L - hi, true);
    a.release(mk);
}

// nothing to link without ends
template <class Acc>
void full_match_loop(const Acc& acc, uint32_t* pre, uint32_t* suf, uint32_t cnt, uint32_t* next, uint32_t* prev,
                     uint16_t* offset, bool passes, unsigned long long* tally, Arena& a, cudaStream_t s) {
    if (cnt == 0 || acc.L < 2) return;
    if (passes)
        full_match_passes(acc, pre, suf, cnt, next, prev, offset, tally, a, s);
    else
        full_match_events(acc, pre, suf, cnt, next, prev, offset, tally, a, s);
}

// *other = 1 when a listed read holds a byte other than A, C, G, N and T.
__global__ void other_symbols_kernel(const uint8_t* __restrict__ r, int L, const uint32_t* __restrict__ ids,
                                     uint32_t m, uint32_t* __restrict__ other) {
    for (uint64_t t = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; t < uint64_t(m) * L;
         t += uint64_t(gridDim.x) * blockDim.x) {
        const uint32_t i = uint32_t(t / L), b = uint32_t(t - uint64_t(i) * L);
        if (other_letter(r[uint64_t(ids[i]) * L + b])) *other = 1;
    }
}

// ASCII reads as rows of big-endian words, zero padded (word order is
// memcmp order).
__global__ void ascii_rows_kernel(const uint8_t* __restrict__ r, int L, const uint32_t* __restrict__ ids, uint32_t m,
                                  int W, uint64_t* __restrict__ rows, uint32_t* __restrict__ idx) {
    const uint64_t t = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= uint64_t(m) * W) return;
    const uint32_t i = uint32_t(t / W), w = uint32_t(t - uint64_t(i) * W);
    const uint8_t* p = r + uint64_t(ids[i]) * L + w * 8;
    uint64_t v = 0;
    for (int b = 0; b < 8; ++b) v = (v << 8) | (int(w * 8) + b < L ? p[b] : 0);
    rows[t] = v;
    if (w == 0) idx[i] = i;
}

__global__ void ascii_dedupe_kernel(const uint8_t* __restrict__ r, int L, const uint32_t* __restrict__ ids, uint32_t m,
                                    uint32_t* next, uint32_t* prev, uint16_t* offset) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i + 1 >= m) return;
    const uint32_t a = ids[i], b = ids[i + 1];
    const uint8_t* x = r + uint64_t(a) * L;
    const uint8_t* y = r + uint64_t(b) * L;
    for (int t = 0; t < L; ++t)
        if (x[t] != y[t]) return;
    prev[b] = a;
    next[a] = b;
    offset[a] = 0;
}

__global__ void ends_flags_kernel(const uint32_t* __restrict__ ids, uint32_t m, const uint32_t* __restrict__ next,
                                  const uint32_t* __restrict__ prev, uint8_t* __restrict__ pf, uint8_t* __restrict__ sf) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    pf[i] = prev[ids[i]] == INVALID;
    sf[i] = next[ids[i]] == INVALID;
}

}  // namespace

void full_match_packed(const BlockParams& p, const uint64_t* db, uint32_t* pre, uint32_t* suf, uint32_t cnt,
                       uint32_t* next, uint32_t* prev, uint16_t* offset, Arena& a, cudaStream_t s,
                       unsigned long long* tally) {
    full_match_loop(PackedAcc{db, p.W, p.L}, pre, suf, cnt, next, prev, offset, p.tune.fm_loop == 0, tally, a, s);
}

void sort_ids_by_ascii(const uint8_t* reads, int L, uint32_t* ids, uint32_t m, Arena& a, cudaStream_t s) {
    // stable lexicographic (memcmp) order
    if (m <= 1) return;
    auto mk = a.mark();
    const int W = (L + 7) / 8;
    uint64_t* rows = a.alloc<uint64_t>(size_t(m) * W);
    uint32_t* idx = a.alloc<uint32_t>(m);
    uint32_t* in = a.alloc<uint32_t>(m);
    CURC_CHECK(cudaMemcpyAsync(in, ids, size_t(m) * 4, cudaMemcpyDeviceToDevice, s));
    ascii_rows_kernel<<<grid_for(uint64_t(m) * W, 256), 256, 0, s>>>(reads, L, ids, m, W, rows, idx);
    CURC_LAUNCH_CHECK();
    sort_rows(rows, W, 8 * (L - 8 * (W - 1)), idx, m, a, s);
    fm_permute_kernel<<<grid_for(m, 256), 256, 0, s>>>(in, idx, m, ids);
    CURC_LAUNCH_CHECK();
    a.release(mk);
}

void full_match_ascii(const BlockParams& p, const uint8_t* reads, uint32_t* ids, uint32_t m, uint32_t n_total,
                      uint32_t* next, uint32_t* prev, uint16_t* offset, Arena& a, cudaStream_t s) {
    // compress.cu:1179-1210: sort, duplicate links, prefix/suffix lists
    unlinked(next, prev, offset, n_total, s);
    if (m == 0) return;
    sort_ids_by_ascii(reads, p.L, ids, m, a, s);
    if (m > 1) {
        ascii_dedupe_kernel<<<grid_for(m, 256), 256, 0, s>>>(reads, p.L, ids, m, next, prev, offset);
        CURC_LAUNCH_CHECK();
    }
    auto mk = a.mark();
    uint8_t* pf = a.alloc<uint8_t>(m);
    uint8_t* sf = a.alloc<uint8_t>(m);
    ends_flags_kernel<<<grid_for(m, 256), 256, 0, s>>>(ids, m, next, prev, pf, sf);
    CURC_LAUNCH_CHECK();
    uint32_t* pre = a.alloc<uint32_t>(m);
    uint32_t* suf = a.alloc<uint32_t>(m);
    uint32_t* counts = a.zeros<uint32_t>(3, s);  // ends of each kind, other symbols seen
    other_symbols_kernel<<<resident_grid(other_symbols_kernel, 256, uint64_t(m) * p.L), 256, 0, s>>>(reads, p.L, ids, m,
                                                                                                  counts + 2);
    CURC_LAUNCH_CHECK();
    select_flagged(ids, pf, pre, m, counts + 0, a, s);
    select_flagged(ids, sf, suf, m, counts + 1, a, s);
    uint32_t h[3];
    read_small(h, counts, 12, s);
    full_match_loop(AsciiAcc{reads, 0, p.L, h[2] != 0}, pre, suf, h[0], next, prev, offset,
                    p.tune.fm_loop == 0 && h[2] == 0, nullptr, a, s);
    a.release(mk);
}

}  // namespace curc
