// a1: 2-bit read packing and N-read separation.
//
// Reference: encode() compress.cu:2151-2180 (one thread per read, strided
// byte loads) and the N test of the host parser, preprocess.cpp:147-193.
//
// B200 design: a persistent grid whose warps walk tiles of 32 reads, each by
// itself.  A tile is 32*L contiguous bytes, moved into the warp's part of
// shared memory by a 1D TMA bulk copy (cp.async.bulk + mbarrier) one tile
// ahead of the packing, so HBM reads are full-line and the copies overlap it.
// The warp then works in two passes: every lane turns 16-byte groups of the
// tile into 32 bits of codes (one 16-byte shared-memory load each), giving the
// tile's bases as one contiguous 2-bit string, and then every lane cuts output
// words (32 bases) out of that string; packed words of a tile are contiguous
// in HBM, so stores coalesce.  Bytes per read: L in, 8*W + 1 out.
#include <mutex>
#include <stdexcept>

#include "stages.cuh"

namespace curc {

namespace {
constexpr int PACK_MAX_READS = 128;  // reads of a warp's tile, at most (a multiple of 16)
constexpr int PACK_STAGES = 2;  // tiles of a warp in shared memory: one is packed while the next is copied
constexpr uint32_t WAIT_LIMIT = 1u << 26;
constexpr int MAX_DEVICES = 64;

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_addr(dst)),
        "l"(src), "r"(bytes), "r"(smem_addr(bar))
        : "memory");
}

// Bits 1 and 2 of four ASCII bases (a little-endian word, first base in the low
// byte), one pair per byte: A/a 0, C/c 1, T/t 2, G/g 3, the Gray code of the
// 2-bit codes A 0, C 1, G 2, T 3.
__device__ __forceinline__ uint32_t gray4(uint32_t x) { return (x >> 1) & 0x03030303u; }

// Four pairs as eight bits, first base in the top two, in the top byte of the
// product (one multiply gathers them; no partial product carries into that
// byte).
__device__ __forceinline__ uint32_t gather4(uint32_t t) { return t * 0x40100401u; }

// Sixteen gathered pairs from Gray code to codes (the top bit of a pair stays,
// the lower one is their sum).
__device__ __forceinline__ uint32_t gray_codes(uint32_t c) { return c ^ ((c >> 1) & 0x55555555u); }

// Zero exactly when the eight bytes of a and b are all A, C, G or T in either
// case (ta, tb: their pairs).  The letters that the pairs stand for are looked
// up, in lower case, four at a time by a byte permute whose selector is four
// nibbles: with b's pairs in the upper nibbles of a's bytes, the low half of
// one word selects the letters of a0 b0 a1 b1 and its high half those of a2 b2
// a3 b3, to compare with the bytes in that order.  Setting bit 5 merges only a
// letter with its other case.
__device__ __forceinline__ uint32_t other8(uint32_t a, uint32_t b, uint32_t ta, uint32_t tb) {
    const uint32_t v = tb * 16u + ta;
    const uint32_t lo = __byte_perm(0x67746361u, 0u, v), hi = __byte_perm(0x67746361u, 0u, v >> 16);
    return (lo ^ (__byte_perm(a, b, 0x5140u) | 0x20202020u)) | (hi ^ (__byte_perm(a, b, 0x7362u) | 0x20202020u));
}

// The letters of four pairs, in lower case.
__device__ __forceinline__ uint32_t letters4(uint32_t t) {
    const uint32_t u = t | (t >> 4);
    return __byte_perm(0x67746361u, 0u, __byte_perm(u, 0u, 0x4420u));
}

// Shared memory of a warp: PACK_STAGES tiles (each a multiple of 128 bytes),
// then the codes of one tile of R reads (R / 16 * L words of 16 bases, and 4
// zero words).
__host__ __device__ inline uint32_t pack_tile_stride(int L, int R) { return (uint32_t(R) * L + 127u) & ~127u; }
__host__ __device__ inline uint32_t pack_warp_bytes(int L, int R) {
    return (PACK_STAGES * pack_tile_stride(L, R) + 4u * (uint32_t(R / 16) * uint32_t(L) + 4u) + 127u) & ~127u;
}
// Tiles of up to 4800 bytes: smaller ones leave lanes idle in the last rounds of
// both passes, larger ones keep fewer warps a SM (1.2 Gbases: 150 bp 414 us with
// 16 reads a tile, 385 with 32, 419 with 48; 36 bp 577 with 32, 452 with 64).
__host__ __device__ inline int pack_reads_of_tile(int L) {
    const int r = 4800 / (16 * L) * 16;
    return r < 16 ? 16 : r > PACK_MAX_READS ? PACK_MAX_READS : r;
}
constexpr int PACK_MAX_WARPS = 4;

// Each warp packs tiles of 32 reads by itself, with no barrier over the block:
// a bulk copy (TMA) brings the tile's bytes, 16 bytes a lane become 32 bits of
// codes (the tile as one 2-bit string), and each lane cuts words of 32 bases
// from three code words, which leave in one coalesced store.  What bounds it:
// logic instructions (about 100 issued per 16 bases of a lane, both passes; 2.5
// a clock and SM), then HBM.  20M reads of 150 bp on B200: 1.12 ms (3.4 TB/s) with
// blocks that packed 64 reads between two block barriers, where a third of the
// cycles went to waiting; 0.99 ms by warps; 0.92 ms with the tile sized by the
// read length; 0.86 ms (4.4 TB/s) with the letters of two words checked
// together and Gray code undone once per 16 bases.
__global__ void __launch_bounds__(32 * PACK_MAX_WARPS) pack_kernel(const uint8_t* __restrict__ seq, uint64_t n, int L,
                                                                   int W, int R, bool use_tma, uint64_t* __restrict__ packed,
                                                                   uint8_t* __restrict__ has_n,
                                                                   uint32_t* __restrict__ err) {
    extern __shared__ __align__(128) uint8_t smem_all[];
    __shared__ __align__(8) uint64_t bars[PACK_MAX_WARPS][PACK_STAGES];
    __shared__ uint8_t nflags[PACK_MAX_WARPS][PACK_MAX_READS];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint8_t* smem = smem_all + warp * pack_warp_bytes(L, R);
    uint64_t* bar = bars[warp];
    uint8_t* nf = nflags[warp];
    const uint32_t tile_bytes = uint32_t(R) * uint32_t(L);
    const uint32_t groups = tile_bytes / 16;
    const uint32_t stride = pack_tile_stride(L, R);
    uint32_t* codes = reinterpret_cast<uint32_t*>(smem + PACK_STAGES * stride);
    const uint64_t tiles = div_up(n, R), step = uint64_t(gridDim.x) * (blockDim.x >> 5);
    auto copied = [&](uint64_t t) { return use_tma && t < tiles && (t + 1) * R <= n; };
    auto issue = [&](uint64_t t, int stage) {
        mbar_expect_tx(&bar[stage], tile_bytes);
        bulk_g2s(smem + stage * stride, seq + t * uint64_t(R) * L, tile_bytes, &bar[stage]);
    };
    if (lane == 0) {
        for (int st = 0; st < PACK_STAGES; ++st) mbar_init(&bar[st], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (uint32_t r = lane; r < uint32_t(R); r += 32) nf[r] = 0;
    if (lane < 4) codes[groups + lane] = 0;
    __syncwarp();
    uint64_t t = uint64_t(blockIdx.x) * (blockDim.x >> 5) + warp;
    if (lane == 0 && copied(t)) issue(t, 0);
    // word q of the tile is word q - r W of read r = q / W, by one multiply
    // (exact for q W < 65536)
    const uint32_t words = uint32_t(R) * uint32_t(W), inv_w = 65536u / uint32_t(W) + 1u;
    const uint64_t tail = ~0ull << (64 * W - 2 * L);  // the last word's bases
    uint32_t uses[PACK_STAGES] = {0, 0};  // copies a stage has received
    for (uint32_t it = 0; t < tiles; t += step, ++it) {
        const int stage = int(it % PACK_STAGES);
        uint8_t* buf = smem + stage * stride;
        const uint64_t nt = t + step;
        if (lane == 0 && copied(nt)) {  // the other stage was read before the last __syncwarp
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            issue(nt, stage ^ 1);
        }
        const uint64_t rem = n - t * R;
        const uint32_t nr = rem < uint64_t(R) ? uint32_t(rem) : uint32_t(R);
        if (copied(t)) {
            uint32_t spins = 0;
            bool late = false;
            while (!mbar_try_wait(&bar[stage], uses[stage] & 1u)) {
                if (++spins > WAIT_LIMIT) {  // never expected
                    late = true;
                    break;
                }
            }
            ++uses[stage];
            if (__any_sync(0xFFFFFFFFu, late)) {
                // report, write nothing of this tile, and leave only once the
                // other stage's copy (if one is in flight) has also landed or
                // had the same bounded wait, so that, as far as waiting can
                // tell, no bulk copy still targets this block's shared memory
                if (lane == 0) {
                    atomicExch(err, 1u);
                    if (copied(nt))
                        for (uint32_t w = 0; w < WAIT_LIMIT && !mbar_try_wait(&bar[stage ^ 1], uses[stage ^ 1] & 1u);
                             ++w) {
                        }
                }
                __syncwarp();
                return;
            }
        } else {
            // the last, partial tile, or reads that do not start on 16 bytes:
            // words cut from two aligned ones, the rest of the tile 'A'
            const uint8_t* src = seq + t * uint64_t(R) * L;
            const uint32_t have = nr * uint32_t(L), by = 8u * uint32_t(reinterpret_cast<uintptr_t>(src) & 3u);
            const uint32_t* p = reinterpret_cast<const uint32_t*>(src - (by >> 3));
            uint32_t* out = reinterpret_cast<uint32_t*>(buf);
#pragma unroll 4
            for (uint32_t i = lane; i < tile_bytes / 4; i += 32) {
                uint32_t v = 0x41414141u;
                if (4 * i + 8 <= have) {  // the second word too lies among the tile's bytes
                    v = by ? __funnelshift_r(p[i], p[i + 1], by) : p[i];
                } else {
                    for (uint32_t b = 0; b < 4; ++b)
                        if (4 * i + b < have)
                            v = (v & ~(0xFFu << (8 * b))) | uint32_t(src[4 * i + b]) << (8 * b);
                }
                out[i] = v;
            }
            __syncwarp();
        }
        // 16 bytes -> 32 bits of codes, first base in the top bits
        for (uint32_t g = lane; g < groups; g += 32) {
            const uint4 x = reinterpret_cast<const uint4*>(buf)[g];
            const uint32_t t0 = gray4(x.x), t1 = gray4(x.y), t2 = gray4(x.z), t3 = gray4(x.w);
            // the top bytes of the four products: byte 3 from the first word
            uint32_t c = __byte_perm(__byte_perm(gather4(t3), gather4(t2), 0x0073u),
                                     __byte_perm(gather4(t1), gather4(t0), 0x0073u), 0x5410u);
            const uint32_t d = other8(x.x, x.y, t0, t1) | other8(x.z, x.w, t2, t3);
            if (d != 0) {
                // N and other letters: code 0, as A
                const uint32_t xs[4] = {x.x, x.y, x.z, x.w};
                const uint32_t ts[4] = {t0, t1, t2, t3};
                c = 0;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint32_t same = __vcmpeq4(letters4(ts[i]), xs[i] | 0x20202020u);
                    c = (c << 8) | (gather4(ts[i] & same) >> 24);
                    for (uint32_t m = __vcmpeq4(xs[i], 0x4E4E4E4Eu); m; m &= m - 1) {
                        const uint32_t bit = uint32_t(__ffs(m)) - 1u;
                        if ((bit & 7u) == 0) nf[(16 * g + 4 * i + (bit >> 3)) / uint32_t(L)] = 1;
                    }
                }
            }
            codes[g] = gray_codes(c);
        }
        __syncwarp();
        // the 32 bases of each word, from the code string
        const uint32_t words_here = nr * uint32_t(W);
        uint64_t* out = packed + t * words;
        for (uint32_t q = lane; q < words_here; q += 32) {
            const uint32_t r = (q * inv_w) >> 16, w = q - r * uint32_t(W);
            const uint32_t o = r * uint32_t(L) + 32u * w;
            const uint32_t k = o >> 4, sh = (o & 15u) * 2u;
            const uint32_t a = codes[k], b = codes[k + 1], c = codes[k + 2];
            uint64_t v = uint64_t(__funnelshift_l(b, a, sh)) << 32 | __funnelshift_l(c, b, sh);
            if (w + 1 == uint32_t(W)) v &= tail;
            out[q] = v;
        }
        for (uint32_t r = lane; r < nr; r += 32) {
            has_n[t * R + r] = nf[r];
            nf[r] = 0;
        }
        __syncwarp();
    }
}

__global__ void invert_flags_kernel(const uint8_t* __restrict__ in, uint8_t* __restrict__ out, uint64_t n) {
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += uint64_t(gridDim.x) * blockDim.x)
        out[i] = in[i] ? 0 : 1;
}

__global__ void gather_reads_ascii_kernel(const uint8_t* __restrict__ seq, const uint32_t* __restrict__ ids,
                                          uint32_t m, int L, uint8_t* __restrict__ out) {
    // one warp per read
    const uint32_t warp = (uint32_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp >= m) return;
    const uint8_t* s = seq + uint64_t(ids[warp]) * L;
    uint8_t* d = out + uint64_t(warp) * L;
    for (int j = lane; j < L; j += 32) d[j] = s[j];
}
}  // namespace

void pack_reads(const uint8_t* seq, uint64_t n, int L, uint64_t* packed, uint8_t* has_n, uint32_t* err,
                cudaStream_t s) {
    if (n == 0) return;
    const int W = (L + 31) / 32;
    const bool aligned = (reinterpret_cast<uintptr_t>(seq) & 15u) == 0;
    // the dynamic shared-memory limit is a per-device attribute: raise it
    // once on every device this process packs on
    static std::mutex mu;
    static bool attr_set[MAX_DEVICES] = {};
    int dev = 0;
    CURC_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= MAX_DEVICES) throw std::runtime_error("device ordinal out of range");
    {
        std::lock_guard<std::mutex> g(mu);
        if (!attr_set[dev]) {
            CURC_CHECK(cudaFuncSetAttribute(pack_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            int(PACK_MAX_WARPS * pack_warp_bytes(512, 16))));
            attr_set[dev] = true;
        }
    }
    const int R = pack_reads_of_tile(L);
    const uint64_t tiles = div_up(n, uint64_t(R));
    // few tiles: spread over the SMs, one warp a block
    const int warps = tiles < uint64_t(SM_COUNT_B200) * PACK_MAX_WARPS ? 1 : PACK_MAX_WARPS, threads = 32 * warps;
    const size_t smem = size_t(warps) * pack_warp_bytes(L, R);
    int per_sm = 0;
    CURC_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pack_kernel, threads, smem));
    const int grid = int(std::min<uint64_t>(div_up(tiles, uint64_t(warps)),
                                            uint64_t(SM_COUNT_B200) * uint64_t(std::max(1, per_sm))));
    pack_kernel<<<grid, threads, smem, s>>>(seq, n, L, W, R, aligned, packed, has_n, err);
    CURC_LAUNCH_CHECK();
}

void split_n_reads(const uint8_t* has_n, uint64_t n, uint32_t* reads_id, uint32_t* n_reads_id, uint32_t* counts,
                   Arena& a, cudaStream_t s) {
    // preprocess.cpp:147-193: ids of reads without N ascending, ids of reads
    // with N ascending.
    auto m = a.mark();
    uint8_t* inv = a.alloc<uint8_t>(n ? n : 1);
    if (n) {
        invert_flags_kernel<<<grid_for(n, 256, 4), 256, 0, s>>>(has_n, inv, n);
        CURC_LAUNCH_CHECK();
    }
    select_indices(inv, reads_id, n, counts + 0, a, s);
    select_indices(has_n, n_reads_id, n, counts + 1, a, s);
    a.release(m);
}

void gather_ascii_rows(const uint8_t* seq, const uint32_t* ids, uint32_t m, int L, uint8_t* out, cudaStream_t s) {
    if (!m) return;
    gather_reads_ascii_kernel<<<grid_for(uint64_t(m) * 32, 256), 256, 0, s>>>(seq, ids, m, L, out);
    CURC_LAUNCH_CHECK();
}

}  // namespace curc
