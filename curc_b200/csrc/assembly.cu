// a8: walk linked reads into a pseudogenome.
//
// Reference: RefRecord::assembly compress.cu:107-217 (a sequential pointer
// chase on the host) and compute_binary_ref compress.cu:229-246.
//
// Output order of the reference: chains in order of their first member in
// the id list; each chain from its head, every read contributing offset[r]
// bases and the tail all L bases; a cycle is cut after its member with the
// largest offset (first maximum met walking from the successor of the
// cycle's first listed member), which becomes the tail.
//
// B200 design: list ranking with a sparse ruling set.  Every chain head and
// one member in 8 (by a hash of its id) is a ruler; one thread per ruler
// walks its sublist up to the next ruler, giving every read its offset
// within the sublist; the rulers (about an eighth of the reads, resident
// in L2) are then ranked by pointer jumping, and one pass over the members
// adds the two.  Each read is touched a constant number of times instead of
// once per jumping round.  Cycles show up as ruler lists whose pointers never
// clear (a cycle without any ruler gets one: its member of smallest list
// index) and are cut in parallel (below); chains are ordered by their first
// list index with a radix sort and placed by exclusive scans; every read
// then writes its bases independently.
#include <mutex>

#include "stages.cuh"

namespace curc {

namespace {

__global__ void scatter_index_kernel(const uint32_t* __restrict__ ids, uint32_t m, uint32_t* __restrict__ pos_in_ids) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < m) pos_in_ids[ids[i]] = i;
}

constexpr uint32_t RULER_SPACING = 8;  // one sampled ruler per 8 members (power of two)

// Pointer-jumping state, 32 bytes so that one jump gathers one sector.  For
// a ruler: acc / cnt = bases / reads of the sublists before its own, mn = the
// smallest list index over its own and the preceding sublists, far = the
// chain's head ruler.  The final per-member state (indexed by list index)
// has the same fields for the read itself: far = the head read, acc = its
// base offset in the chain, cnt = its rank, and mn, which covers at least
// the read's predecessors and is the chain's (or cycle's) minimum at the
// tail (or on a cycle).
struct __align__(32) RankState {
    uint64_t acc;
    uint32_t jump;    // ruler 2^t sublists back, INVALID once past the head
    uint32_t far;
    uint32_t cnt;
    uint32_t mn;
    uint32_t pad0, pad1;
};

// The links of one read in one 16-byte gather: successor, the read's own
// offset to it, list index, ruler index (INVALID unless a ruler).
struct __align__(16) ChainNode {
    uint32_t nx, off, pos, rix;
};

// Position of a read within its ruler's sublist (indexed by list index).
struct __align__(32) SubPos {
    uint64_t la;     // bases from the ruler's first base to this read's
    uint32_t owner;  // ruler index
    uint32_t lc;     // reads between the ruler and this read
    uint32_t lm;     // smallest list index from the ruler to this read
    uint32_t epoch;  // walk that wrote the entry; older entries mean "not reached"
    uint32_t pad1, pad2;
};

// Totals of one ruler's sublist.
struct __align__(16) SubTotal {
    uint64_t acc;   // bases from the ruler's first base to the next ruler's
    uint32_t cnt;   // reads in the sublist
    uint32_t mn;    // smallest list index in the sublist
};

__global__ void ruler_flags_kernel(const uint32_t* __restrict__ ids, uint32_t m, const uint32_t* __restrict__ pv,
                                   const uint8_t* __restrict__ promote, uint8_t* __restrict__ f) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    const uint32_t x = ids[i];
    f[i] = pv[x] == INVALID || (murmur64(x) & (RULER_SPACING - 1)) == 0 || (promote && promote[i]);
}

// One node per read, written in read order (non-members get INVALID
// fields, so a link out of the member set is caught by the walk).
__global__ void chain_nodes_kernel(uint32_t n, const uint32_t* __restrict__ pos_in_ids,
                                   const uint32_t* __restrict__ nx, const uint16_t* __restrict__ offset,
                                   ChainNode* __restrict__ node) {
    for (uint32_t x = blockIdx.x * blockDim.x + threadIdx.x; x < n; x += gridDim.x * blockDim.x) {
        const uint32_t i = pos_in_ids[x];
        if (i == INVALID) {
            node[x] = ChainNode{INVALID, 0u, INVALID, INVALID};
        } else {
            const uint32_t nn = nx[x];
            node[x] = ChainNode{nn, nn == INVALID ? 0u : uint32_t(offset[x]), i, INVALID};
        }
    }
}

__global__ void ruler_index_kernel(const uint32_t* __restrict__ rul, uint32_t nr, ChainNode* __restrict__ node) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < nr) node[rul[t]].rix = t;
}

// One thread per ruler walks its sublist; the walk ends at the next ruler
// or the chain's tail (a walk that comes back to a ruler on a cycle ends
// there too), at most m steps.
__global__ void ruler_walk_kernel(const uint32_t* __restrict__ rul, uint32_t nr, uint32_t m, uint32_t n,
                                  uint32_t epoch, const ChainNode* __restrict__ node, SubPos* __restrict__ loc,
                                  SubTotal* __restrict__ tot, uint32_t* __restrict__ err) {
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < nr; t += gridDim.x * blockDim.x) {
        ChainNode c = node[rul[t]];
        uint64_t la = 0;
        uint32_t lc = 0, lm = c.pos;
        loc[c.pos] = SubPos{0, t, 0, lm, epoch, 0, 0};
        for (uint32_t step = 0; step < m && c.nx != INVALID; ++step) {
            if (c.nx >= n || node[c.nx].pos >= m) {  // a link out of the member set
                atomicExch(err, 1u);
                break;
            }
            const ChainNode d = node[c.nx];
            la += c.off;
            ++lc;
            if (d.rix != INVALID) break;
            lm = min(lm, d.pos);
            loc[d.pos] = SubPos{la, t, lc, lm, epoch, 0, 0};
            c = d;
        }
        tot[t] = SubTotal{la, lc, lm};
    }
}

// Members that no walk reached (cycles without a ruler).
__global__ void __launch_bounds__(256) unreached_kernel(uint32_t m, uint32_t epoch, const SubPos* __restrict__ loc,
                                                        uint8_t* __restrict__ flag, uint32_t* __restrict__ count) {
    uint32_t c = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
        const bool u = loc[i].epoch != epoch;
        flag[i] = u;
        c += u;
    }
    block_tally<uint32_t>(c, count);
}

// On a cycle without a ruler, its member of smallest list index becomes
// one: each member walks the cycle (bounded by m steps) for the minimum.
__global__ void promote_kernel(const uint32_t* __restrict__ ids, uint32_t m, uint32_t n,
                               const uint8_t* __restrict__ unreached,
                               const uint32_t* __restrict__ nx, const uint32_t* __restrict__ pos_in_ids,
                               uint8_t* __restrict__ promote) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m || !unreached[i]) return;
    const uint32_t x = ids[i];
    uint32_t y = nx[x];
    bool smallest = true;
    for (uint32_t step = 0; step < m && y != x && y < n; ++step) {
        if (pos_in_ids[y] < i) {  // non-members hold INVALID
            smallest = false;
            break;
        }
        y = nx[y];
    }
    promote[i] = smallest;
}

// Ruler ranking state: the predecessor ruler owns the read before this
// ruler's first read.
__global__ void ruler_init_kernel(const uint32_t* __restrict__ rul, uint32_t nr, uint32_t m,
                                  const uint32_t* __restrict__ pv,
                                  const uint32_t* __restrict__ pos_in_ids, const SubPos* __restrict__ loc,
                                  const SubTotal* __restrict__ tot, RankState* __restrict__ st) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nr) return;
    const uint32_t p = pv[rul[t]];
    const uint32_t pi = p == INVALID ? INVALID : pos_in_ids[p];
    const uint32_t pr = pi < m ? loc[pi].owner : INVALID;
    RankState r;
    r.jump = pr;
    r.far = pr == INVALID ? t : pr;
    r.acc = pr == INVALID ? 0 : tot[pr].acc;
    r.cnt = pr == INVALID ? 0 : tot[pr].cnt;
    r.mn = tot[t].mn;
    if (pr != INVALID) r.mn = min(r.mn, tot[pr].mn);
    r.pad0 = r.pad1 = 0;
    st[t] = r;
}

// One jump for every ruler (grid-stride); *active counts the rulers whose
// pointer is still set afterwards.
__global__ void __launch_bounds__(512) rank_step_kernel(uint32_t n, const RankState* __restrict__ in,
                                                        RankState* __restrict__ out, uint32_t* __restrict__ active) {
    uint32_t still = 0;
    for (uint32_t x = blockIdx.x * blockDim.x + threadIdx.x; x < n; x += gridDim.x * blockDim.x) {
        RankState st = in[x];
        if (st.jump != INVALID) {
            const RankState a = in[st.jump];
            st.far = a.far;
            st.acc += a.acc;
            st.cnt += a.cnt;
            st.mn = min(st.mn, a.mn);
            st.jump = a.jump;
            still += st.jump != INVALID;
        }
        out[x] = st;
    }
    block_tally<uint32_t>(still, active);
}

// Every round for up to RANK_CLUSTER rulers by one cluster, with a barrier
// between rounds: 17 rounds of 10,000 rulers took 75 us as launches with a
// count read back every four.  Ends when no pointer is left or after `rounds`
// (cycles); done: pointers left, rounds taken.  Ranking of 50k reads' rulers
// 0.25 -> 0.12 ms, 700k reads 0.49 -> 0.25; with up to 300,000 rulers 16 SMs
// are too few (1M pairs 0.40 -> 0.69), with 65,536 they are not (0.31).
constexpr unsigned RANK_BLOCKS = 16;
constexpr uint32_t RANK_CLUSTER = 65536;
__device__ __forceinline__ RankState ld_state(const RankState* p) {  // written by other SMs
    const uint4* q = reinterpret_cast<const uint4*>(p);
    uint4 w[2] = {__ldcg(q), __ldcg(q + 1)};
    RankState r;
    memcpy(&r, w, sizeof(r));
    return r;
}
__global__ void __launch_bounds__(512) rank_rounds_kernel(uint32_t n, RankState* A, RankState* B, uint32_t rounds,
                                                          uint32_t* __restrict__ active, uint32_t* __restrict__ done) {
    const uint32_t me = blockIdx.x * 512 + threadIdx.x;
    for (uint32_t t = 0;; ++t) {
        const RankState* in = t & 1 ? B : A;
        RankState* out = t & 1 ? A : B;
        uint32_t still = 0;
        for (uint32_t x = me; x < n; x += gridDim.x * 512) {
            RankState st = ld_state(in + x);
            if (st.jump != INVALID) {
                const RankState a = ld_state(in + st.jump);
                st.far = a.far;
                st.acc += a.acc;
                st.cnt += a.cnt;
                st.mn = min(st.mn, a.mn);
                st.jump = a.jump;
                still += st.jump != INVALID;
            }
            out[x] = st;
        }
        block_tally<uint32_t>(still, active + t);
        cluster_arrive();
        cluster_wait();
        const uint32_t left = __ldcg(active + t);  // the same for every thread
        if (left == 0 || t + 1 == rounds) {
            if (me == 0) {
                done[0] = left;
                done[1] = t + 1;
            }
            return;
        }
    }
}

// Member state = its ruler's + its place in the sublist.  jump stays set for
// members of a cycle.  The rulers' states are in A or B by the rounds taken.
__global__ void member_state_kernel(uint32_t m, const uint32_t* __restrict__ rul, const SubPos* __restrict__ loc,
                                    const RankState* __restrict__ A, const RankState* __restrict__ B,
                                    const uint32_t* __restrict__ done, RankState* __restrict__ st) {
    const RankState* rs = done[1] & 1 ? B : A;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    const SubPos l = loc[i];
    const RankState r = rs[l.owner];
    RankState o;
    o.acc = r.acc + l.la;
    o.jump = r.jump;
    o.far = rul[r.far];
    o.cnt = r.cnt + l.lc;
    o.mn = min(r.mn, l.lm);
    o.pad0 = o.pad1 = 0;
    st[i] = o;
}

__global__ void cycle_flags_kernel(uint32_t m, const RankState* __restrict__ st, uint8_t* __restrict__ cyc) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < m) cyc[i] = st[i].jump != INVALID;
}

// Cycles are cut in parallel.  The reference walks each cycle from the
// successor h of its first listed read r (the read visited first) round to
// r, and cuts after the first read of largest offset met on the way.  Here:
// (1) a temporary cut between r and h makes each cycle a chain h .. r;
// (2) ranking that chain gives every read its walk position;
// (3) the largest (offset, -position) over the chain picks the cut read;
// (4) the temporary cut is undone and the real one made.

// (1) r = the cycle member whose list index is the cycle's minimum (mn on a
// cycle covers the whole cycle).
__global__ void cycle_open_kernel(const uint32_t* __restrict__ ids, uint32_t m, const RankState* __restrict__ st,
                                  const uint8_t* __restrict__ cyc, uint32_t* nx, uint32_t* pv,
                                  uint32_t* __restrict__ leader_of_head, uint32_t* __restrict__ err) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m || !cyc[i] || st[i].mn != i) return;
    const uint32_t x = ids[i];
    const uint32_t h = nx[x];
    if (h == INVALID || pv[h] != x) {
        atomicExch(err, 1u);
        return;
    }
    leader_of_head[h] = x;
    pv[h] = INVALID;
    nx[x] = INVALID;
}

// (3) per chain head: max of (offset << 32 | ~position)
__global__ void cycle_max_kernel(const uint32_t* __restrict__ ids, uint32_t m, const RankState* __restrict__ st,
                                 const uint8_t* __restrict__ cyc, const uint16_t* __restrict__ offset,
                                 unsigned long long* __restrict__ best) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m || !cyc[i]) return;
    const unsigned long long key = (unsigned long long)offset[ids[i]] << 32 | (0xFFFFFFFFu - st[i].cnt);
    atomicMax(&best[st[i].far], key);
}

// (4) the read that holds its chain's maximum restores the temporary cut and
// makes the real one after itself.
__global__ void cycle_cut_kernel(const uint32_t* __restrict__ ids, uint32_t m, const RankState* __restrict__ st,
                                 const uint8_t* __restrict__ cyc, const unsigned long long* __restrict__ best,
                                 const uint32_t* __restrict__ leader_of_head, uint32_t* nx, uint32_t* pv) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m || !cyc[i]) return;
    const uint32_t h = st[i].far;
    if ((0xFFFFFFFFu - uint32_t(best[h] & 0xFFFFFFFFull)) != st[i].cnt) return;
    const uint32_t r = leader_of_head[h];
    pv[h] = r;
    nx[r] = h;
    const uint32_t x = ids[i];
    const uint32_t nh = nx[x];
    nx[x] = INVALID;
    pv[nh] = INVALID;
}

// The cycle members as a list of their own (in list order).
__global__ void cycle_list_kernel(const uint32_t* __restrict__ ids, const uint32_t* __restrict__ cidx, uint32_t mc,
                                  uint32_t* __restrict__ cids, uint32_t* __restrict__ pos_in_cyc) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= mc) return;
    const uint32_t x = ids[cidx[t]];
    cids[t] = x;
    pos_in_cyc[x] = t;
}

// States of the cut cycles back into the full list (mn to a list index).
__global__ void cycle_merge_kernel(const uint32_t* __restrict__ cidx, uint32_t mc, const RankState* __restrict__ T,
                                   RankState* __restrict__ R) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= mc) return;
    RankState r = T[t];
    r.mn = cidx[r.mn];
    R[cidx[t]] = r;
}

// The chain's first list index, from its tail (whose mn covers the chain).
__global__ void chain_key_kernel(const uint32_t* __restrict__ ids, uint32_t m, const uint32_t* __restrict__ nx,
                                 const RankState* __restrict__ st, uint32_t* __restrict__ key) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < m && nx[ids[i]] == INVALID) key[st[i].far] = st[i].mn;
}

__global__ void head_flags_kernel(const uint32_t* __restrict__ ids, uint32_t m, const uint32_t* __restrict__ pv,
                                  uint8_t* __restrict__ f) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < m) f[i] = pv[ids[i]] == INVALID;
}

__global__ void tail_sizes_kernel(const uint32_t* __restrict__ ids, uint32_t m, const uint32_t* __restrict__ nx,
                                  const RankState* __restrict__ st, int L, uint64_t* __restrict__ chain_bases,
                                  uint32_t* __restrict__ chain_members) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m || nx[ids[i]] != INVALID) return;
    chain_bases[st[i].far] = st[i].acc + uint64_t(L);
    chain_members[st[i].far] = st[i].cnt + 1;
}

__global__ void gather_heads_kernel(const uint32_t* __restrict__ heads, uint32_t nh, const uint32_t* __restrict__ key,
                                    uint32_t* __restrict__ hkey) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < nh) hkey[t] = key[heads[t]];
}

__global__ void chain_sizes_sorted_kernel(const uint32_t* __restrict__ heads, uint32_t nh,
                                          const uint64_t* __restrict__ chain_bases,
                                          const uint32_t* __restrict__ chain_members, uint64_t* __restrict__ cb,
                                          uint32_t* __restrict__ cm, uint32_t* __restrict__ slot) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nh) return;
    const uint32_t h = heads[t];
    cb[t] = chain_bases[h];
    cm[t] = chain_members[h];
    slot[h] = t;
}

__global__ void place_kernel(const uint32_t* __restrict__ ids, uint32_t m, const uint32_t* __restrict__ nx,
                             const RankState* __restrict__ st,
                             const uint32_t* __restrict__ slot, const uint64_t* __restrict__ cpos,
                             const uint32_t* __restrict__ crec, const uint16_t* __restrict__ offset,
                             const uint64_t* __restrict__ db, const uint8_t* __restrict__ ascii, int L, int W,
                             uint8_t is_n, DevRecord* __restrict__ rec, uint8_t* __restrict__ seq) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    const uint32_t x = ids[i];
    const RankState r = st[i];
    const uint32_t c = slot[r.far];
    const uint64_t pos = cpos[c] + r.acc;
    DevRecord d;
    d.read_id = x;
    d.is_n = is_n;
    d.strand = 0;
    d.pad = 0;
    d.pos = pos;
    rec[crec[c] + r.cnt] = d;
    const int nb = nx[x] == INVALID ? L : offset[x];
    uint8_t* out = seq + pos;
    if (ascii) {
        const uint8_t* src = ascii + uint64_t(x) * L;
        for (int j = 0; j < nb; ++j) out[j] = src[j];
    } else {
        const uint64_t* rd = db + uint64_t(x) * W;
        for (int j = 0; j < nb; ++j) out[j] = "ACGT"[code_at(rd, j)];
    }
}

__global__ void pack_ref_kernel(const uint8_t* __restrict__ seq, uint64_t len, uint64_t* __restrict__ packed,
                                uint64_t words) {
    for (uint64_t w = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; w < words; w += uint64_t(gridDim.x) * blockDim.x) {
        uint64_t v = 0;
        const uint64_t b = w * 32;
        for (int j = 0; j < 32; ++j) {
            const uint64_t q = b + j;
            v = (v << 2) | uint64_t(q < len ? ascii_code(seq[q]) : 0);
        }
        packed[w] = v;
    }
}

// ---------------------------------------------------------------- short lists
//
// Up to ASM_SMALL members by one block: links as list indices in shared
// memory, ranks by pointer jumping, cycles cut by one thread each, chains
// placed by a scan over their first list indices.  One launch and one read
// back, where the general path takes 40 launches and six (0.3 ms for a list of
// 20 reads, three lists a block).
constexpr uint32_t ASM_SMALL = 8192;
constexpr int ASM_THREADS = 1024, ASM_EACH = ASM_SMALL / ASM_THREADS;
constexpr uint16_t ASM_NONE = 0xFFFFu;
constexpr size_t asm_small_bytes(uint32_t m) { return size_t(m) * (3 * 2 + 4 + 4 * 2) + 256; }

// out[0] = bases of all chains; *err: a link leaves the list.  place[i] = the
// first base of member i.
__global__ void __launch_bounds__(ASM_THREADS) assemble_small_kernel(
    const uint32_t* __restrict__ ids, uint32_t m, uint32_t n, const uint32_t* __restrict__ next,
    const uint32_t* __restrict__ prev, const uint16_t* __restrict__ offset, int L, uint8_t is_n,
    uint32_t* pos_in_ids, DevRecord* __restrict__ rec, uint64_t* __restrict__ place, uint8_t* __restrict__ tail,
    uint64_t* __restrict__ out, uint32_t* __restrict__ err) {
    extern __shared__ __align__(16) uint8_t asm_smem[];
    uint32_t* acc = reinterpret_cast<uint32_t*>(asm_smem);  // bases before this member (later: per first index)
    uint16_t* nx = reinterpret_cast<uint16_t*>(acc + m);
    uint16_t* pv = nx + m;
    uint16_t* off = pv + m;
    uint16_t* jump = off + m;
    uint16_t* cnt = jump + m;
    uint16_t* mn = cnt + m;
    uint16_t* far = mn + m;
    __shared__ uint32_t s_warp[32], s_warp2[32];
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    for (uint32_t i = t; i < m; i += ASM_THREADS) pos_in_ids[ids[i]] = i;
    __syncthreads();
    // the member's list index of a linked read
    auto index = [&](uint32_t x) -> uint16_t {
        if (x == INVALID) return ASM_NONE;
        const uint32_t p = x < n ? pos_in_ids[x] : INVALID;
        if (p >= m || ids[p] != x) {
            atomicExch(err, 1u);
            return ASM_NONE;
        }
        return uint16_t(p);
    };
    for (uint32_t i = t; i < m; i += ASM_THREADS) {
        const uint32_t x = ids[i];
        nx[i] = index(next[x]);
        pv[i] = index(prev[x]);
        off[i] = nx[i] == ASM_NONE ? 0 : offset[x];
    }
    __syncthreads();
    uint32_t a[ASM_EACH];
    uint16_t j[ASM_EACH], c[ASM_EACH], lo[ASM_EACH], f[ASM_EACH];
    // ranks; returns whether this thread saw a cycle
    auto rank = [&]() -> bool {
#pragma unroll
        for (int e = 0; e < ASM_EACH; ++e) {
            const uint32_t i = t + e * ASM_THREADS;
            if (i >= m) continue;
            const uint16_t p = pv[i];
            jump[i] = p;
            acc[i] = p == ASM_NONE ? 0 : off[p];
            cnt[i] = p != ASM_NONE;
            mn[i] = p == ASM_NONE ? uint16_t(i) : min(uint16_t(i), p);
            far[i] = p == ASM_NONE ? uint16_t(i) : p;
        }
        __syncthreads();
        for (uint32_t span = 1; span < 2 * m; span *= 2) {
#pragma unroll
            for (int e = 0; e < ASM_EACH; ++e) {
                const uint32_t i = t + e * ASM_THREADS;
                j[e] = ASM_NONE;
                if (i >= m || jump[i] == ASM_NONE) continue;
                const uint32_t p = jump[i];
                j[e] = uint16_t(p);
                a[e] = acc[i] + acc[p];
                c[e] = uint16_t(cnt[i] + cnt[p]);
                lo[e] = min(mn[i], mn[p]);
                f[e] = far[p];
            }
            bool any = false;
#pragma unroll
            for (int e = 0; e < ASM_EACH; ++e) any |= j[e] != ASM_NONE;
            if (!__syncthreads_or(any)) return false;
            uint16_t nj[ASM_EACH];
#pragma unroll
            for (int e = 0; e < ASM_EACH; ++e) nj[e] = j[e] == ASM_NONE ? ASM_NONE : jump[j[e]];
            __syncthreads();
#pragma unroll
            for (int e = 0; e < ASM_EACH; ++e) {
                const uint32_t i = t + e * ASM_THREADS;
                if (j[e] == ASM_NONE) continue;
                jump[i] = nj[e];
                acc[i] = a[e];
                cnt[i] = c[e];
                mn[i] = lo[e];
                far[i] = f[e];
            }
            __syncthreads();
        }
        bool cyc = false;
#pragma unroll
        for (int e = 0; e < ASM_EACH; ++e) {
            const uint32_t i = t + e * ASM_THREADS;
            if (i < m) cyc |= jump[i] != ASM_NONE;
        }
        return cyc;
    };
    bool cyc = rank();
    if (__syncthreads_or(cyc)) {
        // the cycle's first listed read r walks it from its successor round to
        // itself and cuts after the first read of largest offset
#pragma unroll
        for (int e = 0; e < ASM_EACH; ++e) {
            const uint32_t r = t + e * ASM_THREADS;
            if (r >= m || jump[r] == ASM_NONE || mn[r] != r) continue;
            uint32_t x = nx[r], best = x;
            for (uint32_t step = 0; step < m && x != r && x < m; ++step) {
                x = nx[x];
                if (x < m && off[x] > off[best]) best = x;
            }
            if (x != r) {
                atomicExch(err, 1u);
                continue;
            }
            pv[nx[best]] = ASM_NONE;
            nx[best] = ASM_NONE;
        }
        __syncthreads();
        cyc = rank();
        if (__syncthreads_or(cyc)) {
            if (t == 0) atomicExch(err, 2u);
            return;
        }
    }
    // what follows needs each member's rank in registers and its chain's first
    // list index; the shared arrays then hold per first index the chain's
    // bases and members, and their exclusive scans
    uint16_t head[ASM_EACH];
#pragma unroll
    for (int e = 0; e < ASM_EACH; ++e) {
        const uint32_t i = t + e * ASM_THREADS;
        if (i >= m) continue;
        a[e] = acc[i];
        c[e] = cnt[i];
        lo[e] = mn[i];
        head[e] = far[i];
    }
    __syncthreads();
    uint16_t* key = jump;  // per head: the chain's first list index
#pragma unroll
    for (int e = 0; e < ASM_EACH; ++e) {
        const uint32_t i = t + e * ASM_THREADS;
        if (i >= m) continue;
        if (nx[i] == ASM_NONE) key[head[e]] = lo[e];  // the tail's minimum covers the chain
        acc[i] = 0;
        cnt[i] = 0;
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < ASM_EACH; ++e) {
        const uint32_t i = t + e * ASM_THREADS;
        if (i < m && nx[i] == ASM_NONE) {
            acc[lo[e]] = a[e] + uint32_t(L);
            cnt[lo[e]] = uint16_t(c[e] + 1);
        }
    }
    __syncthreads();
    // exclusive scans over the list, ASM_EACH consecutive entries per thread
    uint32_t vb = 0, vc = 0;
    for (uint32_t i = t * ASM_EACH; i < (t + 1) * ASM_EACH && i < m; ++i) {
        vb += acc[i];
        vc += cnt[i];
    }
    uint32_t xb = vb, xc = vc;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t yb = __shfl_up_sync(0xFFFFFFFFu, xb, d), yc = __shfl_up_sync(0xFFFFFFFFu, xc, d);
        if (lane >= uint32_t(d)) {
            xb += yb;
            xc += yc;
        }
    }
    if (lane == 31) {
        s_warp[warp] = xb;
        s_warp2[warp] = xc;
    }
    __syncthreads();
    uint32_t ob = xb - vb, oc = xc - vc, total = 0;
    for (uint32_t w = 0; w < 32; ++w) {
        if (w < warp) {
            ob += s_warp[w];
            oc += s_warp2[w];
        }
        total += s_warp[w];
    }
    for (uint32_t i = t * ASM_EACH; i < (t + 1) * ASM_EACH && i < m; ++i) {
        const uint32_t wb = acc[i], wc = cnt[i];
        acc[i] = ob;
        cnt[i] = uint16_t(oc);
        ob += wb;
        oc += wc;
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < ASM_EACH; ++e) {
        const uint32_t i = t + e * ASM_THREADS;
        if (i >= m) continue;
        const uint32_t k = key[head[e]];
        const uint64_t at = uint64_t(acc[k]) + a[e];
        DevRecord d;
        d.read_id = ids[i];
        d.is_n = is_n;
        d.strand = 0;
        d.pad = 0;
        d.pos = at;
        rec[uint32_t(cnt[k]) + c[e]] = d;
        place[i] = at;
        tail[i] = nx[i] == ASM_NONE;
    }
    if (t == 0) out[0] = total;
}

// Each member writes its bases (a warp per member).
__global__ void __launch_bounds__(256) place_small_kernel(const uint32_t* __restrict__ ids, uint32_t m,
                                                          const uint64_t* __restrict__ place,
                                                          const uint8_t* __restrict__ tail,
                                                          const uint16_t* __restrict__ offset,
                                                          const uint64_t* __restrict__ db,
                                                          const uint8_t* __restrict__ ascii, int L, int W,
                                                          uint8_t* __restrict__ seq) {
    const uint32_t i = (blockIdx.x * 256 + threadIdx.x) >> 5;
    if (i >= m) return;
    const uint32_t x = ids[i];
    const int nb = tail[i] ? L : offset[x];
    uint8_t* out = seq + place[i];
    for (int j = int(threadIdx.x & 31u); j < nb; j += 32)
        out[j] = ascii ? ascii[uint64_t(x) * L + j] : uint8_t("ACGT"[code_at(db + uint64_t(x) * W, j)]);
}

inline int rounds_for(uint32_t m) {
    int r = 1;
    while ((1ull << r) < uint64_t(m) + 1) ++r;
    return r + 1;
}

// Scratch of one ranking, sized for m members of n reads.
struct RankScratch {
    ChainNode* node;
    SubPos* loc;
    uint8_t* flags;
    uint8_t* promote;
    uint32_t* rul;
    SubTotal* tot;
    RankState* A;
    RankState* B;
    uint32_t epoch;    // walks so far (loc is zeroed once, so 0 is never current)
};

// Ranks every member: st[i] for list index i.  Returns the number of members
// on cycles (jump still set).
uint32_t rank_members(const uint32_t* ids, uint32_t m, uint32_t n, const uint32_t* nx, const uint32_t* pv,
                      const uint16_t* offset, const uint32_t* pos_in_ids, RankScratch& k, RankState* st,
                      Arena& a, cudaStream_t s) {
    const int g = grid_for(m, 256);
    const uint8_t* promote = nullptr;
    uint32_t nr = 0;
    SubStage sp_walk("assembly.walk");
    // per attempt: rulers, unreached, a link out of the set
    uint32_t* counts = a.zeros<uint32_t>(2 * 3, s);
    chain_nodes_kernel<<<resident_grid(chain_nodes_kernel, 256, n), 256, 0, s>>>(n, pos_in_ids, nx, offset, k.node);
    CURC_LAUNCH_CHECK();
    for (int attempt = 0; attempt < 2; ++attempt) {
        const uint32_t epoch = ++k.epoch;
        ruler_flags_kernel<<<g, 256, 0, s>>>(ids, m, pv, promote, k.flags);
        CURC_LAUNCH_CHECK();
        select_flagged(ids, k.flags, k.rul, m, counts, a, s);
        if (attempt) {  // clear the ruler marks of the first attempt
            chain_nodes_kernel<<<resident_grid(chain_nodes_kernel, 256, n), 256, 0, s>>>(n, pos_in_ids, nx, offset,
                                                                                          k.node);
            CURC_LAUNCH_CHECK();
        }
        nr = read_scalar(counts, s);
        ruler_index_kernel<<<grid_for(nr, 256), 256, 0, s>>>(k.rul, nr, k.node);
        CURC_LAUNCH_CHECK();
        ruler_walk_kernel<<<resident_grid(ruler_walk_kernel, 256, nr), 256, 0, s>>>(k.rul, nr, m, n, epoch, k.node,
                                                                                    k.loc, k.tot, counts + 2);
        CURC_LAUNCH_CHECK();
        unreached_kernel<<<resident_grid(unreached_kernel, 256, m), 256, 0, s>>>(m, epoch, k.loc, k.flags,
                                                                                  counts + 1);
        CURC_LAUNCH_CHECK();
        uint32_t hc[3];
        read_small(hc, counts, 12, s);
        counts += 3;
        if (hc[2]) throw std::runtime_error("assemble: a chain link leaves the member set");
        if (hc[1] == 0) break;
        if (attempt == 1) throw std::runtime_error("assemble: reads left unranked after promoting cycle rulers");
        CURC_CHECK(cudaMemsetAsync(k.promote, 0, m, s));
        promote_kernel<<<g, 256, 0, s>>>(ids, m, n, k.flags, nx, pos_in_ids, k.promote);
        CURC_LAUNCH_CHECK();
        promote = k.promote;
    }
    sp_walk.stop();
    SubStage sp_jump("assembly.jump");
    ruler_init_kernel<<<grid_for(nr, 256), 256, 0, s>>>(k.rul, nr, m, pv, pos_in_ids, k.loc, k.tot, k.A);
    CURC_LAUNCH_CHECK();
    const int R = rounds_for(nr);
    uint32_t* active = a.zeros<uint32_t>(R, s);  // per round
    uint32_t* done = a.zeros<uint32_t>(2, s);
    if (nr <= RANK_CLUSTER) {
        launch_cluster(rank_rounds_kernel, RANK_BLOCKS, 512, s, nr, k.A, k.B, uint32_t(R), active, done);
        member_state_kernel<<<g, 256, 0, s>>>(m, k.rul, k.loc, k.A, k.B, done, st);
        CURC_LAUNCH_CHECK();
        return read_scalar(done, s);
    }
    RankState* A = k.A;
    RankState* B = k.B;
    uint32_t left = 0;
    // the count of pointers left is read every few rounds (a round on
    // converged states changes nothing)
    const int gs = resident_grid(rank_step_kernel, 512, nr);
    for (int t = 0; t < R; ++t) {
        rank_step_kernel<<<gs, 512, 0, s>>>(nr, A, B, active + t);
        CURC_LAUNCH_CHECK();
        std::swap(A, B);
        if (t % 4 != 3 && t + 1 < R) continue;
        left = read_scalar(active + t, s);
        if (left == 0) break;
    }
    member_state_kernel<<<g, 256, 0, s>>>(m, k.rul, k.loc, A, A, done, st);
    CURC_LAUNCH_CHECK();
    return left;
}

}  // namespace

void pack_ascii_ref(const uint8_t* seq, uint64_t len, uint64_t* packed, cudaStream_t s) {
    const uint64_t words = (len + 31) / 32 + 1;
    pack_ref_kernel<<<grid_for(words, 256), 256, 0, s>>>(seq, len, packed, words);
    CURC_LAUNCH_CHECK();
}

namespace {
void assemble_small(const uint64_t* db, const uint8_t* ascii, int L, int W, const uint32_t* ids, uint32_t m,
                    uint32_t n, const uint32_t* next, const uint32_t* prev, const uint16_t* offset, bool is_n,
                    uint32_t* pos_in_ids, Assembled& out, Arena& a, cudaStream_t s) {
    SubStage sp("assembly.small");
    static std::mutex mu;
    static bool done[64] = {};
    int dev = 0;
    CURC_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) throw std::runtime_error("device ordinal out of range");
    {
        std::lock_guard<std::mutex> g(mu);
        if (!done[dev]) {
            CURC_CHECK(cudaFuncSetAttribute(assemble_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            int(asm_small_bytes(ASM_SMALL))));
            done[dev] = true;
        }
    }
    uint64_t* place = a.alloc<uint64_t>(m);
    uint8_t* tail = a.alloc<uint8_t>(m);
    uint64_t* res = a.zeros<uint64_t>(2, s);  // bases, error
    assemble_small_kernel<<<1, ASM_THREADS, asm_small_bytes(m), s>>>(ids, m, n, next, prev, offset, L, is_n ? 1 : 0,
                                                                     pos_in_ids, out.records, place, tail, res,
                                                                     reinterpret_cast<uint32_t*>(res + 1));
    CURC_LAUNCH_CHECK();
    uint64_t h[2];
    read_small(h, res, 16, s);
    if (uint32_t(h[1]) == 1) throw std::runtime_error("assemble: a chain link leaves the member set");
    if (h[1]) throw std::runtime_error("assemble: unresolved chain links after cutting cycles");
    out.len = h[0];
    out.seq = a.alloc<uint8_t>(out.len + 64);
    place_small_kernel<<<grid_for(uint64_t(m) * 32, 256), 256, 0, s>>>(ids, m, place, tail, offset, db, ascii, L, W,
                                                                       out.seq);
    CURC_LAUNCH_CHECK();
    out.packed = a.alloc<uint64_t>((out.len + 31) / 32 + 1);
    pack_ascii_ref(out.seq, out.len, out.packed, s);
}
}  // namespace

void assemble(const uint64_t* db, const uint8_t* ascii, int L, int W, const uint32_t* ids, uint32_t m,
              uint32_t n_total, const uint32_t* next, const uint32_t* prev, const uint16_t* offset, bool is_n,
              Assembled& out, Arena& a, cudaStream_t s) {
    out.n_records = m;
    out.records = a.alloc<DevRecord>(m ? m : 1);
    if (m == 0) {
        out.len = 0;
        out.seq = a.alloc<uint8_t>(1);
        out.packed = a.alloc<uint64_t>(1);
        CURC_CHECK(cudaMemsetAsync(out.packed, 0, 8, s));
        return;
    }
    const size_t n = n_total;
    uint32_t* pos_in_ids = a.alloc<uint32_t>(n);
    if (m <= ASM_SMALL) {
        assemble_small(db, ascii, L, W, ids, m, n_total, next, prev, offset, is_n, pos_in_ids, out, a, s);
        return;
    }
    uint32_t* nx = a.alloc<uint32_t>(n);
    uint32_t* pv = a.alloc<uint32_t>(n);
    CURC_CHECK(cudaMemcpyAsync(nx, next, n * 4, cudaMemcpyDeviceToDevice, s));
    CURC_CHECK(cudaMemcpyAsync(pv, prev, n * 4, cudaMemcpyDeviceToDevice, s));
    const int g = grid_for(m, 256);
    fill<uint32_t>(pos_in_ids, INVALID, n, s);
    scatter_index_kernel<<<g, 256, 0, s>>>(ids, m, pos_in_ids);
    CURC_LAUNCH_CHECK();
    SubStage sp_rank("assembly.ranking");
    RankScratch k;
    k.node = a.alloc<ChainNode>(n);
    k.loc = a.zeros<SubPos>(m, s);
    k.epoch = 0;
    k.flags = a.alloc<uint8_t>(m);
    k.promote = a.alloc<uint8_t>(m);
    k.rul = a.alloc<uint32_t>(m);
    k.tot = a.alloc<SubTotal>(m);
    k.A = a.alloc<RankState>(m);
    k.B = a.alloc<RankState>(m);
    RankState* R = a.alloc<RankState>(m);
    uint32_t left = rank_members(ids, m, n_total, nx, pv, offset, pos_in_ids, k, R, a, s);
    if (left) {
        // Cycles: cut each in parallel.  Only their members are ranked again
        // (a cut cycle is a chain of exactly its members), as a list of its
        // own in list order, and their states are then written back.
        uint8_t* cyc = a.alloc<uint8_t>(m);
        cycle_flags_kernel<<<g, 256, 0, s>>>(m, R, cyc);
        CURC_LAUNCH_CHECK();
        uint32_t* leader_of_head = a.alloc<uint32_t>(n);
        unsigned long long* best = a.alloc<unsigned long long>(n);
        CURC_CHECK(cudaMemsetAsync(best, 0, n * sizeof(unsigned long long), s));
        uint32_t* cut = a.zeros<uint32_t>(2, s);  // members on cycles, a cycle that does not close
        cycle_open_kernel<<<g, 256, 0, s>>>(ids, m, R, cyc, nx, pv, leader_of_head, cut + 1);
        CURC_LAUNCH_CHECK();
        uint32_t* cidx = a.alloc<uint32_t>(m);
        select_indices(cyc, cidx, m, cut, a, s);
        uint32_t hc[2];
        read_small(hc, cut, 8, s);
        if (hc[1]) throw std::runtime_error("assemble: broken cycle");
        const uint32_t mc = hc[0];
        const int gc = grid_for(mc, 256);
        uint32_t* cids = a.alloc<uint32_t>(mc);
        uint32_t* pos_in_cyc = a.alloc<uint32_t>(n);
        fill<uint32_t>(pos_in_cyc, INVALID, n, s);
        cycle_list_kernel<<<gc, 256, 0, s>>>(ids, cidx, mc, cids, pos_in_cyc);
        CURC_LAUNCH_CHECK();
        uint8_t* all = a.alloc<uint8_t>(mc);
        CURC_CHECK(cudaMemsetAsync(all, 1, mc, s));
        RankScratch kc;
        kc.node = k.node;
        kc.loc = a.zeros<SubPos>(mc, s);
        kc.epoch = 0;
        kc.flags = a.alloc<uint8_t>(mc);
        kc.promote = a.alloc<uint8_t>(mc);
        kc.rul = a.alloc<uint32_t>(mc);
        kc.tot = a.alloc<SubTotal>(mc);
        kc.A = a.alloc<RankState>(mc);
        kc.B = a.alloc<RankState>(mc);
        RankState* T = a.alloc<RankState>(mc);
        if (rank_members(cids, mc, n_total, nx, pv, offset, pos_in_cyc, kc, T, a, s))
            throw std::runtime_error("assemble: cycle still closed after its temporary cut");
        cycle_max_kernel<<<gc, 256, 0, s>>>(cids, mc, T, all, offset, best);
        CURC_LAUNCH_CHECK();
        cycle_cut_kernel<<<gc, 256, 0, s>>>(cids, mc, T, all, best, leader_of_head, nx, pv);
        CURC_LAUNCH_CHECK();
        if (rank_members(cids, mc, n_total, nx, pv, offset, pos_in_cyc, kc, T, a, s))
            throw std::runtime_error("assemble: unresolved chain links after cutting cycles");
        cycle_merge_kernel<<<gc, 256, 0, s>>>(cidx, mc, T, R);
        CURC_LAUNCH_CHECK();
    }
    sp_rank.stop();
    SubStage sp_place("assembly.order_place");
    // chain order: first member in list order
    uint32_t* key = a.alloc<uint32_t>(n);
    chain_key_kernel<<<g, 256, 0, s>>>(ids, m, nx, R, key);
    CURC_LAUNCH_CHECK();
    uint8_t* hf = a.alloc<uint8_t>(m);
    head_flags_kernel<<<g, 256, 0, s>>>(ids, m, pv, hf);
    CURC_LAUNCH_CHECK();
    uint32_t* heads = a.alloc<uint32_t>(m);
    uint32_t* cnt = a.alloc<uint32_t>(2);
    select_flagged(ids, hf, heads, m, cnt, a, s);
    const uint32_t nh = read_scalar(cnt, s);
    uint32_t* hkey = a.alloc<uint32_t>(nh);
    gather_heads_kernel<<<grid_for(nh, 256), 256, 0, s>>>(heads, nh, key, hkey);
    CURC_LAUNCH_CHECK();
    int key_bits = 1;  // a key is a list index
    while (key_bits < 32 && (1ull << key_bits) < m) ++key_bits;
    radix_sort_pairs<uint32_t, uint32_t>(hkey, heads, nh, 0, key_bits, a, s);
    uint64_t* chain_bases = a.alloc<uint64_t>(n);
    uint32_t* chain_members = a.alloc<uint32_t>(n);
    tail_sizes_kernel<<<g, 256, 0, s>>>(ids, m, nx, R, L, chain_bases, chain_members);
    CURC_LAUNCH_CHECK();
    uint64_t* cpos = a.alloc<uint64_t>(nh + 1);
    uint32_t* crec = a.alloc<uint32_t>(nh + 1);
    uint32_t* slot = a.alloc<uint32_t>(n);
    chain_sizes_sorted_kernel<<<grid_for(nh, 256), 256, 0, s>>>(heads, nh, chain_bases, chain_members, cpos, crec,
                                                                 slot);
    CURC_LAUNCH_CHECK();
    uint64_t* total = a.alloc<uint64_t>(1);
    exclusive_scan<uint64_t>(cpos, cpos, nh, total, a, s);
    exclusive_scan<uint32_t>(crec, crec, nh, cnt + 1, a, s);
    out.len = read_scalar(total, s);
    out.seq = a.alloc<uint8_t>(out.len + 64);
    place_kernel<<<g, 256, 0, s>>>(ids, m, nx, R, slot, cpos, crec, offset, db, ascii, L, W, is_n ? 1 : 0,
                                   out.records, out.seq);
    CURC_LAUNCH_CHECK();
    out.packed = a.alloc<uint64_t>((out.len + 31) / 32 + 1);
    pack_ascii_ref(out.seq, out.len, out.packed, s);
}

}  // namespace curc
