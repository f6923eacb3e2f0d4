// The kernels that run as one cluster, with 1 to 16 blocks: the walk over
// meetings and the ruler ranking give the same with each.
#include <cstdio>
#include <random>

#include "../../curc_b200/csrc/assembly.cu"
#include "../../curc_b200/csrc/primitives.cu"
#include "../../curc_b200/csrc/walk.cuh"

using namespace curc;

namespace check {
cudaStream_t s;
std::mt19937_64 rng(9);
int bad = 0;

template <class T>
T* up(Arena& a, const std::vector<T>& v) {
    T* d = a.alloc<T>(v.size() + 1);
    CURC_CHECK(cudaMemcpyAsync(d, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, s));
    CURC_CHECK(cudaStreamSynchronize(s));
    return d;
}
template <class T>
std::vector<T> down(const T* d, size_t n) {
    std::vector<T> v(n);
    CURC_CHECK(cudaMemcpyAsync(v.data(), d, n * sizeof(T), cudaMemcpyDeviceToHost, s));
    CURC_CHECK(cudaStreamSynchronize(s));
    return v;
}

void walks(Arena& a, uint32_t reads, int noffs, uint32_t per_off, bool ahead) {
    std::vector<Meeting> item;
    std::vector<uint32_t> start{0}, pre(reads);
    for (uint32_t i = 0; i < reads; ++i) pre[i] = i;
    std::shuffle(pre.begin(), pre.end(), rng);
    for (int o = 0; o < noffs; ++o) {
        // runs of prefixes one behind the other, each met by suffixes of its own
        std::vector<uint32_t> suf(reads);
        for (uint32_t i = 0; i < reads; ++i) suf[i] = i;
        std::shuffle(suf.begin(), suf.end(), rng);
        size_t si = 0;
        for (uint32_t lo = 0; lo < reads && item.size() < start.back() + per_off;) {
            const uint32_t hi = std::min<uint32_t>(reads, lo + 1 + rng() % (rng() % 8 ? 3 : 70));
            for (size_t k = 1 + rng() % (rng() % 8 ? 3 : 70); k > 0 && si < suf.size(); --k)
                item.push_back(Meeting{suf[si++], lo, hi, pre[lo]});
            lo = hi;
        }
        start.push_back(uint32_t(item.size()));
    }
    Meeting* di = up(a, item);
    uint32_t* ds = up(a, start);
    uint32_t* dp = up(a, pre);
    unsigned long long* used = up(a, std::vector<unsigned long long>{0});
    std::vector<uint32_t> wn, wp;
    std::vector<uint16_t> wo;
    for (unsigned blocks : {1u, 2u, 4u, 8u, 16u}) {
        uint32_t* nx = up(a, std::vector<uint32_t>(reads, INVALID));
        uint32_t* pv = up(a, std::vector<uint32_t>(reads, INVALID));
        uint16_t* of = up(a, std::vector<uint16_t>(reads, INVALOFF));
        launch_cluster(ahead ? walk_kernel<true, false> : walk_kernel<false, false>, blocks, WALK_THREADS, s, di, ds, 1, noffs, dp,
                       used, 1u, nx, pv, of, nullptr);
        const auto n = down(nx, reads), p = down(pv, reads);
        const auto o = down(of, reads);
        if (wn.empty()) {
            wn = n;
            wp = p;
            wo = o;
        }
        if (n != wn || p != wp || o != wo) {
            std::printf("walk of %u reads differs with %u blocks\n", reads, blocks);
            ++bad;
        }
    }
}

void ranks(Arena& a, uint32_t n) {
    std::vector<uint32_t> ord(n);
    for (uint32_t i = 0; i < n; ++i) ord[i] = i;
    std::shuffle(ord.begin(), ord.end(), rng);
    std::vector<RankState> st(n);
    std::vector<uint64_t> want(n);
    for (uint32_t k = 0, head = 0; k < n; ++k) {  // lists of up to 5,000, in shuffled order
        if (k % 5000 == 0) head = k;
        RankState r = {};
        const uint32_t prev = k == head ? INVALID : ord[k - 1];
        r.jump = prev;
        r.far = prev == INVALID ? ord[k] : prev;
        r.cnt = prev != INVALID;
        r.acc = prev == INVALID ? 0 : prev % 7;
        r.mn = ord[k];
        st[ord[k]] = r;
        want[ord[k]] = k == head ? 0 : want[ord[k - 1]] + ord[k - 1] % 7;
    }
    const int rounds = rounds_for(n);
    for (unsigned blocks : {1u, 2u, 4u, 8u, 16u}) {
        RankState* A = up(a, st);
        RankState* B = a.alloc<RankState>(n);
        uint32_t* active = up(a, std::vector<uint32_t>(rounds, 0));
        uint32_t* done = up(a, std::vector<uint32_t>(2, 0));
        launch_cluster(rank_rounds_kernel, blocks, 512, s, n, A, B, uint32_t(rounds), active, done);
        const auto d = down(done, 2);
        const auto r = down(d[1] & 1 ? B : A, n);
        bool ok = d[0] == 0;
        for (uint32_t i = 0; i < n; ++i) ok &= r[i].jump == INVALID && r[i].acc == want[i];
        if (!ok) {
            std::printf("ranking of %u differs with %u blocks\n", n, blocks);
            ++bad;
        }
    }
}
}  // namespace check

int main() {
    using namespace check;
    for (unsigned held = 1; held <= 16; ++held) {
        const unsigned b = cluster_fit(16, held);
        if (b > held || 2 * b <= held || cluster_fit(1, held) != 1) ++bad;
    }
    CURC_CHECK(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    Arena a(size_t(256) << 20);
    for (bool ahead : {false, true}) {
        walks(a, 900, 40, 100, ahead);
        walks(a, 20000, 70, 9000, ahead);
    }
    ranks(a, 3);
    ranks(a, 20000);
    ranks(a, 65536);
    std::printf("%s\n", bad ? "FAILED" : "all equal");
    return bad != 0;
}
