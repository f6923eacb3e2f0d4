// The one-launch scan, selection, sort and compaction against the standard
// library, built with CURC_LOOK_SPINS: with 0 a tile never waits for the tiles
// before it and counts what they have not published itself.
#include <algorithm>
#include <cstdio>
#include <numeric>
#include <random>

#include "../../curc_b200/csrc/compact.cuh"
#include "../../curc_b200/csrc/primitives.cu"

using namespace curc;

namespace check {
cudaStream_t s;
int bad = 0;
std::mt19937_64 rng(5);

template <class T>
T* up(Arena& a, const std::vector<T>& v) {
    T* d = a.alloc<T>(v.size() + 1);
    CURC_CHECK(cudaMemcpyAsync(d, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, s));
    return d;
}
template <class T>
std::vector<T> down(const T* d, size_t n) {
    std::vector<T> v(n);
    CURC_CHECK(cudaMemcpyAsync(v.data(), d, n * sizeof(T), cudaMemcpyDeviceToHost, s));
    CURC_CHECK(cudaStreamSynchronize(s));
    return v;
}
void expect(bool ok, const char* what, size_t n) {
    if (!ok) std::printf("differs: %s, %zu items\n", what, n);
    bad += !ok;
}

template <class T>
void scans(Arena& a, size_t n) {
    std::vector<T> in(n), want(n);
    for (auto& x : in) x = T(rng() % 1000);
    T sum = 0;
    for (size_t i = 0; i < n; ++i) {
        want[i] = sum;
        sum += in[i];
    }
    T* d = up(a, in);
    T* o = a.alloc<T>(n);
    T* tot = a.alloc<T>(2);
    exclusive_scan<T>(d, o, n, tot, a, s);
    expect(down(o, n) == want && down(tot, 1)[0] == sum, "scan", n);
    exclusive_scan<T>(d, d, n, tot + 1, a, s);
    expect(down(d, n) == want && down(tot + 1, 1)[0] == sum, "scan in place", n);
}

struct Odd {
    const uint32_t* v;
    __device__ bool operator()(uint32_t i) const { return v[i] & 1u; }
};
struct Put {
    const uint32_t* v;
    uint32_t* o;
    __device__ void operator()(uint32_t i, uint32_t d) const { o[d] = v[i]; }
};

void picks(Arena& a, size_t n) {
    std::vector<uint32_t> in(n), want, idx;
    std::vector<uint8_t> fl(n);
    for (size_t i = 0; i < n; ++i) {
        in[i] = uint32_t(rng());
        fl[i] = in[i] & 1u;
        if (fl[i]) {
            want.push_back(in[i]);
            idx.push_back(uint32_t(i));
        }
    }
    uint32_t* d = up(a, in);
    uint8_t* f = up(a, fl);
    uint32_t* o = a.alloc<uint32_t>(n);
    uint32_t* c = up(a, std::vector<uint32_t>{uint32_t(n), 0, 0, 0, 0});
    select_flagged<uint32_t>(d, f, o, n, c + 1, a, s);
    expect(down(o, want.size()) == want, "select", n);
    select_indices(f, o, n, c + 2, a, s);
    expect(down(o, want.size()) == idx, "select indices", n);
    Compactor cp(uint32_t(n), a, s);
    for (int k = 0; k < 2; ++k) {  // states of two launches
        cp.run(c, uint32_t(n), c + 3 + k, Odd{d}, Put{d, o});
        expect(down(o, want.size()) == want, "compaction", n);
    }
    const auto h = down(c, 5);
    expect(std::all_of(h.begin() + 1, h.end(), [&](uint32_t x) { return x == want.size(); }), "counts", n);
}

template <class K, class V>
void sorts(Arena& a, size_t n, int begin, int end) {
    std::vector<K> k(n);
    std::vector<V> v(n);
    std::vector<uint32_t> ord(n);
    for (size_t i = 0; i < n; ++i) {
        k[i] = i % 3 ? K(rng()) : K(rng() % 7);
        v[i] = V(i);
    }
    std::iota(ord.begin(), ord.end(), 0u);
    auto bits = [&](K x) { return uint64_t(x) << (64 - end) >> (64 - end + begin); };
    std::stable_sort(ord.begin(), ord.end(), [&](uint32_t x, uint32_t y) { return bits(k[x]) < bits(k[y]); });
    K* dk = up(a, k);
    V* dv = up(a, v);
    radix_sort_pairs<K, V>(dk, dv, n, begin, end, a, s);
    const auto rk = down(dk, n);
    const auto rv = down(dv, n);
    bool ok = true;
    for (size_t i = 0; i < n; ++i) ok &= rk[i] == k[ord[i]] && rv[i] == V(ord[i]);
    expect(ok, "sort", n);
}
}  // namespace check

int main() {
    using namespace check;
    CURC_CHECK(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    Arena a(size_t(256) << 20);
    for (size_t n : {size_t(1), size_t(4096), size_t(4097), size_t(133 * 4096), size_t(1000003)}) {
        a.reset();
        a.clear_zeros(s);
        scans<uint32_t>(a, n);
        scans<uint64_t>(a, n);
        picks(a, n);
        sorts<uint64_t, uint32_t>(a, n, 0, 64);
        sorts<uint32_t, uint32_t>(a, n, 3, 24);
        sorts<uint64_t, uint64_t>(a, n, 0, 9);
    }
    std::printf("%s\n", bad ? "FAILED" : "all equal");
    return bad != 0;
}
