// A run that fails behind the emission of the streams leaves none of them
// named, and the next run is a whole one.  Linked with libcurc_b200.so.  The
// failure is the arena's: its scratch ends 256 bytes before the run's largest
// need (which unrelated reads have in their unmapped pseudogenome), and a
// chunk larger than the device is what it asks for next.
#include <cstdio>
#include <random>
#include <map>
#include <memory>
#include <string>
#include <vector>
#include <future>

#define private public
#include "../../curc_b200/csrc/block.cuh"
#undef private

using namespace curc;

int main() {
    const uint32_t n = 30000;
    const int L = 250;
    std::mt19937 rng(3);
    std::vector<uint8_t> reads(size_t(n) * L);
    for (auto& c : reads) c = "ACGT"[rng() & 3u];
    uint8_t* d = nullptr;
    CURC_CHECK(cudaMalloc(&d, reads.size() + 16));
    CURC_CHECK(cudaMemcpy(d, reads.data(), reads.size(), cudaMemcpyHostToDevice));
    Block b;
    b.run(d, n, L, false, false);
    std::map<std::string, std::vector<uint8_t>> want;
    for (const auto& h : b.host) want[h.first].assign(h.second.ptr, h.second.ptr + h.second.size);
    const size_t need = b.arena.high_water();
    if (b.arena.chunks_.size() != 1) return std::printf("more than one chunk\n"), 1;

    b.arena.reset();
    b.arena.chunk_ = size_t(1) << 50;
    b.arena.alloc_bytes(b.arena.chunks_[0].size - need + 256);
    b.off_all = nullptr;
    bool threw = false;
    try {
        b.run(d, n, L, false, false);
    } catch (const CudaError&) {
        threw = true;
    }
    int bad = 0;
    if (!threw || !b.off_all) {
        std::printf("the run did not fail behind the streams' emission\n");
        ++bad;
    }
    for (const char* nm : {"strand", "mis_cnt", "mis_base", "read_off", "decoder_table", "mis_off_1", "ref", "sizes"})
        if (b.host.count(nm)) {
            std::printf("%s is named after a failed run\n", nm);
            ++bad;
        }
    for (const char* nm : {"packed", "sorted_ids", "next", "map_mm"})  // complete when it failed
        if (!b.host.count(nm) || want[nm] != std::vector<uint8_t>(b.host[nm].ptr, b.host[nm].ptr + b.host[nm].size)) {
            std::printf("%s is missing or differs\n", nm);
            ++bad;
        }

    b.arena.chunk_ = size_t(1) << 30;
    b.arena.reset();
    b.run(d, n, L, false, false);
    for (const auto& h : want)
        if (!b.host.count(h.first) ||
            (h.first != "stats" &&
             h.second != std::vector<uint8_t>(b.host[h.first].ptr, b.host[h.first].ptr + b.host[h.first].size))) {
            std::printf("%s differs in the next run\n", h.first.c_str());
            ++bad;
        }
    std::printf("%s\n", bad ? "FAILED" : "all equal");
    return bad != 0;
}
