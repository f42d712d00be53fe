// Counts the queue entries that one step of a persistent traversal leaves, warp by warp as the kernels do,
// for a given split of its pieces over phases, CTAs and appends.
//   queue_bound V E ctas seed keep few phase...      phase: appends:pieces_per_append
// Appends go to warps at random (few = 1: a third of them to a few CTAs).  keep = 1: a warp's open block lasts until the step's last phase, as in
// the kernels; 0: it is closed at the end of each.  Prints "used reserved pieces".
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "eg_queue.cuh"

int main(int argc, char** argv) {
    using namespace eg;
    if (argc < 8) return 2;
    const uint64_t V = strtoull(argv[1], nullptr, 10), E = strtoull(argv[2], nullptr, 10);
    const uint64_t ctas = strtoull(argv[3], nullptr, 10);
    std::mt19937_64 rng(strtoull(argv[4], nullptr, 10));
    const bool keep = atoi(argv[5]) != 0, few = atoi(argv[6]) != 0;
    const uint64_t warps_per_cta = kPersistThreads / 32, warps = ctas * warps_per_cta;
    std::vector<WarpBlock> wb(warps);
    std::vector<uint64_t> reserved(ctas), filled(ctas);
    uint64_t used = 0, pieces = 0;
    for (int a = 7; a < argc; ++a) {
        unsigned long long appends = 0, per = 0;
        if (sscanf(argv[a], "%llu:%llu", &appends, &per) != 2) return 2;
        std::fill(reserved.begin(), reserved.end(), 0);
        std::fill(filled.begin(), filled.end(), ~0ull);
        for (uint64_t i = 0; i < appends; ++i) {
            const uint64_t w = rng() % (few && i % 3 == 0 ? (warps + 63) / 64 : warps), c = w / warps_per_cta;
            pieces += per;
            if (filled[c] == ~0ull) {  // the CTA's shared queue has not overflowed yet
                const uint64_t at = reserved[c];
                reserved[c] += per;
                if (at + per <= kLocalQueue) continue;
                filled[c] = at;
            }
            const uint32_t block = wb[w].wants((uint32_t)per);
            wb[w].took((uint32_t)per, (uint32_t)used, block);
            used += block;
        }
        for (uint64_t c = 0; c < ctas; ++c) used += reserved[c] < filled[c] ? reserved[c] : filled[c];
        for (auto& b : wb) b.phase_done(!keep || a == argc - 1);
    }
    printf("%llu %llu %llu\n", (unsigned long long)used, (unsigned long long)queue_entries(V, E, ctas),
           (unsigned long long)pieces);
    return 0;
}
