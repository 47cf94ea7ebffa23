// Whatever number of a launch's blocks is resident (the others never start, or
// start when the work is gone), its warps claim every seed exactly once by the
// rule of seed_claim.h, and a resident grid deals its first seeds evenly.
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>

#include "seed_claim.h"

int main() {
    for (uint32_t blocks : {1u, 3u, 37u, 592u})
        for (uint32_t warps : {1u, 8u})
            for (uint32_t total : {0u, 1u, blocks - 1, blocks, blocks + 1, 2 * blocks + 1, blocks * warps - 1,
                                   blocks * warps, blocks * warps + 1, 5 * blocks * warps + 7})
                for (uint32_t resident : {1u, (blocks + 1) / 2, blocks})
                    for (bool patient : {false, true}) {
                        std::atomic<uint32_t> counter[2] = {};
                        std::vector<std::atomic<int>> taken(total);
                        for (auto& t : taken) t = 0;
                        std::atomic<uint32_t> most{0};
                        auto add = [&](uint32_t i, uint32_t n) { return counter[i].fetch_add(n); };
                        auto peek = [&](uint32_t i) { return counter[i].load(); };
                        std::vector<uint32_t> row(resident);
                        for (auto& r : row) r = add(1, 1);
                        auto run = [&](uint32_t b0, uint32_t b1, const std::vector<uint32_t>& rows) {
                            std::vector<uint32_t> from((b1 - b0) * warps, cgb::kSeedFirst), own((b1 - b0) * warps);
                            for (bool any = true; any;) {  // the warps take turns, a seed each
                                any = false;
                                for (uint32_t k = 0; k < from.size(); ++k) {
                                    if (from[k] == cgb::kSeedLater) {  // the wait is over
                                        from[k] = peek(1) < blocks ? cgb::kSeedNext : cgb::kSeedNone;
                                        any = true;
                                    }
                                    if (from[k] > cgb::kSeedNext) continue;
                                    const uint32_t first = from[k] == cgb::kSeedFirst;
                                    const uint32_t s = cgb::seed_claim(from[k], own[k], rows[b0 + k / warps], k % warps, total,
                                                                       blocks, warps, patient, add, peek);
                                    if (s >= total) continue;
                                    any = true;
                                    ++taken[s];
                                    if (first && s >= blocks * warps) ++most;
                                }
                            }
                        };
                        std::thread t1([&] { run(0, resident / 2, row); }), t2([&] { run(resident / 2, resident, row); });
                        t1.join();
                        t2.join();
                        std::vector<uint32_t> late(1, add(1, 1));  // a block that starts after all that
                        run(0, 1, late);
                        bool ok = most == 0;
                        for (auto& t : taken) ok &= t == 1;
                        if (!ok) {
                            std::printf("blocks %u warps %u total %u resident %u\n", blocks, warps, total, resident);
                            return 1;
                        }
                    }
    std::puts("ok");
}
