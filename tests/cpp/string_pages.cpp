// floor_plan (csrc/string_pages.h): whatever the rows' order, its pages are the ones that the rows' places take, each with
// a row at least and no more than it holds.
#include "string_pages.h"

#include <algorithm>
#include <cstdio>
#include <random>
#include <vector>

int main() {
    std::mt19937_64 rng(1);
    long ambiguous = 0, plans = 0;
    for (int round = 0; round < 4000; round++) {
        const uint64_t longest = 1 + rng() % (round % 3 ? 8187 : 600);
        std::vector<uint64_t> cost(1 + rng() % (round % 10 ? 400 : 20000));
        for (uint64_t& c : cost) c = rng() % 4 ? 1 + rng() % longest : rng() % 2 ? longest : 1;
        uint64_t total = 0, maxc = 0;
        for (uint64_t c : cost) total += c, maxc = std::max(maxc, c);
        const bj::FloorPlan p = bj::floor_plan(total, maxc);
        if (!p.pages) {
            std::printf("no plan for %lu of at most %lu\n", (unsigned long)total, (unsigned long)maxc);
            return 1;
        }
        plans++;
        uint64_t fewest = ~0ull, most = 0;  // pages of a packing by the highest cp, for comparison
        for (int order = 0; order < 6; order++) {
            if (order == 1) std::sort(cost.begin(), cost.end());
            else if (order == 2) std::sort(cost.rbegin(), cost.rend());
            else std::shuffle(cost.begin(), cost.end(), rng);
            uint64_t at = 0, page = 0, held = 0;
            for (size_t i = 0; i < cost.size(); at += cost[i++]) {
                const uint64_t pg = at / p.cp;
                if (pg != page) {
                    if (pg != page + 1 || held == 0) {
                        std::printf("page %lu without a row\n", (unsigned long)page + 1);
                        return 1;
                    }
                    page = pg;
                    held = 0;
                }
                held += cost[i];
                if (held > bj::kStrPageUnits) {
                    std::printf("a page of %lu units\n", (unsigned long)held);
                    return 1;
                }
            }
            if (page + 1 != p.pages) {
                std::printf("%lu pages in one order, %lu planned\n", (unsigned long)page + 1, (unsigned long)p.pages);
                return 1;
            }
            const uint64_t plain = (total - cost.back()) / (bj::kStrPageUnits - maxc) + 1;
            fewest = std::min(fewest, plain);
            most = std::max(most, plain);
        }
        ambiguous += fewest != most;
        if (p.pages > 2 * (total / bj::kStrPageUnits) + 2) {
            std::printf("%lu pages for %lu units\n", (unsigned long)p.pages, (unsigned long)total);
            return 1;
        }
    }
    if (!ambiguous) {
        std::puts("no set of rows whose pages depend on their order was tried");
        return 1;
    }
    // Large results: a plan is found at once.
    for (uint64_t total : {uint64_t(1) << 32, (uint64_t(1) << 36) + 12345, uint64_t(1) << 45})
        for (uint64_t maxc : {uint64_t(1), uint64_t(300), uint64_t(8187)})
            for (uint64_t more = 0; more < 70000; more += 17) {
                const bj::FloorPlan p = bj::floor_plan(total + more, maxc);
                if (!p.pages || (total + more - maxc) / p.cp + 1 != p.pages || (total + more - 1) / p.cp + 1 != p.pages) {
                    std::printf("total %lu longest %lu: %lu pages of %lu\n", (unsigned long)(total + more),
                                (unsigned long)maxc, (unsigned long)p.pages, (unsigned long)p.cp);
                    return 1;
                }
            }
    std::printf("ok: %ld of %ld sets of rows have pages that depend on their order\n", ambiguous, plans);
    return 0;
}
