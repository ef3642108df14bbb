// How many pages the strings of a result column take when they are packed by
// their costs' prefix sums (k_output.cu, "floor packing").
#pragma once

#include <cstdint>

namespace bj {

constexpr uint64_t kStrPageUnits = 65496;  // eighth-bytes a page may hold

struct FloorPlan {
    uint64_t cp = 0;     // row i lies on page start_i / cp
    uint64_t pages = 0;  // 0: the rows are packed one by one instead
};

// For rows of costs 1 to maxc, `total` together, in whatever order: rows of a
// join come in no particular one, and a captured query, whose page count is that
// of its recording, runs in another each time. The last row begins somewhere in
// [total - maxc, total - 1]: cp is chosen so that this lies on one page. (Every
// page has a row, as cp > maxc, and no more than it holds, as cp + maxc is at
// most that.)
inline FloorPlan floor_plan(uint64_t total, uint64_t maxc) {
    if (total == 0) return {};
    uint64_t cp = kStrPageUnits - maxc;
    while (cp > kStrPageUnits / 2) {
        const uint64_t last = (total - 1) / cp;
        if ((total - maxc) / cp == last) return {cp, last + 1};
        cp = (total - maxc) / last;  // the largest that brings the page's first unit to total - maxc or below
    }
    return {};
}

} // namespace bj
