// Which draw an item (a triangle, a varying record) belongs to: plain C++, for the kernels,
// for the host that builds the tables and for the CPU test.
#pragma once

#include <stdint.h>

#include <vector>

#ifdef __CUDACC__
#define RZ_HD __host__ __device__ __forceinline__
#else
#define RZ_HD inline
#endif

namespace rz {

constexpr int kDrawTableShift = 8;  // a table entry for every 256th item

// The last draw of [lo, hi] whose first item, base(draw), is at most `at`; draws are in the
// order of their first items, and draw lo starts at or before `at`.
template <class Base>
RZ_HD uint32_t draw_between(uint32_t lo, uint32_t hi, uint32_t at, Base base) {
    while (lo < hi) {
        const uint32_t mid = lo + (hi - lo + 1) / 2;
        if (base(mid) <= at) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Item `at`'s draw from the table of its list: the draw lies between its entry and the next
// one, so that one draw for all 256 items costs no further load, two cost one, and n draws
// log2 n in a chain. 640x360, 131,072 triangles of a few pixels, in draws of 1, 4 and 64:
// 125, 89 and 79 us a frame with a search of all the draws, 255, 101 and 65 with a walk from
// the entry, 107, 75 and 65 so.
template <class Entry, class Base>
RZ_HD uint32_t draw_in_table(uint32_t at, Entry entry, Base base) {
    const uint32_t g = at >> kDrawTableShift;
    return draw_between(entry(g), entry(g + 1), at, base);
}

// Appends the table of n draws of `end` items to `out`: entry g is the last draw that starts
// at or before item 256 g, and one entry past the last item is the last draw.
template <class Base>
inline void add_draw_table(std::vector<uint32_t>& out, uint32_t n, uint64_t end, Base base) {
    uint32_t d = 0;
    for (uint64_t at = 0;; at += 1u << kDrawTableShift) {
        while (d + 1 < n && base(d + 1) <= at) ++d;
        out.push_back(d);
        if (at >= end) return;
    }
}

}  // namespace rz
