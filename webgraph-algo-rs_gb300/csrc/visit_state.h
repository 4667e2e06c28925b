// What a breadth-first visit carries from level to level (visit_level.cuh);
// plain C++ where no CUDA compiler reads it.
#pragma once
#include <algorithm>
#include <cstdint>

#ifdef __CUDACC__
#define HBL_BOTH __host__ __device__ __forceinline__
#else
#define HBL_BOTH inline
#endif

namespace hbl {

// A level's work is cut into units of up to 2^lg arcs of one node.
constexpr uint32_t UNIT_LG = 3, UNIT = 1u << UNIT_LG;

// units of a graph at most, and the tiles of 32 units of its largest possible level
inline uint64_t units(uint64_t n, uint64_t m, uint32_t lg) { return (m >> lg) + n; }
inline uint64_t tiles(uint64_t n, uint64_t m, uint32_t lg) { return units(n, m, lg) / 32 + 1; }

// What a visit keeps for each node. The wide form has a 16-byte word of every
// node's arcs and one of every queued node's (Entry), units of 2^UNIT_LG arcs
// and 32-bit sums of them. The lean form reads the offsets instead, keeps the
// queued nodes' units alone, and takes longer units, so that no graph that has
// room beside its offsets and queue is refused.
struct Form {
    bool lean;
    uint32_t lg;
};

// sums of units in 32 bits with room for what a launch adds to them
constexpr uint64_t MAX_WIDE_UNITS = 0xf0000000ull;
// Device bytes that the wide form may take more than the lean one without asking,
// and as a share of the free ones: a visit stands beside the program's other
// data. (The lean form is the slower one: visits of web-like graphs of 3e5, 4e6 and
// 1.6e7 nodes take 0.135, 0.54 and 1.79 ms of kernels instead of 0.103, 0.41 and
// 1.46, sweeps of 6e4 and 2.6e5 nodes 10.4 and 15.4 ms instead of 8.7 and 12.9.)
constexpr uint64_t WIDE_BYTES = 1ull << 30, WIDE_SHARE = 8;

inline Form choose_form(uint64_t n, uint64_t m, uint64_t longest_row, uint64_t wide_bytes, uint64_t free_bytes) {
    if (units(n, m, UNIT_LG) <= MAX_WIDE_UNITS && longest_row < (1ull << 32) &&
        (wide_bytes <= WIDE_BYTES || wide_bytes <= free_bytes / WIDE_SHARE))
        return Form{false, UNIT_LG};
    // the tiles of both levels then take half a byte a node
    Form f{true, UNIT_LG};
    while (units(n, m, f.lg) > 0xffffffffull || (m >> f.lg) > n) f.lg++;
    return f;
}

// The longest row, where it may be longer than 32 bits count.
inline uint64_t longest_row(const uint64_t* off, uint64_t n, uint64_t m) {
    uint64_t d = 0;
    if (m >> 32)
        for (uint64_t v = 0; v < n; v++) d = std::max(d, off[v + 1] - off[v]);
    return d;
}

// The frontier is queue slots [b, e) with `units` units; d is the distance its
// successors get, last the largest distance that reached a node. An ended visit
// has no units. One block may store an ended state over the one in front of it
// while others of its launch still read that: of any mixture of their words the
// units are the older level's, which is the storing block's alone, or none. (32
// bytes: the words of a state never come from two sectors.)
struct alignas(32) State {
    uint32_t b, e, units, d, last;
};

// nothing left to expand
HBL_BOTH bool done(const State& s) { return s.units == 0; }

// The first level: start nodes in slots [b, e), where `units` units long.
HBL_BOTH State first_level(uint32_t b, uint32_t e, uint32_t units, uint32_t max_d) {
    return State{b, e, max_d >= 1 ? units : 0, 1, 0};
}

// The state after level s, whose nodes' queue ends at `tail` (slots | units <<
// 32), when nodes farther than max_d are not visited.
HBL_BOTH State advance(const State& s, unsigned long long tail, uint32_t max_d) {
    State t;
    t.b = s.e;
    t.e = (uint32_t)tail;
    t.d = s.d + 1;
    t.units = t.d > max_d ? 0u : (uint32_t)(tail >> 32);
    t.last = t.e > t.b ? s.d : s.last;
    return t;
}

}  // namespace hbl
