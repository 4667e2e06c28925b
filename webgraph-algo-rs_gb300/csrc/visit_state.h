// What a breadth-first visit carries from level to level (visit_level.cuh);
// plain C++ where no CUDA compiler reads it.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define HBL_BOTH __host__ __device__ __forceinline__
#else
#define HBL_BOTH inline
#endif

namespace hbl {

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
