// One level of a breadth-first visit, shared by the visits (visits.cu) and
// ExactSumSweep (sum_sweep.cu).
//
// A level's work is cut by arcs, not by nodes. A queued node's entry holds its
// arcs and the number of units of UNIT arcs that stand before it in its level:
// slots and units are reserved by one 64-bit atomicAdd, so slot order is unit
// order. Whoever queues the node that holds unit 32 t of its level notes its
// slot in tile[t]; a warp takes a run of such tiles and walks one (up to 256
// arcs) at a time: eight successor loads in flight per lane, then eight visited
// bits, then the claims.
// A node of a hundred thousand arcs is spread over the whole grid, one of three
// arcs takes eight lanes of a warp.
//
// Visited nodes are a bitmap: the test is a plain load that L1 may answer (a
// stale zero costs an atomicOr that tells the truth), the claim an atomicOr.
//
// A level is a chain of dependent accesses, five to ten microseconds whatever
// it holds, so a level of at most SMALL units runs in the first block alone,
// which then goes on with the next levels behind block barriers for as long as
// they stay small: the narrow levels at the two ends of a visit, or all of a
// small graph's. Their entries stay in shared memory, and so does the bitmap
// of a graph of up to BITS nodes, which leaves two round trips a level (the
// successors, and the claimed nodes' offsets). A launch reads its level from
// st[in] and leaves the next one in st[in ^ 1], so no block sees a state that
// changes under it; an ended visit's state is left in both.
//
// Measured: the visit of a web-like graph of 4e6 nodes (42 M arcs) from one node
// takes 0.41 ms of kernels (0.54 in the lean form, see visit_state.h), where a warp per frontier node, a block per node
// above 4096 arcs and a host round trip per level took 2.6 ms. What bounds its two widest
// levels (160 and 121 us of it) is the SM's load unit, at one lane a cycle for
// scattered words: a test an arc, and a claim, an entry and a distance a node.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "launch_chain.cuh"
#include "visit_state.h"

namespace hbl {

constexpr int THREADS = 1024, WARPS = THREADS / 32;
constexpr int MAX_SMALL = 1024;  // small levels of one launch
// a warp queues its claimed nodes GROUP at a time, and when it holds as many; it
// takes those of half a tile at once
constexpr int GROUP = 64, RUN = GROUP + 128;
// Units of a level that one block takes: where the visited bits stand in shared
// memory and where they don't (a test of 32 scattered bits takes the block's one
// load unit about 4 cycles there, 32 in global memory). Device time of whole
// visits, us, with 0 / 512 / 1024 / 2048 / 4096 units: bits in shared memory,
// web-like 2.6e5 143 / 130 / 122 / 123 / 130, out-regular 2.6e5 140 / 121 / 121 /
// 118 / 150, out-regular 6e4 119 / 98 / 97 / 94 / 115; in global memory, out-regular
// 6e5 173 / 159 / 160 / 160 / 216, web-like 4e6 471 / 453 / 458 / 453 / 452,
// out-regular 4e6 471 / 449 / 452 / 451 / 515.
constexpr uint32_t SMALL = 2048, SMALL_GLOBAL = 512;
// Any level of a graph of at most this many units, whose launches are then one
// block each. Visits in one block / cut by level, us: web-like, 3,000 units 39 / 40,
// 6,700 53 / 58, 10,100 68 / 73, 13,600 74 / 67, 20,400 94 / 81; out-regular, 8,000
// units 46 / 50, 12,000 55 / 54, 16,000 62 / 54. Sweeps of symmetric graphs, ms:
// 6,000 units 144 / 155, 8,000 232 / 262, 10,000 313 / 319, 13,000 365 / 337.
constexpr uint32_t TINY = 10240;
constexpr uint32_t CAP = 512;          // entries of a level in shared memory
constexpr uint32_t BITS = 512 * 1024;  // nodes whose visited bits fit shared memory

// A node's arcs and, where it is queued, the units before it in its level. One
// such 16-byte word per node (Level::info) replaces two reads of the offsets: a
// warp's scattered access takes the SM's load unit 32 cycles whatever its width.
struct __align__(16) Entry {
    uint64_t off;
    uint32_t deg, unit;
};

struct Control {
    State st[2];
    unsigned long long tail;   // next free slot | units of the level being filled << 32
    unsigned long long known;  // arcs that led to visited nodes
    uint32_t ticket;           // blocks that finished this launch
    uint32_t launches;         // launches that had a level to expand
};

struct Level {
    const Entry* info;     // every node's arcs (k_info), or, in the lean form,
    const uint64_t* off;   // the offsets
    const uint32_t* succ;
    const uint32_t* comp;  // a visit stays inside its start nodes' components (COMP)
    uint32_t* visited;     // bitmap
    uint32_t* dist;        // distance and
    uint32_t* pred;        // predecessor (PRED) of every node visited, or null
    uint32_t* queue;       // visited nodes in visit order,
    Entry* entry;          // their entries, or, in the lean form,
    uint32_t* unit;        // the units before them in their level (see end_of_level),
    uint32_t* tile[2];     // a level's slots by units / 32, and the next level's (tiles() words each)
    uint32_t* qpred;       // their predecessors and
    uint32_t* qdist;       // their distances (PRED; not in the lean form), or null
    Control* ctl;
    uint64_t n;
    uint32_t lg;           // a unit's arcs (lean; else UNIT_LG)
    uint32_t max_d;        // nodes farther away are not visited
    uint32_t small;        // units of a level that the first block takes alone
};

inline uint32_t small_units(uint64_t n, uint64_t m, uint32_t lg) {
    if (units(n, m, UNIT_LG) <= TINY) return TINY;
    return std::max<uint32_t>((n <= BITS ? SMALL : SMALL_GLOBAL) >> std::min(lg - UNIT_LG, 31u), 1);
}

// what the queue keeps beside a node
template <bool LEAN>
using Slot = std::conditional_t<LEAN, uint32_t, Entry>;
__device__ __forceinline__ uint32_t unit_of(const Entry& e) { return e.unit; }
__device__ __forceinline__ uint32_t unit_of(uint32_t u) { return u; }

// The entries and tiles of a level and of the next, in a block that goes on alone.
template <bool LEAN>
struct Local {
    uint32_t tile[2][SMALL / 32];
    Slot<LEAN> entry[2][CAP];
    uint32_t node[2][CAP];
};

// A warp's claimed nodes, and the tile in hand: the first arc and the number of
// arcs of each unit.
template <bool PRED>
struct Run {
    uint32_t node[RUN];
    uint32_t pred[PRED ? RUN : 4];
    uint32_t unit_pred[PRED ? 32 : 4];
    ulonglong2 unit[32];
};

__device__ __forceinline__ Entry load_entry(const Entry* p) {
    const ulonglong2 t = __ldg(reinterpret_cast<const ulonglong2*>(p));
    return Entry{t.x, (uint32_t)t.y, (uint32_t)(t.y >> 32)};
}

__device__ __forceinline__ bool visited(const uint32_t* bits, uint32_t s) { return (bits[s >> 5] >> (s & 31)) & 1u; }
__device__ __forceinline__ bool claim(uint32_t* bits, uint32_t s) {
    const uint32_t bit = 1u << (s & 31);
    return !(atomicOr(bits + (s >> 5), bit) & bit);
}

// Queues nodes [from, fill) of the warp's run, at most GROUP of them, as nodes
// at distance d (every lane). With `next`, the first CAP entries from slot
// `first` on also go to next->entry[side].
template <bool PRED, bool LEAN>
__device__ __forceinline__ void put_group(const Level& a, unsigned long long* tail, const Run<PRED>& run, int from, int fill,
                                          uint32_t d, Local<LEAN>* next, int side, uint32_t first, uint32_t* tile) {
    constexpr int G = GROUP / 32;
    const int lane = threadIdx.x & 31;
    uint32_t v[G], own[G], units = 0;
    Entry en[G];
#pragma unroll
    for (int i = 0; i < G; i++) {
        const int k = from + i * 32 + lane;
        v[i] = k < fill ? run.node[k] : 0u;
        en[i] = Entry{0, 0, 0};
        if constexpr (LEAN) {
            own[i] = k < fill ? (uint32_t)((__ldg(a.off + v[i] + 1) - __ldg(a.off + v[i]) + (1ull << a.lg) - 1) >> a.lg) : 0u;
        } else {
            if (k < fill) en[i] = load_entry(a.info + v[i]);
            own[i] = (en[i].deg + UNIT - 1) / UNIT;
        }
    }
#pragma unroll
    for (int i = 0; i < G; i++) {
        const uint32_t u = own[i];
        uint32_t x = u;  // inclusive scan
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        en[i].unit = units + x - u;
        units += __shfl_sync(0xffffffffu, x, 31);
    }
    unsigned long long at = 0;
    if (lane == 0) at = atomicAdd(tail, ((unsigned long long)units << 32) | (uint32_t)(fill - from));
    at = __shfl_sync(0xffffffffu, at, 0);
#pragma unroll
    for (int i = 0; i < G; i++) {
        const int k = from + i * 32 + lane;
        const uint32_t slot = (uint32_t)at + i * 32 + lane;
        uint32_t t0 = 0, t1 = 0;  // the tiles that start in the node's units
        if (k < fill) {
            en[i].unit += (uint32_t)(at >> 32);
            using Sum = std::conditional_t<LEAN, uint64_t, uint32_t>;
            t0 = (uint32_t)(((Sum)en[i].unit + 31) / 32);
            t1 = (uint32_t)(((Sum)en[i].unit + own[i] + 31) / 32);
            Slot<LEAN> kept;
            if constexpr (LEAN) a.unit[slot] = kept = en[i].unit;
            else a.entry[slot] = kept = en[i];
            a.queue[slot] = v[i];
            if (next && slot - first < CAP) {
                next->entry[side][slot - first] = kept;
                next->node[side][slot - first] = v[i];
            }
            if (a.dist) a.dist[v[i]] = d;
            if constexpr (PRED) {
                if (a.qpred) a.qpred[slot] = run.pred[k];
                if constexpr (!LEAN)
                    if (a.qdist) a.qdist[slot] = d;
                if (a.pred) a.pred[v[i]] = run.pred[k];
            }
            if (t1 == t0 + 1) {
                tile[t0] = slot;
                if (next && t0 < SMALL / 32) next->tile[side][t0] = slot;
            }
        }
        // a node of several tiles: the whole warp writes them
        for (unsigned many = __ballot_sync(0xffffffffu, t1 > t0 + 1); many; many &= many - 1u) {
            const int w = __ffs(many) - 1;
            const uint32_t b = __shfl_sync(0xffffffffu, t0, w), e = __shfl_sync(0xffffffffu, t1, w);
            for (uint32_t t = b + lane; t < e; t += 32) {
                tile[t] = slot - lane + w;
                if (next && t < SMALL / 32) next->tile[side][t] = slot - lane + w;
            }
        }
    }
}

// Queues the warp's run down to fewer than GROUP nodes, or all of it.
template <bool PRED, bool LEAN>
__device__ __forceinline__ void flush(const Level& a, unsigned long long* tail, const Run<PRED>& run, int& fill, bool all,
                                      uint32_t d, Local<LEAN>* next, int side, uint32_t first, uint32_t* tile) {
    __syncwarp();
    while (fill >= GROUP || (all && fill > 0)) {
        const int from = max(fill - GROUP, 0);
        put_group<PRED, LEAN>(a, tail, run, from, fill, d, next, side, first, tile);
        fill = from;
    }
    __syncwarp();
}

// Warp w of nw: its share of the level s, whose entries come from the queue
// or, with `local`, from loc->entry[side ^ 1]; what it claims goes to the queue and,
// with loc, to loc->entry[side].
template <bool COMP, bool PRED, bool LEAN>
__device__ __forceinline__ void expand(const Level& a, const State& s, unsigned long long* tail, uint32_t w,
                                       uint32_t nw, Run<PRED>& run, unsigned long long& known, uint32_t* bits,
                                       Local<LEAN>* loc, int side, bool local) {
    using Sum = std::conditional_t<LEAN, uint64_t, uint32_t>;  // of units
    const int lane = threadIdx.x & 31;
    const uint32_t lg = LEAN ? a.lg : UNIT_LG;
    const Sum ntiles = ((Sum)s.units + 31) / 32, per = (ntiles + nw - 1) / nw;
    if ((uint64_t)w * per >= ntiles) return;
    Sum u = w * per * 32;
    const Sum u1 = min(u + per * 32, (Sum)s.units);
    const Slot<LEAN>* entry;
    if constexpr (LEAN) entry = a.unit;
    else entry = a.entry;
    if (local) entry = loc->entry[side ^ 1] - s.b;
    const uint32_t* queue = local ? loc->node[side ^ 1] - s.b : a.queue;
    int fill = 0;
    for (uint32_t base = (local ? loc->tile[side ^ 1] : a.tile[(s.d & 1) ^ 1])[u / 32]; u < u1; base += 32) {
        // 32 slots at a time, one per lane
        const uint32_t slot = base + lane;
        uint32_t v = 0, cv = 0;
        Sum qu = ~(Sum)0;
        std::conditional_t<LEAN, uint64_t, uint32_t> deg = 0;
        uint64_t o = 0;
        if (slot < s.e) {
            const Slot<LEAN> en = entry[slot];
            qu = unit_of(en);
            if constexpr (PRED || COMP || LEAN) v = queue[slot];
            if constexpr (LEAN) {
                o = __ldg(a.off + v);
                deg = __ldg(a.off + v + 1) - o;
            } else {
                o = en.off;
                deg = en.deg;
            }
            if constexpr (COMP) cv = __ldg(a.comp + v);
        }
        const Sum lim = s.e - base > 32 ? min(u1, (Sum)unit_of(entry[base + 32])) : u1;
        for (; u < lim; u += min((Sum)32, lim - u)) {
            // lane l: unit u + l, in the last of the slots that starts at or before it
            const Sum x = u + lane;
            int idx = 0;
#pragma unroll
            for (int st = 16; st > 0; st >>= 1)
                if (__shfl_sync(0xffffffffu, qu, idx + st) <= x) idx += st;
            const auto skip = (x - __shfl_sync(0xffffffffu, qu, idx)) << lg;
            uint64_t first = __shfl_sync(0xffffffffu, o, idx) + skip;
            const auto rest = __shfl_sync(0xffffffffu, deg, idx) - skip;
            uint64_t left = x < lim ? min(rest, (Sum)1 << lg) : (Sum)0;
            const uint32_t c0 = COMP ? __shfl_sync(0xffffffffu, cv, idx) : 0u;
            if constexpr (PRED) run.unit_pred[lane] = __shfl_sync(0xffffffffu, v, idx);
            // UNIT arcs of each of the 32 units at a time (the lean form's may be longer)
            for (bool more = true; more;) {
                const uint32_t len = LEAN ? (uint32_t)min(left, (uint64_t)UNIT) : (uint32_t)left;
                run.unit[lane] = make_ulonglong2(first, COMP ? len | ((uint64_t)c0 << 32) : len);
                __syncwarp();
                uint32_t src[UNIT], cw[COMP ? UNIT : 1];
                uint32_t have = 0, hit = 0;
#pragma unroll
                for (int j = 0; j < (int)UNIT; j++) {
                    const ulonglong2 un = run.unit[j * 4 + (lane >> 3)];  // eight lanes per unit
                    src[j] = 0;
                    if constexpr (COMP) cw[j] = (uint32_t)(un.y >> 32);
                    if ((lane & 7u) < (uint32_t)un.y) {
                        src[j] = __ldg(a.succ + un.x + (lane & 7));
                        have |= 1u << j;
                    }
                }
#pragma unroll
                for (int j = 0; j < (int)UNIT; j++) {
                    bool c = ((have >> j) & 1u) && !visited(bits, src[j]);
                    if constexpr (COMP) c = c && __ldg(a.comp + src[j]) == cw[j];
                    hit |= (uint32_t)c << j;
                }
                if (hit) {
#pragma unroll
                    for (int j = 0; j < (int)UNIT; j++)
                        if (((hit >> j) & 1u) && !claim(bits, src[j])) hit &= ~(1u << j);
                }
                if constexpr (PRED) known += __popc(have & ~hit);
                if (__any_sync(0xffffffffu, hit != 0u)) {
#pragma unroll
                    for (int half = 0; half < 2; half++) {
                        // the lanes' claimed nodes, one lane after the other, into the run
                        constexpr int H = UNIT / 2;
                        const uint32_t mine = __popc((hit >> (half * H)) & ((1u << H) - 1u));
                        uint32_t y = mine;
#pragma unroll
                        for (int o = 1; o < 32; o <<= 1) {
                            const uint32_t z = __shfl_up_sync(0xffffffffu, y, o);
                            if (lane >= o) y += z;
                        }
                        uint32_t at = fill + y - mine;
#pragma unroll
                        for (int j = half * H; j < half * H + H; j++)
                            if ((hit >> j) & 1u) {
                                run.node[at] = src[j];
                                if constexpr (PRED) run.pred[at] = run.unit_pred[j * 4 + (lane >> 3)];
                                at++;
                            }
                        fill += __shfl_sync(0xffffffffu, y, 31);
                        flush<PRED, LEAN>(a, tail, run, fill, false, s.d, loc, side, s.e, a.tile[s.d & 1]);
                    }
                }
                __syncwarp();
                more = false;
                if constexpr (LEAN) {
                    first += len;
                    left -= len;
                    more = __any_sync(0xffffffffu, left != 0);
                }
            }
        }
    }
    flush<PRED, LEAN>(a, tail, run, fill, true, s.d, loc, side, s.e, a.tile[s.d & 1]);
}

// In the lean form an expanded level leaves its end where its first slot's units
// (none) stood, so that the host can tell the levels of a visit's events apart: a
// zero there is the last level's.
template <bool PRED, bool LEAN>
__device__ __forceinline__ void end_of_level(const Level& a, const State& s) {
    if constexpr (PRED && LEAN) a.unit[s.b] = s.e;
}

template <bool COMP, bool PRED, bool LEAN>
__global__ void __launch_bounds__(THREADS, 1) k_level(const Level a, int in) {
    extern __shared__ __align__(16) uint8_t smem[];
    Run<PRED>& run = reinterpret_cast<Run<PRED>*>(smem)[threadIdx.x >> 5];
    __shared__ unsigned long long s_tail;
    wait_for_launch();
    Control* ctl = a.ctl;
    State s = ctl->st[in];
    const bool small = s.units <= a.small;
    if (done(s) || (small && blockIdx.x != 0)) return;
    unsigned long long known = 0;
    if (small) {
        Local<LEAN>* loc = reinterpret_cast<Local<LEAN>*>(smem + sizeof(Run<PRED>) * WARPS);
        uint32_t* bits = a.visited;
        const uint32_t words = (uint32_t)((a.n + 31) / 32);
        const bool mine = a.n <= BITS;
        if (mine) {
            bits = reinterpret_cast<uint32_t*>(loc + 1);
            for (uint32_t i = threadIdx.x; i < words; i += THREADS) bits[i] = a.visited[i];
        }
        int side = 1;  // the level is in entry[side ^ 1], the next goes to entry[side]
        auto fits = [&] { return s.e - s.b <= CAP && s.units <= SMALL; };
        if (fits()) {
            for (uint32_t i = threadIdx.x; i < s.e - s.b; i += THREADS) {
                if constexpr (LEAN) loc->entry[0][i] = a.unit[s.b + i];
                else loc->entry[0][i] = a.entry[s.b + i];
                loc->node[0][i] = a.queue[s.b + i];
            }
            for (uint32_t i = threadIdx.x; i * 32 < s.units; i += THREADS)
                loc->tile[0][i] = a.tile[(s.d & 1) ^ 1][i];
        }
        if (threadIdx.x == 0) s_tail = s.e;
        __syncthreads();
        int left = MAX_SMALL;
        do {
            expand<COMP, PRED, LEAN>(a, s, &s_tail, threadIdx.x >> 5, WARPS, run, known, bits, loc, side, fits());
            __syncthreads();
            const unsigned long long t = s_tail;
            __syncthreads();
            if (threadIdx.x == 0) end_of_level<PRED, LEAN>(a, s);
            s = advance(s, t, a.max_d);
            if (threadIdx.x == 0) s_tail = s.e;  // read again behind the barriers of the next level
            side ^= 1;
            __syncthreads();
        } while (--left > 0 && !done(s) && s.units <= a.small);
        if (mine)
            for (uint32_t i = threadIdx.x; i < words; i += THREADS) a.visited[i] = bits[i];
        if (threadIdx.x == 0) {
            ctl->st[in ^ 1] = s;
            // an ended visit stands in both: a block that still reads st[in] finds
            // no units there, or those of the level that was small
            if (done(s)) ctl->st[in] = s;
            ctl->tail = s.e;
            ctl->launches++;
        }
    } else {
        expand<COMP, PRED, LEAN>(a, s, &ctl->tail, blockIdx.x * WARPS + (threadIdx.x >> 5), gridDim.x * WARPS, run, known,
                                 a.visited, nullptr, 0, false);
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            if (atomicAdd(&ctl->ticket, 1u) == gridDim.x - 1) {
                // the last block: the queue is complete
                end_of_level<PRED, LEAN>(a, s);
                const State t = advance(s, atomicAdd(&ctl->tail, 0ull), a.max_d);
                ctl->st[in ^ 1] = t;
                if (done(t)) ctl->st[in] = t;
                ctl->tail = t.e;
                ctl->ticket = 0;
                ctl->launches++;
            }
        }
    }
    if constexpr (PRED) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) known += __shfl_xor_sync(0xffffffffu, known, o);
        if ((threadIdx.x & 31) == 0 && known) atomicAdd(&ctl->known, known);
    }
}

// info[v] = node v's arcs
static __global__ void k_info(const uint64_t* __restrict__ off, uint64_t n, Entry* info) {
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x)
        info[v] = Entry{off[v], (uint32_t)(off[v + 1] - off[v]), 0};
}

// The start nodes not yet visited, at distance 0: the first level of a visit,
// in st[0] and st[1]. They are queued from slot `from` on, where ctl->tail stood before
// the first of the launches that bring them; `last` marks the last one.
template <bool PRED, bool LEAN>
__global__ void __launch_bounds__(THREADS, 1) k_starts(const Level a, const uint32_t* __restrict__ starts, uint64_t count,
                                                       uint32_t from, bool last) {
    extern __shared__ __align__(16) uint8_t smem[];
    Run<PRED>& run = reinterpret_cast<Run<PRED>*>(smem)[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    Control* ctl = a.ctl;
    int fill = 0;
    const uint64_t limit = (count + 31) & ~31ull;  // whole warps go round together
    for (uint64_t i = (uint64_t)blockIdx.x * THREADS + threadIdx.x; i < limit; i += (uint64_t)gridDim.x * THREADS) {
        const uint32_t r = i < count ? starts[i] : 0u;
        const bool c = i < count && claim(a.visited, r);
        const unsigned mask = __ballot_sync(0xffffffffu, c);
        if (c) {
            const int k = fill + __popc(mask & ((1u << lane) - 1u));
            run.node[k] = r;
            if constexpr (PRED) run.pred[k] = r;
        }
        fill += __popc(mask);
        flush<PRED, LEAN>(a, &ctl->tail, run, fill, false, 0, nullptr, 0, 0, a.tile[0]);
    }
    flush<PRED, LEAN>(a, &ctl->tail, run, fill, true, 0, nullptr, 0, 0, a.tile[0]);
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&ctl->ticket, 1u) == gridDim.x - 1) {
            ctl->ticket = 0;
            ctl->launches = 0;
            if (last) {
                const unsigned long long tail = atomicAdd(&ctl->tail, 0ull);
                // in both: a first level without units is the end
                ctl->st[0] = ctl->st[1] = first_level(from, (uint32_t)tail, (uint32_t)(tail >> 32), a.max_d);
                ctl->tail = (uint32_t)tail;
            }
        }
    }
}

template <bool PRED, bool LEAN>
inline cudaError_t launch_starts_as(const Level& a, const uint32_t* starts, uint64_t count, uint32_t from, bool last,
                                    int sms, cudaStream_t s) {
    constexpr size_t smem = sizeof(Run<PRED>) * WARPS;
    static OncePerDevice once;
    if (const cudaError_t e = allow_shared(once, k_starts<PRED, LEAN>, smem); e != cudaSuccess) return e;
    const int grid = (int)std::min<uint64_t>((count + THREADS - 1) / THREADS, (uint64_t)sms);
    k_starts<PRED, LEAN><<<grid, THREADS, smem, s>>>(a, starts, count, from, last);
    return cudaGetLastError();
}

template <bool PRED>
inline cudaError_t launch_starts(const Level& a, const uint32_t* starts, uint64_t count, uint32_t from, bool last, int sms,
                                 cudaStream_t s) {
    return a.off ? launch_starts_as<PRED, true>(a, starts, count, from, last, sms, s)
                 : launch_starts_as<PRED, false>(a, starts, count, from, last, sms, s);
}

template <bool COMP, bool PRED, bool LEAN>
inline cudaError_t launch_levels_as(const Level& a, int count, int& in, int sms, cudaStream_t s) {
    // shared memory comes out of L1, which answers a wide level's tests: a graph
    // whose bits would not fit it takes less
    constexpr size_t base = sizeof(Run<PRED>) * WARPS + sizeof(Local<LEAN>), most = base + BITS / 8;
    static_assert(most <= 227 * 1024 - 64, "one block per SM");
    static OncePerDevice once;
    if (const cudaError_t e = allow_shared(once, k_level<COMP, PRED, LEAN>, most); e != cudaSuccess) return e;
    const size_t smem = a.n <= BITS ? base + ((a.n + 31) / 32 * 4 + 15) / 16 * 16 : base;
    const int grid = a.small == TINY ? 1 : sms;  // TINY: every level is the first block's
    for (int k = 0; k < count; k++) {
        const cudaError_t e = chain(k_level<COMP, PRED, LEAN>, grid, THREADS, smem, s, a, in);
        if (e != cudaSuccess) return e;
        in ^= 1;
    }
    return cudaSuccess;
}

// `count` launches of level kernels, of which the first reads st[in]; one past
// the last level does nothing (and costs about 1.4 us)
template <bool COMP, bool PRED>
inline cudaError_t launch_levels(const Level& a, int count, int& in, int sms, cudaStream_t s) {
    return a.off ? launch_levels_as<COMP, PRED, true>(a, count, in, sms, s)
                 : launch_levels_as<COMP, PRED, false>(a, count, in, sms, s);
}

}  // namespace hbl
