// ExactSumSweep on the device: the GB300 counterpart of the reference's
// ExactSumSweep (src/algo/exact_sum_sweep/computer.rs, scc_graph.rs,
// output_level.rs; Borassi et al., "Fast diameter and radius BFS-based
// computation in (weakly connected) real-world graphs", TCS 586, 2015).
//
// The work of the algorithm is its breadth-first visits (forward on the
// graph, backward on the transpose) and, after each, an update of per-node
// bounds; between visits it picks the next start node with a filtered
// argmax / argmin over all nodes. A step is one run of launches with one
// synchronisation at its end:
//   k_sw_select               filtered argmax / argmin, with the reference's tie
//                             rules (larger / smaller value, then tie value, then
//                             smaller node); the start stays on the device;
//   k_sw_begin                distances and visited bits cleared, the start queued;
//   hbl::k_level              the levels of the visit (visit_level.cuh), as many
//                             launches as the visits before it took; an optional
//                             component array keeps a visit inside each start
//                             node's strongly connected component
//                             (computer.rs:745-800: all pivots at once);
//   k_sw_forward / k_sw_backward, k_sw_missing
//                             the per-node bound updates of a forward /
//                             backward visit (computer.rs:572-693), a new minimal
//                             radius as an atomicMin of (eccentricity << 32 |
//                             node), and the five counts of find_missing_nodes;
//                             the last block writes what the host needs into
//                             page-locked memory. When the visit has not ended,
//                             they do nothing and the host adds levels.
// and for all_cc_upper_bound:
//   k_sw_pivot_*              the best pivot of every component
//                             (computer.rs:418-475) by three atomicMin passes;
//   k_sw_refine               the node pass.
// What bounds a step is the chain of its launches and, inside a level, of its
// accesses. Web-like 2.6e5 (2.6 M arcs), 621 visits: 0.15 ms a visit, where three
// launches a level, eight levels at a time, and four synchronisations took
// 0.69; every eccentricity of a symmetric graph of 3000 nodes, whose visits one
// block runs: 54 us a step where it took 130.
// The strongly connected component of the largest out-degree node comes from
// two device visits (one for a symmetric graph); the host runs Tarjan's
// algorithm (sccs/tarjan.rs) or the symmetric labelling (sccs/symm_seq.rs) on
// the nodes outside it (see directed_components, symmetric_components). The
// arcs between components are listed on the device (cross_arcs); the host picks
// one per pair of components (scc_graph.rs) and runs the two passes over
// the component DAG of all_cc_upper_bound (computer.rs:829-873), which touch
// one value per component and per DAG arc.
//
// Where the reference's parallel visits leave a choice open (which of the
// nodes reaching a new minimal radius in one step becomes the radial vertex)
// this takes the smallest node; everything else follows the reference's
// sequence of steps exactly, so the iteration counts match too.
#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>

#include <algorithm>
#include <chrono>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "hb_internal.h"
#include "visit_level.cuh"

namespace hbs {

constexpr uint32_t INF = 0xffffffffu;
constexpr int SW_THREADS = 256;

struct Best {
    uint64_t val, tie;
    uint64_t idx;  // ~0: none
};

// What the kernels of a step keep on the device between launches.
struct Scratch {
    Best pick;                     // the selected start
    unsigned long long key;        // radius candidate (~0: none)
    unsigned long long count[5];   // missing nodes
    uint32_t ticket;
};

// What a step tells the host (page-locked memory).
struct Result {
    uint64_t done;                 // 0: the visit needs more levels
    uint64_t start;                // ~0: no node qualified, the step did nothing
    uint64_t ecc, visited, launches;
    uint64_t radial;               // the start is a radial vertex
    uint64_t key;
    uint64_t count[5];
};

// One start node (the selected one, or `root` when pick is null): every
// distance unknown, every bit clear but the start's.
__global__ void k_sw_begin(const hbl::Level a, uint64_t n, const Scratch* pick, uint32_t root) {
    hbl::wait_for_launch();
    const uint64_t t0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t r = pick ? pick->pick.idx : root;
    for (uint64_t v = t0; v < n; v += stride) a.dist[v] = v == r ? 0u : INF;
    for (uint64_t w = t0; w < (n + 31) / 32; w += stride) a.visited[w] = w == r >> 5 ? 1u << (r & 31) : 0u;
    uint64_t units = 0;  // the first level is the start's units
    if (r != ~0ull) units = a.off ? (a.off[r + 1] - a.off[r] + (1ull << a.lg) - 1) >> a.lg
                                  : ((uint64_t)a.info[r].deg + hbl::UNIT - 1) / hbl::UNIT;
    for (uint64_t t = t0; t * 32 < units; t += stride) a.tile[0][t] = 0;
    if (t0 == 0) {
        hbl::State s{0, 0, 0, 1, 0};
        if (r != ~0ull) {
            s.e = 1;
            s.units = (uint32_t)units;
            if (a.off) a.unit[0] = 0;
            else a.entry[0] = a.info[r];
            a.queue[0] = (uint32_t)r;
        }
        // in both: of a start without arcs no launch has a level to expand, and
        // each writes nothing
        a.ctl->st[0] = a.ctl->st[1] = s;
        a.ctl->tail = s.e;
        a.ctl->ticket = 0;
        a.ctl->launches = 0;
    }
}

// the five counts of computer.rs:929-973: radial below the radius bound,
// incomplete forward and backward above the diameter bound, incomplete forward,
// incomplete backward
struct Counts {
    uint32_t r = 0, df = 0, db = 0, af = 0, ab = 0;
    __device__ __forceinline__ void add(uint64_t fl, uint64_t fh, uint64_t bl, uint64_t bh, bool radial,
                                        uint64_t diameter_low, uint64_t radius_high) {
        if (fl != fh) {
            af++;
            df += fh > diameter_low;
            r += radial && fl < radius_high;
        }
        if (bl != bh) {
            ab++;
            db += bh > diameter_low;
        }
    }
};

// Adds the block's counts to s->count; the last block to arrive gives the
// host its result and clears the scratch for the next step.
__device__ __forceinline__ void finish_counts(Counts c, Scratch* s, const hbl::Control* ctl, const uint8_t* radial,
                                              bool step, Result* out) {
    __shared__ uint32_t sum[5][SW_THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t v[5] = {c.r, c.df, c.db, c.af, c.ab};
#pragma unroll
    for (int k = 0; k < 5; k++) {
        const uint32_t t = __reduce_add_sync(0xffffffffu, v[k]);
        if (lane == 0) sum[k][warp] = t;
    }
    __syncthreads();
    if (threadIdx.x < 5) {
        unsigned long long t = 0;
        for (int w = 0; w < SW_THREADS / 32; w++) t += sum[threadIdx.x][w];
        if (t) atomicAdd(&s->count[threadIdx.x], t);
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x != 0 || atomicAdd(&s->ticket, 1u) != gridDim.x - 1) return;
    __threadfence();
    const hbl::State st = ctl->st[0];
    const uint64_t start = step ? s->pick.idx : ~0ull;
    out->done = 1;
    out->start = start;
    out->ecc = st.last;
    out->visited = st.e;
    out->launches = ctl->launches;
    out->radial = start != ~0ull && radial[start] != 0;
    out->key = atomicAdd(&s->key, 0ull);
    for (int k = 0; k < 5; k++) {
        out->count[k] = atomicAdd(&s->count[k], 0ull);
        s->count[k] = 0;
    }
    s->key = ~0ull;
    s->ticket = 0;
}

// true (and the host told) when the visit has not ended
__device__ __forceinline__ bool unfinished(const hbl::Control* ctl, Result* out) {
    if (hbl::done(ctl->st[0])) return false;
    if (blockIdx.x == 0 && threadIdx.x == 0) out->done = 0;
    return true;
}

// computer.rs:652-678 (forward visit): backward totals and lower bounds, the
// start's forward bounds; then the missing counts
__global__ void __launch_bounds__(SW_THREADS) k_sw_forward(
    uint64_t n, const uint32_t* __restrict__ dist, uint64_t* bt, uint64_t* bl, const uint64_t* __restrict__ bh,
    uint64_t* fl, uint64_t* fh, const uint8_t* __restrict__ radial, uint64_t diameter_low, uint64_t radius_high,
    Scratch* s, const hbl::Control* ctl, Result* out) {
    hbl::wait_for_launch();
    if (unfinished(ctl, out)) return;
    const uint64_t start = s->pick.idx, ecc = ctl->st[0].last;
    if (start != ~0ull) {
        diameter_low = max(diameter_low, ecc);
        if (radial[start] && radius_high > ecc) radius_high = ecc;
    }
    Counts c;
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t d = dist[v];
        uint64_t l = bl[v], f = fl[v], g = fh[v];
        const uint64_t u = bh[v];
        if (d != INF) {
            bt[v] += d;
            if (l != u && l < d) bl[v] = l = d;
        }
        if (v == start) fl[v] = fh[v] = f = g = ecc;
        c.add(f, g, l, u, radial[v] != 0, diameter_low, radius_high);
    }
    finish_counts(c, s, ctl, radial, true, out);
}

// computer.rs:586-626 (backward visit): forward totals and lower bounds; a
// node whose bounds meet becomes a radius candidate; the start's backward bounds
__global__ void __launch_bounds__(SW_THREADS) k_sw_backward(
    uint64_t n, const uint32_t* __restrict__ dist, uint64_t* ft, uint64_t* fl, const uint64_t* __restrict__ fh,
    uint64_t* bl, uint64_t* bh, const uint8_t* __restrict__ radial, Scratch* s, const hbl::Control* ctl, Result* out) {
    hbl::wait_for_launch();
    if (unfinished(ctl, out)) return;
    const uint64_t start = s->pick.idx, ecc = ctl->st[0].last;
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t d = dist[v];
        if (d != INF) {
            ft[v] += d;
            const uint64_t l = fl[v], u = fh[v];
            if (l != u && l < d) {
                fl[v] = d;
                if (d == u && radial[v]) atomicMin(&s->key, (unsigned long long)((d << 32) | v));
            }
        }
        if (v == start) bl[v] = bh[v] = ecc;
    }
}

// The missing counts alone: after a backward visit (`step`: with the bounds it
// leaves) or after all_cc_upper_bound.
__global__ void __launch_bounds__(SW_THREADS) k_sw_missing(
    uint64_t n, const uint64_t* __restrict__ fl, const uint64_t* __restrict__ fh, const uint64_t* __restrict__ bl,
    const uint64_t* __restrict__ bh, const uint8_t* __restrict__ radial, uint64_t diameter_low, uint64_t radius_high,
    int step, Scratch* s, const hbl::Control* ctl, Result* out) {
    hbl::wait_for_launch();
    if (step) {
        if (unfinished(ctl, out)) return;
        if (s->pick.idx != ~0ull) diameter_low = max(diameter_low, (uint64_t)ctl->st[0].last);
        if (s->key != ~0ull) radius_high = min(radius_high, (uint64_t)(s->key >> 32));
    }
    Counts c;
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x)
        c.add(fl[v], fh[v], bl[v], bh[v], radial[v] != 0, diameter_low, radius_high);
    finish_counts(c, s, ctl, radial, step != 0, out);
}

// the visited nodes become radial vertices
__global__ void k_sw_mark(uint64_t n, const uint32_t* __restrict__ dist, uint8_t* radial) {
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x)
        if (dist[v] != INF) radial[v] = 1;
}

// a pivot's eccentricity inside its component: the largest distance there.
// Most warps see one component (the giant one), so the warp agrees first; the
// plain read in front keeps the atomics to the ones that raise the maximum.
__global__ void k_sw_pivot_ecc(uint64_t n, const uint32_t* __restrict__ dist, const uint32_t* __restrict__ comp,
                               unsigned long long* ecc) {
    const uint64_t limit = (n + 31) & ~31ull;
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < limit; v += (uint64_t)gridDim.x * blockDim.x) {
        const bool in = v < n && dist[v] != INF;
        const uint32_t c = in ? comp[v] : 0xffffffffu, d = in ? dist[v] : 0u;
        int same;
        __match_all_sync(0xffffffffu, c, &same);
        const uint32_t m = __reduce_max_sync(0xffffffffu, d);
        if (!in || (same && (threadIdx.x & 31) != 0)) continue;
        const unsigned long long x = same ? m : d;
        if (*(volatile unsigned long long*)(ecc + c) < x) atomicMax(ecc + c, x);
    }
}

// a better than b: larger (val, tie) when maximizing, smaller when
// minimizing, then the smaller node (argmax.rs, argmin.rs)
__device__ __host__ __forceinline__ bool better(const Best& a, const Best& b, bool maximize) {
    if (a.idx == ~0ull) return false;
    if (b.idx == ~0ull) return true;
    if (a.val != b.val) return maximize ? a.val > b.val : a.val < b.val;
    if (a.tie != b.tie) return maximize ? a.tie > b.tie : a.tie < b.tie;
    return a.idx < b.idx;
}

// s[0] = the best of the block's b
__device__ __forceinline__ void block_best(Best b, Best* s, bool maximize) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto over = [&](int lanes) {
        for (int o = lanes / 2; o > 0; o >>= 1) {
            const Best c{__shfl_xor_sync(0xffffffffu, b.val, o), __shfl_xor_sync(0xffffffffu, b.tie, o),
                         __shfl_xor_sync(0xffffffffu, b.idx, o)};
            if (better(c, b, maximize)) b = c;
        }
    };
    over(32);
    __syncthreads();
    if (lane == 0) s[warp] = b;
    __syncthreads();
    if (warp == 0) {
        b = lane < SW_THREADS / 32 ? s[lane] : Best{0, 0, ~0ull};
        over(SW_THREADS / 32);
        if (lane == 0) s[0] = b;
    }
    __syncthreads();
}

// filter: 0 fa[i] != fb[i] (bounds not met), 1 radial[i]; val == nullptr:
// the out-degree from off (the start of the SumSweep heuristic)
__global__ void k_sw_select(uint64_t n, const uint64_t* __restrict__ val, const uint64_t* __restrict__ tie,
                            const uint64_t* __restrict__ off, int maximize, int filter,
                            const uint64_t* __restrict__ fa, const uint64_t* __restrict__ fb,
                            const uint8_t* __restrict__ radial, Best* part, Scratch* scr, uint64_t* host) {
    hbl::wait_for_launch();
    __shared__ Best s[SW_THREADS / 32];
    __shared__ bool last;
    Best b{0, 0, ~0ull};
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        bool keep = true;
        if (filter == 0) keep = fa[i] != fb[i];
        else if (filter == 1) keep = radial[i] != 0;
        if (!keep) continue;
        Best c;
        c.val = val ? val[i] : off[i + 1] - off[i];
        c.tie = tie ? tie[i] : 0;
        c.idx = i;
        if (better(c, b, maximize)) b = c;
    }
    block_best(b, s, maximize);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = s[0];
        __threadfence();
        last = atomicAdd(&scr->ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    // the last block: the best of the blocks (written in this launch: not cached)
    __threadfence();
    b = Best{0, 0, ~0ull};
    for (int k = threadIdx.x; k < (int)gridDim.x; k += SW_THREADS) {
        const Best c{__ldcg(&part[k].val), __ldcg(&part[k].tie), __ldcg(&part[k].idx)};
        if (better(c, b, maximize)) b = c;
    }
    block_best(b, s, maximize);
    if (threadIdx.x == 0) {
        scr->pick = s[0];
        scr->ticket = 0;
        if (host) *host = s[0].idx;
    }
}

// computer.rs:424-466: per component the node of the smallest
// (bl + fl + n [forward bounds met] + n [backward bounds met], ft + bt, node)
__device__ __forceinline__ uint64_t pivot_score(uint64_t v, uint64_t n, const uint64_t* fl, const uint64_t* fh,
                                                const uint64_t* bl, const uint64_t* bh) {
    return bl[v] + fl[v] + (fl[v] != fh[v] ? 0 : n) + (bl[v] != bh[v] ? 0 : n);
}
__global__ void k_sw_pivot_pass(int pass, uint64_t n, const uint32_t* __restrict__ comp,
                                const uint64_t* __restrict__ fl, const uint64_t* __restrict__ fh,
                                const uint64_t* __restrict__ bl, const uint64_t* __restrict__ bh,
                                const uint64_t* __restrict__ ft, const uint64_t* __restrict__ bt,
                                unsigned long long* best_score, unsigned long long* best_tot, uint32_t* pivot) {
    // Most warps see one component (the giant one), whose minimum is one word:
    // such a warp agrees on its own first, and a plain read keeps the atomics
    // to the ones that lower the minimum.
    const uint64_t limit = (n + 31) & ~31ull;
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < limit; v += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t c = v < n ? comp[v] : 0xffffffffu;
        uint64_t x = ~0ull;
        if (v < n) {
            const uint64_t sc = pivot_score(v, n, fl, fh, bl, bh);
            if (pass == 0) {
                x = sc;
            } else if (sc == best_score[c]) {
                const uint64_t tot = ft[v] + bt[v];
                if (pass == 1) x = tot;
                else if (tot == best_tot[c]) x = v;
            }
        }
        int same;
        __match_all_sync(0xffffffffu, c, &same);
        if (same) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) x = min(x, __shfl_xor_sync(0xffffffffu, x, o));
        }
        if (x == ~0ull || (same && (threadIdx.x & 31) != 0)) continue;
        if (pass == 2) {
            if (*(volatile uint32_t*)(pivot + c) > (uint32_t)x) atomicMin(pivot + c, (uint32_t)x);
        } else {
            unsigned long long* best = (pass == 0 ? best_score : best_tot) + c;
            if (*(volatile unsigned long long*)best > x) atomicMin(best, (unsigned long long)x);
        }
    }
}

// gathers: out[k] = src[idx[k]]
__global__ void k_sw_gather(const uint32_t* __restrict__ idx, uint64_t count, const uint32_t* __restrict__ src,
                            uint32_t* out) {
    for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < count; k += (uint64_t)gridDim.x * blockDim.x)
        out[k] = src[idx[k]];
}
__global__ void k_sw_gather64(const uint32_t* __restrict__ idx, uint64_t count, const uint64_t* __restrict__ src,
                              uint64_t* out) {
    for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < count; k += (uint64_t)gridDim.x * blockDim.x)
        out[k] = src[idx[k]];
}

// computer.rs:879-915: the node pass of all_cc_upper_bound
__global__ void k_sw_refine(uint64_t n, const uint32_t* __restrict__ comp, const uint32_t* __restrict__ df,
                            const uint32_t* __restrict__ db, const uint64_t* __restrict__ ef,
                            const uint64_t* __restrict__ eb, const uint64_t* __restrict__ fl, uint64_t* fh,
                            uint64_t* bh, const uint8_t* __restrict__ radial, unsigned long long* key) {
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t c = comp[v];
        uint64_t h = fh[v];
        const uint64_t pv = (uint64_t)db[v] + ef[c];
        if (pv < h) {
            fh[v] = pv;
            h = pv;
        }
        if (h == fl[v] && radial[v]) atomicMin(key, (h << 32) | v);
        const uint64_t pb = (uint64_t)df[v] + eb[c];
        if (pb < bh[v]) bh[v] = pb;
    }
}

__global__ void k_sw_fill64(uint64_t* p, uint64_t count, uint64_t value) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (uint64_t)gridDim.x * blockDim.x)
        p[i] = value;
}

__global__ void k_sw_validate(const uint64_t* __restrict__ off, const uint32_t* __restrict__ succ, uint64_t n,
                              uint64_t m, int* bad) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t t0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (uint64_t v = t0; v < n; v += stride)
        if (off[v] > off[v + 1]) *bad = 1;
    for (uint64_t x = t0; x < m; x += stride)
        if (succ[x] >= n) *bad = 1;
}

}  // namespace hbs

namespace {

using u64 = uint64_t;
constexpr u64 NONE = ~0ull;

thread_local std::string t_sweep_err;

struct SweepError {
    int code;
    std::string msg;
};

[[noreturn]] void fail(int code, const std::string& msg) { throw SweepError{code, msg}; }

void ck(cudaError_t e, const char* what) {
    if (e == cudaSuccess) return;
    cudaGetLastError();
    const int code = e == cudaErrorMemoryAllocation ? HB_ERR_OOM : HB_ERR_CUDA;
    fail(code, std::string(what) + ": " + cudaGetErrorString(e));
}

struct HostCsr {
    u64 n;
    const u64* off;
    const uint32_t* succ;
    u64 deg(u64 v) const { return off[v + 1] - off[v]; }
};

// sccs/tarjan.rs: components numbered as they are emitted (reverse
// topological order), roots in node order, successors in arc order
// With `group` given, only the nodes v with group[v] == want and the arcs
// between them take part (the other entries of comp are left as they are),
// and the components are numbered from ncomp on.
void tarjan_into(const HostCsr& g, std::vector<uint32_t>& comp, u64& ncomp, const uint8_t* group = nullptr,
                 uint8_t want = 0) {
    const u64 n = g.n;
    auto in = [&](u64 v) { return !group || group[v] == want; };
    std::vector<uint32_t> index(n, 0xffffffffu), low(n, 0);
    std::vector<uint8_t> on_stack(n, 0);
    std::vector<uint32_t> stack;
    std::vector<std::pair<uint32_t, u64>> call;
    uint32_t counter = 0;
    for (u64 r = 0; r < n; r++) {
        if (index[r] != 0xffffffffu || !in(r)) continue;
        index[r] = low[r] = counter++;
        stack.push_back((uint32_t)r);
        on_stack[r] = 1;
        call.push_back({(uint32_t)r, g.off[r]});
        while (!call.empty()) {
            const uint32_t v = call.back().first;
            u64& e = call.back().second;
            if (e < g.off[v + 1]) {
                const uint32_t w = g.succ[e++];
                if (!in(w)) continue;
                if (index[w] == 0xffffffffu) {
                    index[w] = low[w] = counter++;
                    stack.push_back(w);
                    on_stack[w] = 1;
                    call.push_back({w, g.off[w]});
                } else if (on_stack[w] && index[w] < low[v]) {
                    low[v] = index[w];
                }
                continue;
            }
            if (low[v] == index[v]) {
                for (;;) {
                    const uint32_t w = stack.back();
                    stack.pop_back();
                    on_stack[w] = 0;
                    comp[w] = (uint32_t)ncomp;
                    if (w == v) break;
                }
                ncomp++;
            }
            call.pop_back();
            if (!call.empty() && low[v] < low[call.back().first]) low[call.back().first] = low[v];
        }
    }
}

std::vector<uint32_t> tarjan(const HostCsr& g, u64& ncomp) {
    std::vector<uint32_t> comp(g.n, 0);
    ncomp = 0;
    tarjan_into(g, comp, ncomp);
    return comp;
}

// sccs/symm_seq.rs: components of a symmetric graph in order of their
// smallest node (nodes already labelled are skipped, the others numbered
// from ncomp on)
void symm_into(const HostCsr& g, std::vector<uint32_t>& comp, u64& ncomp) {
    std::vector<uint32_t> st;
    for (u64 r = 0; r < g.n; r++) {
        if (comp[r] != 0xffffffffu) continue;
        comp[r] = (uint32_t)ncomp;
        st.push_back((uint32_t)r);
        while (!st.empty()) {
            const uint32_t v = st.back();
            st.pop_back();
            for (u64 e = g.off[v]; e < g.off[v + 1]; e++)
                if (comp[g.succ[e]] == 0xffffffffu) {
                    comp[g.succ[e]] = (uint32_t)ncomp;
                    st.push_back(g.succ[e]);
                }
        }
        ncomp++;
    }
}

std::vector<uint32_t> symm_components(const HostCsr& g, u64& ncomp) {
    std::vector<uint32_t> comp(g.n, 0xffffffffu);
    ncomp = 0;
    symm_into(g, comp, ncomp);
    return comp;
}

struct Sweeper {
    int device = 0;
    cudaStream_t s = nullptr;
    bool own_stream = false;
    u64 n = 0, m = 0;
    bool undirected = false;
    int level = 0;
    int sms = 1;
    // device state
    u64 *d_off = nullptr, *d_toff = nullptr;
    uint32_t *d_succ = nullptr, *d_tsucc = nullptr;
    uint32_t *d_dist = nullptr, *d_queue = nullptr, *d_visited = nullptr, *d_comp = nullptr;
    uint32_t *d_df = nullptr, *d_db = nullptr;
    u64 *d_fl = nullptr, *d_fh = nullptr, *d_bl = nullptr, *d_bh = nullptr, *d_ft = nullptr, *d_bt = nullptr;
    uint8_t* d_radial = nullptr;
    hbl::Form form{false, hbl::UNIT_LG};
    void* wide = nullptr;                 // the wide form's arrays:
    hbl::Entry *d_entry = nullptr, *d_info = nullptr, *d_tinfo = nullptr;
    uint32_t* d_tile[2] = {nullptr, nullptr};
    hbl::Control* d_ctl = nullptr;
    hbs::Scratch* d_scr = nullptr;
    unsigned long long *d_ecc_f = nullptr, *d_ecc_b = nullptr, *d_best_score = nullptr, *d_best_tot = nullptr;
    uint32_t* d_pivot = nullptr;
    u64 *d_ef = nullptr, *d_eb = nullptr;
    uint32_t *d_cstart = nullptr, *d_cend = nullptr, *d_gather = nullptr;
    u64* d_gather64 = nullptr;
    hbs::Best* d_best = nullptr;          // the blocks' results of a selection
    hbs::Result* h_res = nullptr;         // page-locked
    int* d_bad = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    int ahead[2] = {4, 4};                // launches of the next forward / backward visit
    float device_ms = 0.f;
    u64 sweeps = 0;
    // host state (computer.rs:38-89)
    std::vector<uint32_t> comp;
    u64 ncomp = 0;
    std::vector<u64> seg;
    std::vector<uint32_t> cstart, cend, ctarget;
    u64 diameter_low = 0, radius_high = NONE, diameter_vertex = 0, radius_vertex = 0, iterations = 0;
    u64 radius_it = NONE, diameter_it = NONE, forward_it = NONE, all_it = NONE;
    bool compute_radial = true;
    int grid = 1;

    ~Sweeper() {
        cudaSetDevice(device);
        if (s) cudaStreamSynchronize(s);
        // a symmetric graph is its own transpose: each block once
        std::vector<void*> ps = {d_off, d_toff, d_succ, d_tsucc, d_dist, d_queue, wide, d_tile[0], d_tile[1], d_visited, d_comp,
                                 d_df, d_db, d_fl, d_fh, d_bl, d_bh, d_ft, d_bt, d_radial, d_ctl, d_scr, d_bad,
                                 d_ecc_f, d_ecc_b, d_best_score, d_best_tot, d_pivot, d_ef,
                                 d_eb, d_cstart, d_cend, d_gather, d_gather64, d_best};
        std::sort(ps.begin(), ps.end());
        ps.erase(std::unique(ps.begin(), ps.end()), ps.end());
        for (void* p : ps)
            if (p) cudaFree(p);
        if (h_res) cudaFreeHost(h_res);
        if (ev0) cudaEventDestroy(ev0);
        if (ev1) cudaEventDestroy(ev1);
        if (own_stream && s) cudaStreamDestroy(s);
    }

    template <class T>
    void alloc(T** p, u64 count) {
        ck(cudaMalloc((void**)p, std::max<u64>(count, 1) * sizeof(T)), "cudaMalloc");
    }
    int blocks(u64 work) const { return (int)std::min<u64>((work + hbs::SW_THREADS - 1) / hbs::SW_THREADS + 1, (u64)grid); }
    void sync() { ck(cudaStreamSynchronize(s), "cudaStreamSynchronize"); }

    hbl::Level level_args(bool backward, bool in_comp) const {
        hbl::Level a{};
        a.info = backward ? d_tinfo : d_info;
        a.off = form.lean ? backward ? d_toff : d_off : nullptr;
        a.lg = form.lg;
        a.unit = d_db;  // (lean) written between visits alone
        a.succ = backward ? d_tsucc : d_succ;
        a.comp = in_comp ? d_comp : nullptr;
        a.visited = d_visited;
        a.dist = d_dist;
        a.queue = d_queue;
        a.entry = d_entry;
        a.tile[0] = d_tile[0];
        a.tile[1] = d_tile[1];
        a.ctl = d_ctl;
        a.n = n;
        a.small = hbl::small_units(n, m, form.lg);
        a.max_d = hbs::INF;
        return a;
    }

    // The wide form's arrays, in one allocation: the entries, and every node's row
    // forward and backward. The transpose's offsets stand where the entries come
    // once its rows are known. Where they take more than their share of the free
    // memory the visits take the lean form (hbl::choose_form): up to 60 bytes a
    // component are still to come.
    void alloc_rows(const u64* off, const u64* toff) {
        const u64 entries = std::max<u64>(n * sizeof(hbl::Entry), (n + 1) * 8), rows = n * sizeof(hbl::Entry);
        const u64 bytes = entries + (undirected ? 1 : 2) * rows;
        const u64 more = bytes - (undirected ? 0 : (n + 1) * 8);
        size_t free_bytes = 0, all = 0;
        ck(cudaMemGetInfo(&free_bytes, &all), "cudaMemGetInfo");
        const u64 longest = std::max(hbl::longest_row(off, n, m), undirected ? 0 : hbl::longest_row(toff, n, m));
        form = hbl::choose_form(n, m, longest, more <= free_bytes / hbl::WIDE_SHARE ? more : UINT64_MAX, free_bytes);
        if (!form.lean) {
            const cudaError_t e = hbk::fail_allocation() ? cudaErrorMemoryAllocation : cudaMalloc(&wide, bytes);
            if (e == cudaErrorMemoryAllocation) {
                cudaGetLastError();
                wide = nullptr;
                form = hbl::choose_form(n, m, UINT64_MAX, 0, 0);
            } else {
                ck(e, "cudaMalloc");
                char* p = static_cast<char*>(wide);
                d_entry = reinterpret_cast<hbl::Entry*>(p);
                d_info = reinterpret_cast<hbl::Entry*>(p + entries);
                d_tinfo = undirected ? d_info : d_info + n;
            }
        }
        if (undirected) d_toff = d_off;
        else if (form.lean) alloc(&d_toff, n + 1);
    }

    // `count` more level launches of a visit (in: the parity of the next)
    void levels(const hbl::Level& a, int count, int& in) {
        ck(a.comp ? hbl::launch_levels<true, false>(a, count, in, sms, s)
                  : hbl::launch_levels<false, false>(a, count, in, sms, s),
           "k_level");
    }

    // after a visit that took `launches` launches with work
    void learn(bool backward, u64 launches) {
        // an idle launch costs about 1.4 us, a visit that needs another
        // synchronisation 20: the estimate falls by one launch a visit at most
        const int want = (int)std::max<u64>(1, std::min<u64>(launches, 64));
        ahead[backward] = std::max(want, ahead[backward] - 1);
    }

    // runs the levels of a visit to its end
    void run_levels(const hbl::Level& a, bool backward) {
        int in = 0;
        for (int k = ahead[backward];; k = 2) {
            levels(a, k, in);
            hbl::Control* c = reinterpret_cast<hbl::Control*>(h_res + 1);
            ck(cudaMemcpyAsync(c, d_ctl, sizeof *c, cudaMemcpyDeviceToHost, s), "cudaMemcpyAsync");
            sync();
            if (hbl::done(c->st[0])) {
                learn(backward, c->launches);
                return;
            }
        }
    }

    // A visit from `root` on the graph or its transpose: distances in d_dist.
    void visit(u64 root, bool backward) {
        const hbl::Level a = level_args(backward, false);
        ck(hbl::chain(hbs::k_sw_begin, blocks(n), hbs::SW_THREADS, 0, s, a, n, nullptr, (uint32_t)root), "k_sw_begin");
        ck(cudaGetLastError(), "k_sw_begin");
        run_levels(a, backward);
    }

    // One visit from all components' pivots, inside the components.
    void visit_components(bool backward) {
        const hbl::Level a = level_args(backward, true);
        ck(cudaMemsetAsync(d_dist, 0xff, n * 4, s), "cudaMemsetAsync");
        ck(cudaMemsetAsync(d_visited, 0, (n + 31) / 32 * 4, s), "cudaMemsetAsync");
        ck(cudaMemsetAsync(d_ctl, 0, sizeof *d_ctl, s), "cudaMemsetAsync");
        ck(hbl::launch_starts<false>(a, d_pivot, ncomp, 0, true, sms, s), "k_starts");
        run_levels(a, backward);
    }

    // argmax / argmin over nodes (filter 0: bounds fa, fb not met; 1 radial; 2
    // none); the start stays in d_scr->pick
    void select(const u64* val, const u64* tie, bool maximize, int filter, const u64* fa, const u64* fb,
                u64* host = nullptr) {
        ck(hbl::chain(hbs::k_sw_select, blocks(n), hbs::SW_THREADS, 0, s, n, val, tie, d_off, maximize ? 1 : 0, filter, fa, fb,
                                                              d_radial, d_best, d_scr, host), "k_sw_select");
        ck(cudaGetLastError(), "k_sw_select");
    }

    // the node of the largest out-degree
    u64 largest() {
        select(nullptr, nullptr, true, 2, nullptr, nullptr, &h_res->start);
        sync();
        return h_res->start;
    }

    // The strongly connected components of a directed graph, numbered in a
    // reverse topological order (sccs/tarjan.rs numbers them as Tarjan's
    // algorithm emits them). The component of the largest out-degree node
    // is found on the device, as the nodes that both reach it and are reached
    // from it (two visits). The other nodes are split into those reached from it
    // (their components can only lead to components reached from it) and the
    // rest (whose components can lead to everything). Tarjan's algorithm runs
    // on each part alone, on the host, the first part numbered first, then the
    // pivot's component, then the rest: every arc between components goes
    // from a higher number to a lower one, as in Tarjan's numbering. The
    // numbering of the reference matters only when two components share the
    // largest size (computer.rs:498-506 takes the first); then the whole
    // graph goes through Tarjan's algorithm in node order instead.
    std::vector<uint32_t> directed_components(const HostCsr& hg) {
        const u64 p = largest();
        std::vector<uint32_t> fw(n), bw(n);
        visit(p, false);
        ck(cudaMemcpyAsync(fw.data(), d_dist, n * 4, cudaMemcpyDeviceToHost, s), "cudaMemcpyAsync");
        visit(p, true);
        ck(cudaMemcpyAsync(bw.data(), d_dist, n * 4, cudaMemcpyDeviceToHost, s), "cudaMemcpyAsync");
        sync();
        // group 0: reached from p only; 1: the component of p; 2: the rest
        std::vector<uint8_t> group(n);
        for (u64 v = 0; v < n; v++) {
            const bool f = fw[v] != hbs::INF, b = bw[v] != hbs::INF;
            group[v] = f && b ? 1 : f ? 0 : 2;
        }
        std::vector<uint32_t> comp(n, 0);
        u64 nc = 0;
        tarjan_into(hg, comp, nc, group.data(), 0);
        const uint32_t pc = (uint32_t)nc++;
        for (u64 v = 0; v < n; v++)
            if (group[v] == 1) comp[v] = pc;
        tarjan_into(hg, comp, nc, group.data(), 2);
        std::vector<u64> sizes(nc, 0);
        for (u64 v = 0; v < n; v++) sizes[comp[v]]++;
        const u64 big = *std::max_element(sizes.begin(), sizes.end());
        if (std::count(sizes.begin(), sizes.end(), big) > 1) return tarjan(hg, ncomp);
        ncomp = nc;
        return comp;
    }

    // The components of a symmetric graph: the one of the largest-degree
    // node from one device visit, the others on the host (symm_seq.rs). The
    // numbering (symm_seq.rs numbers by smallest node) matters only when two
    // components share the largest size; then all of them come from the host
    // in the reference's order.
    std::vector<uint32_t> symmetric_components(const HostCsr& hg) {
        const u64 p = largest();
        std::vector<uint32_t> d(n);
        visit(p, false);
        ck(cudaMemcpyAsync(d.data(), d_dist, n * 4, cudaMemcpyDeviceToHost, s), "cudaMemcpyAsync");
        sync();
        std::vector<uint32_t> comp(n, 0xffffffffu);
        u64 nc = 0;
        for (u64 v = 0; v < n; v++)
            if (d[v] != hbs::INF) comp[v] = 0;
        nc = 1;
        symm_into(hg, comp, nc);
        std::vector<u64> sizes(nc, 0);
        for (u64 v = 0; v < n; v++) sizes[comp[v]]++;
        const u64 big = *std::max_element(sizes.begin(), sizes.end());
        if (std::count(sizes.begin(), sizes.end(), big) > 1) return symm_components(hg, ncomp);
        ncomp = nc;
        return comp;
    }

    // The arcs between components (comp, and d_comp on the device), in arc order.
    // A host pass over every arc took 5.9 ms on a web-like graph of 2.6 M arcs.
    // The list and its counts stand in the bounds' arrays, which are set later;
    // what does not fit there is allocated, up to LISTED arcs (an acyclic graph
    // lists all of its arcs, 8 bytes each here and 16 on the host). False: more,
    // or no room, and nothing is listed.
    static constexpr u64 LISTED = 1ull << 27;
    bool cross_arcs(std::vector<uint32_t>& src, std::vector<uint32_t>& dst) {
        const u64 nt = hbk::arc_tiles(m);
        if (nt == 0) return true;
        struct Temp {
            std::vector<void*> ps;
            ~Temp() {
                for (void* p : ps) cudaFree(p);
            }
        } temp;
        // `count` words in `place` (n of 64 bits), or else in an allocation
        auto get = [&](auto** p, u64 count, u64* place) {
            using T = std::remove_reference_t<decltype(**p)>;
            if (count * sizeof(T) <= n * 8) {
                *p = reinterpret_cast<T*>(place);
                return true;
            }
            void* q = nullptr;
            const cudaError_t e = hbk::fail_allocation() ? cudaErrorMemoryAllocation : cudaMalloc(&q, count * sizeof(T));
            if (e == cudaErrorMemoryAllocation) {
                cudaGetLastError();
                return false;
            }
            ck(e, "cudaMalloc");
            temp.ps.push_back(q);
            *p = static_cast<T*>(q);
            return true;
        };
        uint32_t *tile = nullptr, *d_src = nullptr, *d_dst = nullptr;
        unsigned long long *count = nullptr, *scratch = nullptr;
        u64* at = nullptr;
        const u64 sl = hbk::scan_scratch_len(nt + 1);
        if (!get(&tile, nt, d_fl) || !get(&count, nt + 1, d_fh) || !get(&at, nt + 1, d_bl) || !get(&scratch, sl, d_bh))
            return false;
        auto launch = [&](int e, const char* what) { ck((cudaError_t)e, what); };
        ck(cudaMemsetAsync(count + nt, 0, 8, s), "cudaMemsetAsync");
        launch(hbk::launch_tile_start(d_off, n, tile, s), "k_tile_start");
        launch(hbk::launch_cross_arcs(d_off, n, m, tile, d_succ, d_comp, count, nullptr, nullptr, nullptr, s), "k_cross_arcs");
        launch(hbk::launch_exclusive_scan_u64(count, at, nt + 1, scratch, sl, s), "scan");
        u64 total = 0;
        ck(cudaMemcpyAsync(&total, at + nt, 8, cudaMemcpyDeviceToHost, s), "cudaMemcpyAsync");
        sync();
        if (total == 0) return true;
        if (total > LISTED || !get(&d_src, total, d_ft) || !get(&d_dst, total, d_bt)) return false;
        launch(hbk::launch_cross_arcs(d_off, n, m, tile, d_succ, d_comp, count, at, d_src, d_dst, s), "k_cross_arcs");
        src.resize(total);
        dst.resize(total);
        ck(cudaMemcpyAsync(src.data(), d_src, total * 4, cudaMemcpyDeviceToHost, s), "cudaMemcpyAsync");
        ck(cudaMemcpyAsync(dst.data(), d_dst, total * 4, cudaMemcpyDeviceToHost, s), "cudaMemcpyAsync");
        sync();
        return true;
    }

    // computer.rs:487-542
    void compute_radial_vertices() {
        std::vector<u64> sizes(ncomp, 0);
        for (u64 v = 0; v < n; v++) sizes[comp[v]]++;
        u64 big = 0;
        for (u64 c = 1; c < ncomp; c++)
            if (sizes[c] > sizes[big]) big = c;
        u64 v = n;
        while (v > 0) {
            v--;
            if (comp[v] == big) break;
        }
        visit(v, true);
        hbs::k_sw_mark<<<blocks(n), hbs::SW_THREADS, 0, s>>>(n, d_dist, d_radial);
        ck(cudaGetLastError(), "k_sw_mark");
        sweeps++;
    }

    void radius_candidate(u64 key) {
        if (key != NONE && (key >> 32) < radius_high) {
            radius_high = key >> 32;
            radius_vertex = key & 0xffffffffull;
        }
    }

    // computer.rs:554-570, 572-693: a visit from the selected start (none
    // qualified: nothing), its bound updates, and the missing counts after it
    void step(bool forward) {
        const hbl::Level a = level_args(!forward, false);
        ck(hbl::chain(hbs::k_sw_begin, blocks(n), hbs::SW_THREADS, 0, s, a, n, d_scr, 0), "k_sw_begin");
        hbs::Result& r = *h_res;
        int in = 0;
        for (int k = ahead[!forward];; k = 2) {
            levels(a, k, in);
            if (forward) {
                ck(hbl::chain(hbs::k_sw_forward, blocks(n), hbs::SW_THREADS, 0, s, n, d_dist, d_bt, d_bl, d_bh, d_fl, d_fh, d_radial,
                                                                       diameter_low, radius_high, d_scr, d_ctl, h_res), "k_sw_forward");
            } else {
                ck(hbl::chain(hbs::k_sw_backward, blocks(n), hbs::SW_THREADS, 0, s, n, d_dist, d_ft, d_fl, d_fh, d_bl, d_bh,
                                                                        d_radial, d_scr, d_ctl, h_res), "k_sw_backward");
                ck(hbl::chain(hbs::k_sw_missing, blocks(n), hbs::SW_THREADS, 0, s, n, d_fl, d_fh, d_bl, d_bh, d_radial, diameter_low,
                                                                       radius_high, 1, d_scr, d_ctl, h_res), "k_sw_missing");
            }
            ck(cudaGetLastError(), "k_sw_forward");
            sync();
            if (r.done) break;
        }
        if (r.start == NONE) return;
        learn(!forward, r.launches);
        sweeps++;
        iterations++;
        if (!forward) radius_candidate(r.key);
        if (diameter_low < r.ecc) {
            diameter_low = r.ecc;
            diameter_vertex = r.start;
        }
        if (forward && r.radial && radius_high > r.ecc) {
            radius_high = r.ecc;
            radius_vertex = r.start;
        }
    }

    // computer.rs:818-921
    void all_cc_upper_bound() {
        const u64 nc = ncomp;
        ck(cudaMemsetAsync(d_best_score, 0xff, nc * 8, s), "cudaMemsetAsync");
        ck(cudaMemsetAsync(d_best_tot, 0xff, nc * 8, s), "cudaMemsetAsync");
        ck(cudaMemsetAsync(d_pivot, 0xff, nc * 4, s), "cudaMemsetAsync");
        for (int pass = 0; pass < 3; pass++) {
            hbs::k_sw_pivot_pass<<<blocks(n), hbs::SW_THREADS, 0, s>>>(pass, n, d_comp, d_fl, d_fh, d_bl, d_bh, d_ft,
                                                                      d_bt, d_best_score, d_best_tot, d_pivot);
            ck(cudaGetLastError(), "k_sw_pivot_pass");
        }
        // distances from the pivots inside each component, both directions
        visit_components(false);
        ck(cudaMemsetAsync(d_ecc_f, 0, nc * 8, s), "cudaMemsetAsync");
        hbs::k_sw_pivot_ecc<<<blocks(n), hbs::SW_THREADS, 0, s>>>(n, d_dist, d_comp, d_ecc_f);
        ck(cudaGetLastError(), "k_sw_pivot_ecc");
        ck(cudaMemcpyAsync(d_df, d_dist, n * 4, cudaMemcpyDeviceToDevice, s), "cudaMemcpyAsync");
        visit_components(true);
        ck(cudaMemsetAsync(d_ecc_b, 0, nc * 8, s), "cudaMemsetAsync");
        hbs::k_sw_pivot_ecc<<<blocks(n), hbs::SW_THREADS, 0, s>>>(n, d_dist, d_comp, d_ecc_b);
        ck(cudaGetLastError(), "k_sw_pivot_ecc");
        ck(cudaMemcpyAsync(d_db, d_dist, n * 4, cudaMemcpyDeviceToDevice, s), "cudaMemcpyAsync");
        sweeps += 2;
        // what the passes over the component DAG read, to the host
        const u64 nconn = ctarget.size();
        std::vector<u64> ef(nc), eb(nc), fhp(nc), bhp(nc);
        std::vector<uint32_t> dfs(nconn), dbe(nconn);
        ck(cudaMemcpyAsync(ef.data(), d_ecc_f, nc * 8, cudaMemcpyDeviceToHost, s), "cudaMemcpyAsync");
        ck(cudaMemcpyAsync(eb.data(), d_ecc_b, nc * 8, cudaMemcpyDeviceToHost, s), "cudaMemcpyAsync");
        hbs::k_sw_gather64<<<blocks(nc), hbs::SW_THREADS, 0, s>>>(d_pivot, nc, d_fh, d_gather64);
        ck(cudaMemcpyAsync(fhp.data(), d_gather64, nc * 8, cudaMemcpyDeviceToHost, s), "cudaMemcpyAsync");
        hbs::k_sw_gather64<<<blocks(nc), hbs::SW_THREADS, 0, s>>>(d_pivot, nc, d_bh, d_gather64);
        ck(cudaMemcpyAsync(bhp.data(), d_gather64, nc * 8, cudaMemcpyDeviceToHost, s), "cudaMemcpyAsync");
        if (nconn) {
            hbs::k_sw_gather<<<blocks(nconn), hbs::SW_THREADS, 0, s>>>(d_cstart, nconn, d_df, d_gather);
            ck(cudaMemcpyAsync(dfs.data(), d_gather, nconn * 4, cudaMemcpyDeviceToHost, s), "cudaMemcpyAsync");
            sync();
            hbs::k_sw_gather<<<blocks(nconn), hbs::SW_THREADS, 0, s>>>(d_cend, nconn, d_db, d_gather);
            ck(cudaMemcpyAsync(dbe.data(), d_gather, nconn * 4, cudaMemcpyDeviceToHost, s), "cudaMemcpyAsync");
        }
        ck(cudaGetLastError(), "k_sw_gather");
        sync();
        // computer.rs:829-873: forward bounds in component order (children
        // first), backward bounds in reverse order (parents first)
        for (u64 c = 0; c < nc; c++) {
            const u64 e1 = c + 1 < nc ? seg[c + 1] : nconn;
            for (u64 k = seg[c]; k < e1; k++) {
                ef[c] = std::max(ef[c], (u64)dfs[k] + 1 + dbe[k] + ef[ctarget[k]]);
                if (ef[c] >= fhp[c]) {
                    ef[c] = fhp[c];
                    break;
                }
            }
        }
        for (u64 c = nc; c-- > 0;) {
            const u64 e1 = c + 1 < nc ? seg[c + 1] : nconn;
            for (u64 k = seg[c]; k < e1; k++) {
                const u64 t = ctarget[k];
                eb[t] = std::max(eb[t], (u64)dfs[k] + 1 + dbe[k] + eb[c]);
                if (eb[t] >= bhp[t]) eb[t] = bhp[t];
            }
        }
        ck(cudaMemcpyAsync(d_ef, ef.data(), nc * 8, cudaMemcpyHostToDevice, s), "cudaMemcpyAsync");
        ck(cudaMemcpyAsync(d_eb, eb.data(), nc * 8, cudaMemcpyHostToDevice, s), "cudaMemcpyAsync");
        hbs::k_sw_refine<<<blocks(n), hbs::SW_THREADS, 0, s>>>(n, d_comp, d_df, d_db, d_ef, d_eb, d_fl, d_fh, d_bh,
                                                              d_radial, &d_scr->key);
        ck(cudaGetLastError(), "k_sw_refine");
        unsigned long long* key = reinterpret_cast<unsigned long long*>(&h_res->key);
        ck(cudaMemcpyAsync(key, &d_scr->key, 8, cudaMemcpyDeviceToHost, s), "cudaMemcpyAsync");
        ck(cudaMemsetAsync(&d_scr->key, 0xff, 8, s), "cudaMemsetAsync");
        sync();
        radius_candidate(*key);
        iterations += 3;
        ck(hbl::chain(hbs::k_sw_missing, blocks(n), hbs::SW_THREADS, 0, s, n, d_fl, d_fh, d_bl, d_bh, d_radial, diameter_low,
                                                               radius_high, 0, d_scr, d_ctl, h_res), "k_sw_missing");
        ck(cudaGetLastError(), "k_sw_missing");
        sync();
    }

    // computer.rs:929-1015
    u64 missing() {
        const uint64_t* c = h_res->count;  // of the last step
        const u64 mr = c[0], mdf = c[1], mdb = c[2], maf = c[3], mab = c[4];
        if (mr == 0 && radius_it == NONE) radius_it = iterations;
        if ((mdf == 0 || mdb == 0) && diameter_it == NONE) diameter_it = iterations;
        if (maf == 0 && forward_it == NONE) forward_it = iterations;
        if (maf == 0 && mab == 0) all_it = iterations;
        switch (level) {
            case HB_SWEEP_RADIUS: return mr;
            case HB_SWEEP_DIAMETER: return std::min(mdf, mdb);
            case HB_SWEEP_RADIUS_DIAMETER: return mr + std::min(mdf, mdb);
            case HB_SWEEP_ALL_FORWARD: return maf;
            default: return mab + maf;
        }
    }

    // computer.rs:282-409
    void compute() {
        if (compute_radial) compute_radial_vertices();
        select(nullptr, nullptr, true, 2, nullptr, nullptr);
        step(true);
        for (int i = 2; i <= 6; i++) {
            if (i % 2 == 0) {
                select(d_bt, d_bl, true, 0, d_bl, d_bh);
                step(false);
            } else {
                select(d_ft, d_fl, true, 0, d_fl, d_fh);
                step(true);
            }
        }
        double points[5];
        for (double& p : points) p = (double)n;
        u64 miss = missing();
        while (miss > 0) {
            int st = 0;
            for (int i = 1; i < 5; i++)
                if (points[i] > points[st]) st = i;
            switch (st) {
                case 0: all_cc_upper_bound(); break;
                case 1:
                    select(d_fh, d_ft, true, 0, d_fl, d_fh);
                    step(true);
                    break;
                case 2:
                    select(d_fl, d_ft, false, 1, nullptr, nullptr);
                    step(true);
                    break;
                case 3:
                    select(d_bh, d_bt, true, 0, d_bl, d_bh);
                    step(false);
                    break;
                default:
                    select(d_bt, d_bh, true, 0, d_bl, d_bh);
                    step(false);
                    break;
            }
            const u64 old = miss;
            miss = missing();
            if (miss > old) fail(HB_ERR_CUDA, "ExactSumSweep: the number of missing nodes grew");
            points[st] = (double)(old - miss);
            for (int i = 0; i < 5; i++)
                if (i != st && points[i] >= 0.0) points[i] += 2.0 / (double)iterations;
        }
    }
};

int run(const hb_graph_view* g, const hb_graph_view* t, int level, const uint8_t* radial, int device,
        void* stream, uint64_t* fecc, uint64_t* becc, hb_sweep_result* out) {
    if (!g || !out) fail(HB_ERR_INVALID, "graph and out must not be NULL");
    if (level < HB_SWEEP_ALL || level > HB_SWEEP_RADIUS) fail(HB_ERR_INVALID, "level must be 0..4");
    const u64 n = g->num_nodes, m = g->num_arcs;
    if (!g->offsets || (m && !g->successors)) fail(HB_ERR_INVALID, "graph arrays must not be NULL");
    if (n >= 0xffffffffull) fail(HB_ERR_INVALID, "node ids must fit u32");
    if (g->offsets[0] != 0 || g->offsets[n] != m)
        fail(HB_ERR_INVALID, "offsets[0] must be 0 and offsets[num_nodes] must equal num_arcs");
    if (t) {
        if (t->num_nodes != n || t->num_arcs != m) fail(HB_ERR_INVALID, "the transpose must have the graph's nodes and arcs");
        if (!t->offsets || (m && !t->successors)) fail(HB_ERR_INVALID, "transpose arrays must not be NULL");
        if (t->offsets[0] != 0 || t->offsets[n] != m)
            fail(HB_ERR_INVALID, "offsets[0] must be 0 and offsets[num_nodes] must equal num_arcs");
    }
    Sweeper w;
    w.undirected = t == nullptr;
    // computer.rs:109-114: a symmetric graph has only forward eccentricities
    w.level = (w.undirected && level == HB_SWEEP_ALL) ? HB_SWEEP_ALL_FORWARD : level;
    std::memset(out, 0, sizeof *out);
    static const char* kNames[] = {"All", "AllForward", "RadiusDiameter", "Diameter", "Radius"};
    if (n == 0) {
        // output_level.rs: the output builders assert that their fields were
        // computed; the first assert of each level fails on an empty graph
        const char* what = w.level == HB_SWEEP_RADIUS           ? "the radius computed"
                           : w.level == HB_SWEEP_ALL            ? "all eccentricities computed"
                           : w.level == HB_SWEEP_ALL_FORWARD    ? "all forward eccentricities computed"
                                                                : "the diameter computed";
        fail(HB_ERR_INVALID, std::string("Trying to build ") + kNames[level] + " without " + what);
    }
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        fail(HB_ERR_NO_DEVICE, "no CUDA device available (this library has no CPU path)");
    }
    w.device = device;
    w.n = n;
    w.m = m;
    ck(cudaSetDevice(device), "cudaSetDevice");
    if (stream) {
        w.s = (cudaStream_t)stream;
    } else {
        ck(cudaStreamCreateWithFlags(&w.s, cudaStreamNonBlocking), "cudaStreamCreate");
        w.own_stream = true;
    }
    cudaDeviceGetAttribute(&w.sms, cudaDevAttrMultiProcessorCount, device);
    w.grid = w.sms * 4;
    ck(cudaEventCreate(&w.ev0), "cudaEventCreate");
    ck(cudaEventCreate(&w.ev1), "cudaEventCreate");
    // HB_TRACE=1: the phases' host time on stderr
    const bool trace = std::getenv("HB_TRACE") != nullptr;
    auto t_mark = std::chrono::steady_clock::now();
    auto mark = [&](const char* what) {
        if (!trace) return;
        const auto now = std::chrono::steady_clock::now();
        std::fprintf(stderr, "hb_exact_sum_sweep %-22s %9.2f ms\n", what,
                     std::chrono::duration<double, std::milli>(now - t_mark).count());
        t_mark = now;
    };
    HostCsr hg{n, g->offsets, g->successors};
    HostCsr ht = t ? HostCsr{n, t->offsets, t->successors} : hg;
    // the graph on the device first: the components use its visits
    w.alloc(&w.d_off, n + 1);
    w.alloc(&w.d_succ, m);
    if (t) w.alloc(&w.d_tsucc, m);
    else w.d_tsucc = w.d_succ;
    for (uint32_t** p : {&w.d_dist, &w.d_queue, &w.d_comp, &w.d_df, &w.d_db}) w.alloc(p, n);
    w.alloc(&w.d_visited, (n + 31) / 32);
    for (u64** p : {&w.d_fl, &w.d_fh, &w.d_bl, &w.d_bh, &w.d_ft, &w.d_bt}) w.alloc(p, n);
    w.alloc(&w.d_radial, n);
    w.alloc(&w.d_ctl, 1);
    w.alloc(&w.d_scr, 1);
    w.alloc(&w.d_bad, 1);
    w.alloc(&w.d_best, (u64)w.grid);
    // the rest of the state, and what the components and the levels need
    w.alloc_rows(g->offsets, t ? t->offsets : nullptr);
    for (uint32_t** p : {&w.d_tile[0], &w.d_tile[1]}) w.alloc(p, hbl::tiles(n, m, w.form.lg));
    u64* d_toff = w.form.lean ? w.d_toff : reinterpret_cast<u64*>(w.d_entry);
    ck(cudaMallocHost((void**)&w.h_res, sizeof(hbs::Result) + sizeof(hbl::Control)), "cudaMallocHost");
    cudaStream_t s = w.s;
    ck(cudaMemcpyAsync(w.d_off, g->offsets, (n + 1) * 8, cudaMemcpyHostToDevice, s), "cudaMemcpyAsync");
    if (m) ck(cudaMemcpyAsync(w.d_succ, g->successors, m * 4, cudaMemcpyHostToDevice, s), "cudaMemcpyAsync");
    if (t) {
        ck(cudaMemcpyAsync(d_toff, t->offsets, (n + 1) * 8, cudaMemcpyHostToDevice, s), "cudaMemcpyAsync");
        if (m) ck(cudaMemcpyAsync(w.d_tsucc, t->successors, m * 4, cudaMemcpyHostToDevice, s), "cudaMemcpyAsync");
    }
    // the CSR is checked before any kernel indexes with it
    {
        int bad = 0;
        int* d_bad = w.d_bad;
        ck(cudaMemsetAsync(d_bad, 0, 4, s), "cudaMemsetAsync");
        ck(cudaMemsetAsync(w.d_scr, 0, sizeof *w.d_scr, s), "cudaMemsetAsync");
        ck(cudaMemsetAsync(&w.d_scr->key, 0xff, 8, s), "cudaMemsetAsync");
        hbs::k_sw_validate<<<w.blocks(std::max(n, m)), hbs::SW_THREADS, 0, s>>>(w.d_off, w.d_succ, n, m, d_bad);
        if (t) hbs::k_sw_validate<<<w.blocks(std::max(n, m)), hbs::SW_THREADS, 0, s>>>(d_toff, w.d_tsucc, n, m, d_bad);
        ck(cudaGetLastError(), "k_sw_validate");
        ck(cudaMemcpyAsync(&bad, d_bad, 4, cudaMemcpyDeviceToHost, s), "cudaMemcpyAsync");
        w.sync();
        if (bad) fail(HB_ERR_INVALID, "graph has decreasing offsets or successors >= num_nodes");
    }
    if (!w.form.lean) {
        hbl::k_info<<<w.blocks(n), hbs::SW_THREADS, 0, s>>>(w.d_off, n, w.d_info);
        if (t) hbl::k_info<<<w.blocks(n), hbs::SW_THREADS, 0, s>>>(d_toff, n, w.d_tinfo);
        ck(cudaGetLastError(), "k_info");
    }
    mark("device graph");
    // components and the arcs between them
    if (w.undirected) w.comp = w.symmetric_components(hg);
    else w.comp = w.directed_components(hg);
    w.seg.assign(w.ncomp, 0);
    ck(cudaMemcpyAsync(w.d_comp, w.comp.data(), n * 4, cudaMemcpyHostToDevice, s), "cudaMemcpyAsync");
    mark("components");
    if (!w.undirected) {
        // scc_graph.rs:118-227: of the arcs between two components the one with the
        // largest value; a component's arcs in arc order, as the reference meets them
        std::vector<uint32_t> bs(w.ncomp, 0xffffffffu), be(w.ncomp, 0);
        std::vector<uint32_t> children;
        auto value = [&](u64 a, u64 b) { return ht.deg(a) + hg.deg(b); };
        auto meet = [&](uint32_t v, uint32_t x) {
            const uint32_t xc = w.comp[x];
            if (bs[xc] == 0xffffffffu) {
                bs[xc] = v;
                be[xc] = x;
                children.push_back(xc);
            }
            if (value(v, x) > value(bs[xc], be[xc])) {
                bs[xc] = v;
                be[xc] = x;
            }
        };
        auto close = [&](u64 c) {
            w.seg[c] = w.ctarget.size();
            for (uint32_t ch : children) {
                w.ctarget.push_back(ch);
                w.cstart.push_back(bs[ch]);
                w.cend.push_back(be[ch]);
                bs[ch] = 0xffffffffu;
            }
            children.clear();
        };
        // keys grouped by component, each group in order
        auto grouped = [&](u64 count, auto&& comp_of, auto& order) {
            std::vector<u64> first(w.ncomp + 1, 0);
            for (u64 k = 0; k < count; k++) first[comp_of(k) + 1]++;
            for (u64 c = 0; c < w.ncomp; c++) first[c + 1] += first[c];
            std::vector<u64> at(first.begin(), first.end() - 1);
            order.resize(count);
            for (u64 k = 0; k < count; k++) order[at[comp_of(k)]++] = k;
            return first;
        };
        std::vector<uint32_t> src, dst;
        if (w.cross_arcs(src, dst)) {
            std::vector<u64> order;
            const auto first = grouped(src.size(), [&](u64 k) { return w.comp[src[k]]; }, order);
            for (u64 c = 0; c < w.ncomp; c++) {
                for (u64 k = first[c]; k < first[c + 1]; k++) meet(src[order[k]], dst[order[k]]);
                close(c);
            }
        } else {
            // node by node, with nothing kept for an arc
            std::vector<uint32_t> members;
            const auto first = grouped(n, [&](u64 v) { return w.comp[v]; }, members);
            for (u64 c = 0; c < w.ncomp; c++) {
                for (u64 k = first[c]; k < first[c + 1]; k++) {
                    const uint32_t v = members[k];
                    for (u64 e = hg.off[v]; e < hg.off[v + 1]; e++)
                        if (w.comp[hg.succ[e]] != c) meet(v, hg.succ[e]);
                }
                close(c);
            }
        }
    }
    mark("component arcs");
    const u64 nc = w.ncomp, nconn = w.ctarget.size();
    w.alloc(&w.d_ecc_f, nc);
    w.alloc(&w.d_ecc_b, nc);
    w.alloc(&w.d_best_score, nc);
    w.alloc(&w.d_best_tot, nc);
    w.alloc(&w.d_pivot, nc);
    w.alloc(&w.d_ef, nc);
    w.alloc(&w.d_eb, nc);
    w.alloc(&w.d_gather64, nc);
    w.alloc(&w.d_cstart, nconn);
    w.alloc(&w.d_cend, nconn);
    w.alloc(&w.d_gather, nconn);
    if (nconn) {
        ck(cudaMemcpyAsync(w.d_cstart, w.cstart.data(), nconn * 4, cudaMemcpyHostToDevice, s), "cudaMemcpyAsync");
        ck(cudaMemcpyAsync(w.d_cend, w.cend.data(), nconn * 4, cudaMemcpyHostToDevice, s), "cudaMemcpyAsync");
    }
    // computer.rs:213-240: lower bounds 0, upper bounds n, totals 0
    ck(cudaMemsetAsync(w.d_fl, 0, n * 8, s), "cudaMemsetAsync");
    ck(cudaMemsetAsync(w.d_bl, 0, n * 8, s), "cudaMemsetAsync");
    ck(cudaMemsetAsync(w.d_ft, 0, n * 8, s), "cudaMemsetAsync");
    ck(cudaMemsetAsync(w.d_bt, 0, n * 8, s), "cudaMemsetAsync");
    hbs::k_sw_fill64<<<w.blocks(n), hbs::SW_THREADS, 0, s>>>(w.d_fh, n, n);
    hbs::k_sw_fill64<<<w.blocks(n), hbs::SW_THREADS, 0, s>>>(w.d_bh, n, n);
    ck(cudaGetLastError(), "k_sw_fill64");
    if (radial) {
        ck(cudaMemcpyAsync(w.d_radial, radial, n, cudaMemcpyHostToDevice, s), "cudaMemcpyAsync");
        w.compute_radial = false;
    } else {
        ck(cudaMemsetAsync(w.d_radial, 0, n, s), "cudaMemsetAsync");
    }
    w.sync();
    mark("device state");
    ck(cudaEventRecord(w.ev0, s), "cudaEventRecord");
    w.compute();
    ck(cudaEventRecord(w.ev1, s), "cudaEventRecord");
    w.sync();
    mark("visits and bounds");
    cudaEventElapsedTime(&w.device_ms, w.ev0, w.ev1);
    // output_level.rs: what each level reports, and its asserts
    out->diameter = w.diameter_low;
    out->radius = w.radius_high;
    out->diametral_vertex = w.diameter_vertex;
    out->radial_vertex = w.radius_vertex;
    out->radius_iterations = w.radius_it;
    out->diameter_iterations = w.diameter_it;
    out->forward_iterations = w.forward_it;
    out->all_iterations = w.all_it;
    out->sweeps = w.sweeps;
    out->device_ms = w.device_ms;
    const int lv = w.level;
    auto need = [&](bool ok, const char* what) {
        if (!ok) fail(HB_ERR_INVALID, std::string("Trying to build ") + kNames[level] + " without " + what);
    };
    if (lv == HB_SWEEP_ALL) need(w.all_it != NONE, "all eccentricities computed");
    if (lv == HB_SWEEP_ALL || lv == HB_SWEEP_ALL_FORWARD) need(w.forward_it != NONE, "all forward eccentricities computed");
    if (lv != HB_SWEEP_RADIUS) need(w.diameter_it != NONE, "the diameter computed");
    if (lv != HB_SWEEP_DIAMETER) need(w.radius_it != NONE, "the radius computed");
    if (fecc && (lv == HB_SWEEP_ALL || lv == HB_SWEEP_ALL_FORWARD))
        ck(cudaMemcpyAsync(fecc, w.d_fl, n * 8, cudaMemcpyDeviceToHost, s), "cudaMemcpyAsync");
    if (becc && lv == HB_SWEEP_ALL)
        ck(cudaMemcpyAsync(becc, w.d_bh, n * 8, cudaMemcpyDeviceToHost, s), "cudaMemcpyAsync");
    w.sync();
    return HB_OK;
}

}  // namespace

extern "C" {

int hb_exact_sum_sweep(const hb_graph_view* graph, const hb_graph_view* transpose, int level,
                       const uint8_t* radial_vertices, int device, void* stream, uint64_t* forward_eccentricities,
                       uint64_t* backward_eccentricities, hb_sweep_result* out) {
    nvtxRangePushA("hb_exact_sum_sweep");
    struct Pop {
        ~Pop() { nvtxRangePop(); }
    } pop;
    try {
        return run(graph, transpose, level, radial_vertices, device, stream, forward_eccentricities,
                   backward_eccentricities, out);
    } catch (const SweepError& e) {
        t_sweep_err = e.msg;
        return e.code;
    } catch (const std::bad_alloc&) {
        t_sweep_err = "host allocation failed";
        return HB_ERR_OOM;
    }
}

const char* hb_sweep_last_error(void) { return t_sweep_err.c_str(); }

}  // extern "C"
