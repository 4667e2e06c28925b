// Breadth-first visits on the device: the GB300 counterpart of the
// reference's fair parallel breadth-first visit (ParFair,
// src/algo/visits/breadth_first/par_fair.rs:92-330) and, run root by root,
// of the sequential one (seq.rs:113-224).
//
// State: the graph in device CSR, a visited bitmap that persists across
// visits until hb_visit_reset (par_fair.rs:101, 322-324), and a queue that
// holds every node visited since the last reset in visit order, with its
// predecessor and distance. A visit is level-synchronous like the reference's
// frontier loop (par_fair.rs:169-213): hbl::k_starts marks the roots not yet
// visited, hbl::k_level (visit_level.cuh) claims a level's successors; levels are
// launched as many at a time as the last visit took, and the host looks when
// they are through.
// The Unknown events of the reference (node, pred, distance) are the queue
// slots of the visit; Known events are counted. Within a level the order is
// unspecified, as in the reference's parallel visit; distances are exact, and
// the predecessor of a node is a node of the previous level with an arc to it.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "hb_internal.h"
#include "visit_level.cuh"

namespace hbv {

__global__ void k_visit_validate(const uint64_t* __restrict__ off, const uint32_t* __restrict__ succ,
                                 uint64_t n, uint64_t m, int* bad) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t t0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (uint64_t v = t0; v < n; v += stride)
        if (off[v] > off[v + 1]) *bad = 1;
    for (uint64_t x = t0; x < m; x += stride)
        if (succ[x] >= n) *bad = 1;
}

}  // namespace hbv

struct hb_visit {
    int device = 0;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    uint64_t n = 0, m = 0;
    void* block = nullptr;         // holds the arrays below
    hbl::Form form{false, hbl::UNIT_LG};
    uint64_t* d_off = nullptr;     // (wide form: only while the handle is made)
    uint32_t* d_succ = nullptr;
    hbl::Entry* d_info = nullptr;  // (wide form)
    uint32_t* d_visited = nullptr;
    uint32_t* d_queue = nullptr;   // every node visited since the last reset, in visit order,
    hbl::Entry* d_entry = nullptr; // its entry in its level (wide form)
    uint32_t* d_unit = nullptr;    // or the units before it there (lean form),
    uint32_t* d_tile[2] = {nullptr, nullptr};
    uint32_t* d_qpred = nullptr;   // its predecessor
    uint32_t* d_qdist = nullptr;   // and distance (wide form; lean: hbl::end_of_level)
    uint32_t* d_dist = nullptr;    // hb_visit_each: distances by node where d_qpred is the predecessors (lean form)
    uint32_t* d_roots = nullptr;   // a piece of the roots of the current visit
    hbl::Control* d_ctl = nullptr;
    hbl::Control* h_ctl = nullptr; // page-locked copy
    int* d_bad = nullptr;
    int ahead = 2;                 // level launches of the next visit
    uint64_t tail = 0;
    int sms = 1;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    std::vector<uint32_t> host_visited;    // copy of d_visited (visit_each)
    std::string err;
};

static thread_local std::string t_visit_err;

static int visit_err(hb_visit* v, int code, const std::string& msg) {
    if (v) v->err = msg;
    t_visit_err = msg;
    return code;
}

static int visit_cuda(hb_visit* v, cudaError_t e, const char* what) {
    if (e == cudaSuccess) return HB_OK;
    cudaGetLastError();
    const int code = e == cudaErrorMemoryAllocation ? HB_ERR_OOM
                     : (e == cudaErrorNoDevice || e == cudaErrorInsufficientDriver) ? HB_ERR_NO_DEVICE
                                                                                     : HB_ERR_CUDA;
    return visit_err(v, code, std::string(what) + ": " + cudaGetErrorString(e));
}

#define VC(v, call, what)                               \
    do {                                                \
        int _r = visit_cuda((v), (call), (what));       \
        if (_r) return _r;                              \
    } while (0)

// The roots that go to the device at once: every node's, or 16 MB of them (their
// copy takes ten times the wait between two pieces).
static uint64_t root_piece(uint64_t n) { return std::max<uint64_t>(std::min<uint64_t>(n, 1u << 22), 1); }

// The arrays of a visit, all in one allocation: a handle of 3e5 nodes takes 0.40
// ms to make and 0.26 to free, with an allocation for each array 0.66 and 0.50
// (4e6 nodes: 1.5 and 0.40 instead of 1.8 and 0.79). Places them from `base` on
// (null: nowhere yet) and returns their bytes. In the wide form the offsets stand
// where the entries come once k_info has read them.
static size_t visit_layout(hb_visit* v, const hbl::Form& f, char* base) {
    const uint64_t n = v->n, m = v->m, rows = (n + 1) * 8;
    size_t total = 0;
    auto place = [&](auto** p, uint64_t bytes) {
        if (base) *p = reinterpret_cast<std::remove_reference_t<decltype(*p)>>(base + total);
        total += (std::max<uint64_t>(bytes, 1) + 255) / 256 * 256;
    };
    place(&v->d_succ, m * 4);
    place(&v->d_off, f.lean ? rows : std::max<uint64_t>(n * sizeof(hbl::Entry), rows));
    if (f.lean) {
        place(&v->d_unit, n * 4);
    } else {
        v->d_entry = reinterpret_cast<hbl::Entry*>(v->d_off);
        place(&v->d_info, n * sizeof(hbl::Entry));
        place(&v->d_qdist, n * 4);
    }
    place(&v->d_visited, (n + 31) / 32 * 4);
    place(&v->d_queue, n * 4);
    place(&v->d_qpred, n * 4);
    place(&v->d_roots, root_piece(n) * 4);
    place(&v->d_tile[0], hbl::tiles(n, m, f.lg) * 4);
    place(&v->d_tile[1], hbl::tiles(n, m, f.lg) * 4);
    place(&v->d_ctl, sizeof(hbl::Control));
    place(&v->d_bad, sizeof(int));
    return total;
}

static cudaError_t visit_alloc(hb_visit* v, const uint64_t* off) {
    const uint64_t n = v->n, m = v->m;
    const hbl::Form lean = hbl::choose_form(n, m, UINT64_MAX, 0, 0);
    const size_t wide = visit_layout(v, hbl::Form{false, hbl::UNIT_LG}, nullptr);
    const size_t more = wide - visit_layout(v, lean, nullptr);
    size_t free_bytes = 0, all = 0;
    if (more > hbl::WIDE_BYTES)
        if (const cudaError_t e = cudaMemGetInfo(&free_bytes, &all); e != cudaSuccess) return e;
    v->form = hbl::choose_form(n, m, hbl::longest_row(off, n, m), more, free_bytes);
    cudaError_t e = hbk::fail_allocation() ? cudaErrorMemoryAllocation
                                           : cudaMalloc(&v->block, visit_layout(v, v->form, nullptr));
    if (e == cudaErrorMemoryAllocation && !v->form.lean) {
        cudaGetLastError();
        v->form = lean;
        e = hbk::fail_allocation() ? cudaErrorMemoryAllocation : cudaMalloc(&v->block, visit_layout(v, lean, nullptr));
    }
    if (e == cudaSuccess) visit_layout(v, v->form, (char*)v->block);
    return e;
}

// One visit from the given roots; dist and pred (by node, device) get its
// nodes' entries, or are null. They may stand where the queue's predecessors and
// distances do, which are then not written. On return the stream is idle.
static int visit_levels(hb_visit* v, const uint64_t* roots, size_t nroots, uint64_t max_distance, uint32_t* dist,
                        uint32_t* pred, hb_visit_stats& st) {
    if (nroots == 0) return HB_OK;
    cudaStream_t s = v->stream;
    const uint64_t q0 = v->tail;
    hbl::Level a{};
    a.info = v->d_info;
    a.off = v->form.lean ? v->d_off : nullptr;
    a.lg = v->form.lg;
    a.succ = v->d_succ;
    a.visited = v->d_visited;
    a.dist = dist;
    a.pred = pred;
    a.queue = v->d_queue;
    a.entry = v->d_entry;
    a.unit = v->d_unit;
    auto unless_by_node = [&](uint32_t* p) { return p == dist || p == pred ? nullptr : p; };
    a.qpred = unless_by_node(v->d_qpred);
    a.qdist = unless_by_node(v->d_qdist);
    a.ctl = v->d_ctl;
    a.max_d = (uint32_t)std::min<uint64_t>(max_distance, 0xffffffffull);
    a.tile[0] = v->d_tile[0];
    a.tile[1] = v->d_tile[1];
    a.n = v->n;
    a.small = hbl::small_units(v->n, v->m, v->form.lg);
    std::vector<uint32_t> r32(nroots);
    for (size_t i = 0; i < nroots; i++) r32[i] = (uint32_t)roots[i];
    *v->h_ctl = hbl::Control{};
    v->h_ctl->tail = q0;
    VC(v, cudaMemcpyAsync(v->d_ctl, v->h_ctl, sizeof(hbl::Control), cudaMemcpyHostToDevice, s), "cudaMemcpyAsync");
    VC(v, cudaEventRecord(v->ev0, s), "cudaEventRecord");
    // d_roots holds root_piece(n) roots: longer lists go in pieces
    const uint64_t nr = std::min<uint64_t>(nroots, root_piece(v->n));
    for (size_t at = 0; at < nroots; at += nr) {
        const uint64_t k = std::min<uint64_t>(nr, nroots - at);
        // the next piece's copy must not overwrite roots still being read
        if (at) VC(v, cudaStreamSynchronize(s), "cudaStreamSynchronize");
        VC(v, cudaMemcpyAsync(v->d_roots, r32.data() + at, k * 4, cudaMemcpyHostToDevice, s), "cudaMemcpyAsync");
        VC(v, hbl::launch_starts<true>(a, v->d_roots, k, (uint32_t)q0, at + nr >= nroots, v->sms, s), "k_starts");
    }
    // levels, as many launches as the last visit took; one past the last level does nothing
    int in = 0;
    for (int k = v->ahead;; k = 2) {
        VC(v, (hbl::launch_levels<false, true>(a, k, in, v->sms, s)), "k_level");
        VC(v, cudaEventRecord(v->ev1, s), "cudaEventRecord");
        VC(v, cudaMemcpyAsync(v->h_ctl, v->d_ctl, sizeof(hbl::Control), cudaMemcpyDeviceToHost, s), "cudaMemcpyAsync");
        VC(v, cudaStreamSynchronize(s), "cudaStreamSynchronize");
        if (hbl::done(v->h_ctl->st[0])) break;
    }
    const hbl::Control& c = *v->h_ctl;
    v->ahead = (int)std::max<uint32_t>(1, std::min<uint32_t>(c.launches, 64));
    v->tail = c.st[0].e;
    st.visited = v->tail - q0;
    st.levels = st.visited ? c.st[0].last + 1 : 0;
    st.known_arcs = c.known;
    float ms = 0.f;
    cudaEventElapsedTime(&ms, v->ev0, v->ev1);
    st.device_ms = ms;
    return HB_OK;
}

// The first k events of the visit that began at queue slot q0 and reached `count`
// nodes, into the caller's arrays (null: not wanted). On return the stream is idle.
static int visit_events(hb_visit* v, uint64_t q0, uint64_t count, uint64_t k, uint32_t* nodes, uint32_t* preds,
                        uint32_t* dists) {
    if (k == 0 || !(nodes || preds || dists)) return HB_OK;
    cudaStream_t s = v->stream;
    if (nodes)
        VC(v, cudaMemcpyAsync(nodes, v->d_queue + q0, k * 4, cudaMemcpyDeviceToHost, s), "cudaMemcpyAsync");
    if (preds)
        VC(v, cudaMemcpyAsync(preds, v->d_qpred + q0, k * 4, cudaMemcpyDeviceToHost, s), "cudaMemcpyAsync");
    if (dists)
        VC(v, cudaMemcpyAsync(dists, (v->form.lean ? v->d_unit : v->d_qdist) + q0, k * 4, cudaMemcpyDeviceToHost, s),
           "cudaMemcpyAsync");
    VC(v, cudaStreamSynchronize(s), "cudaStreamSynchronize");
    if (dists && v->form.lean) {
        // each expanded level's first entry is its end (hbl::end_of_level)
        uint32_t d = 0;
        for (uint64_t b = 0; b < k; d++) {
            const uint64_t e = std::min<uint64_t>(k, dists[b] ? dists[b] - q0 : count);
            std::fill(dists + b, dists + e, d);
            b = e;
        }
    }
    return HB_OK;
}

static void visit_free(hb_visit* v) {
    if (!v) return;
    cudaSetDevice(v->device);
    if (v->stream) cudaStreamSynchronize(v->stream);
    cudaFree(v->block);
    cudaFree(v->d_dist);
    if (v->h_ctl) cudaFreeHost(v->h_ctl);
    if (v->ev0) cudaEventDestroy(v->ev0);
    if (v->ev1) cudaEventDestroy(v->ev1);
    if (v->own_stream && v->stream) cudaStreamDestroy(v->stream);
    delete v;
}

extern "C" {

int hb_visit_create(const hb_graph_view* g, int device, void* stream, hb_visit** out) {
    if (!out) return visit_err(nullptr, HB_ERR_INVALID, "out is NULL");
    *out = nullptr;
    if (!g || !g->offsets || (g->num_arcs && !g->successors))
        return visit_err(nullptr, HB_ERR_INVALID, "graph arrays must not be NULL");
    if (g->num_nodes >= 0xffffffffull)
        return visit_err(nullptr, HB_ERR_INVALID, "node ids must fit u32");
    if (g->offsets[0] != 0 || g->offsets[g->num_nodes] != g->num_arcs)
        return visit_err(nullptr, HB_ERR_INVALID,
                         "offsets[0] must be 0 and offsets[num_nodes] must equal num_arcs");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        return visit_err(nullptr, HB_ERR_NO_DEVICE, "no CUDA device available (this library has no CPU path)");
    }
    hb_visit* v = new hb_visit();
    v->device = device;
    v->n = g->num_nodes;
    v->m = g->num_arcs;
    const uint64_t n = v->n, m = v->m, words = (n + 31) / 32;
    auto fail = [&](int r) {
        visit_free(v);
        return r;
    };
    int r;
    if ((r = visit_cuda(v, cudaSetDevice(device), "cudaSetDevice"))) return fail(r);
    if (stream) {
        v->stream = (cudaStream_t)stream;
    } else {
        if ((r = visit_cuda(v, cudaStreamCreateWithFlags(&v->stream, cudaStreamNonBlocking),
                            "cudaStreamCreate")))
            return fail(r);
        v->own_stream = true;
    }
    cudaDeviceGetAttribute(&v->sms, cudaDevAttrMultiProcessorCount, device);
    if ((r = visit_cuda(v, visit_alloc(v, g->offsets), "cudaMalloc")) ||
        (r = visit_cuda(v, cudaMallocHost((void**)&v->h_ctl, sizeof(hbl::Control)), "cudaMallocHost")))
        return fail(r);
    if ((r = visit_cuda(v, cudaMemcpyAsync(v->d_off, g->offsets, (n + 1) * 8, cudaMemcpyHostToDevice, v->stream),
                        "cudaMemcpyAsync")))
        return fail(r);
    if (m && (r = visit_cuda(v, cudaMemcpyAsync(v->d_succ, g->successors, m * 4, cudaMemcpyHostToDevice,
                                                v->stream),
                             "cudaMemcpyAsync")))
        return fail(r);
    // the CSR is checked before any kernel indexes with it
    int* d_bad = v->d_bad;
    int bad = 0;
    if ((r = visit_cuda(v, cudaMemsetAsync(d_bad, 0, sizeof(int), v->stream), "cudaMemsetAsync"))) return fail(r);
    const int grid = (int)std::min<uint64_t>((std::max(n, m) + 255) / 256 + 1, 8192);
    hbv::k_visit_validate<<<grid, 256, 0, v->stream>>>(v->d_off, v->d_succ, n, m, d_bad);
    if ((r = visit_cuda(v, cudaGetLastError(), "k_visit_validate")) ||
        (r = visit_cuda(v, cudaMemcpyAsync(&bad, d_bad, sizeof(int), cudaMemcpyDeviceToHost, v->stream),
                        "cudaMemcpyAsync")) ||
        (r = visit_cuda(v, cudaStreamSynchronize(v->stream), "cudaStreamSynchronize")))
        return fail(r);
    if (bad) return fail(visit_err(v, HB_ERR_INVALID, "graph has decreasing offsets or successors >= num_nodes"));
    if (!v->form.lean) {
        hbl::k_info<<<(int)std::min<uint64_t>(n / 256 + 1, 8192), 256, 0, v->stream>>>(v->d_off, n, v->d_info);
        if ((r = visit_cuda(v, cudaGetLastError(), "k_info"))) return fail(r);
    }
    v->host_visited.assign(std::max<uint64_t>(words, 1), 0);
    if ((r = visit_cuda(v, cudaEventCreate(&v->ev0), "cudaEventCreate")) ||
        (r = visit_cuda(v, cudaEventCreate(&v->ev1), "cudaEventCreate")))
        return fail(r);
    if ((r = visit_cuda(v, cudaMemsetAsync(v->d_visited, 0, std::max<uint64_t>(words, 1) * 4, v->stream),
                        "cudaMemsetAsync")) ||
        (r = visit_cuda(v, cudaStreamSynchronize(v->stream), "cudaStreamSynchronize")))
        return fail(r);
    *out = v;
    return HB_OK;
}

void hb_visit_destroy(hb_visit* v) { visit_free(v); }

int hb_visit_reset(hb_visit* v) {
    if (!v) return visit_err(nullptr, HB_ERR_INVALID, "visit is NULL");
    VC(v, cudaSetDevice(v->device), "cudaSetDevice");
    const uint64_t words = (v->n + 31) / 32;
    VC(v, cudaMemsetAsync(v->d_visited, 0, std::max<uint64_t>(words, 1) * 4, v->stream), "cudaMemsetAsync");
    VC(v, cudaStreamSynchronize(v->stream), "cudaStreamSynchronize");
    v->tail = 0;
    return HB_OK;
}

int hb_visit_run(hb_visit* v, const uint64_t* roots, size_t nroots, uint64_t max_distance,
                 uint32_t* nodes, uint32_t* preds, uint32_t* dists, size_t capacity,
                 hb_visit_stats* stats) {
    if (!v) return visit_err(nullptr, HB_ERR_INVALID, "visit is NULL");
    if (nroots && !roots) return visit_err(v, HB_ERR_INVALID, "roots is NULL");
    for (size_t i = 0; i < nroots; i++)
        if (roots[i] >= v->n) return visit_err(v, HB_ERR_INVALID, "root " + std::to_string(roots[i]) + " >= num_nodes");
    VC(v, cudaSetDevice(v->device), "cudaSetDevice");
    hb_visit_stats st{};
    const uint64_t q0 = v->tail;
    if (int r = visit_levels(v, roots, nroots, max_distance, nullptr, nullptr, st)) return r;
    const uint64_t count = st.visited;
    // the events into the caller's buffers
    if (int r = visit_events(v, q0, count, std::min<uint64_t>(capacity, count), nodes, preds, dists)) return r;
    if (stats) *stats = st;
    if (capacity < count)
        return visit_err(v, HB_ERR_INVALID, "capacity holds fewer than the " + std::to_string(count) +
                                                " events of the visit (the first ones were written)");
    return HB_OK;
}

int hb_visit_each(hb_visit* v, const uint64_t* roots, size_t nroots, uint32_t* dist, uint32_t* pred,
                  size_t len) {
    if (!v) return visit_err(nullptr, HB_ERR_INVALID, "visit is NULL");
    if ((dist && len != v->n) || (pred && len != v->n))
        return visit_err(v, HB_ERR_INVALID, "dist and pred must hold num_nodes entries");
    const uint64_t words = (v->n + 31) / 32;
    if (nroots == 0 || words == 0)
        return nroots ? visit_err(v, HB_ERR_INVALID, "root " + std::to_string(roots[0]) + " >= num_nodes") : HB_OK;
    VC(v, cudaSetDevice(v->device), "cudaSetDevice");
    cudaStream_t s = v->stream;
    VC(v, cudaMemcpyAsync(v->host_visited.data(), v->d_visited, words * 4, cudaMemcpyDeviceToHost, s),
       "cudaMemcpyAsync");
    // The caller's entries, which the visits write over by node on the device (in
    // place of a pass of scattered host writes over the events, which is left for
    // a device without room for them). They stand where the events' would.
    uint32_t *by_dist = nullptr, *by_pred = pred ? v->d_qpred : nullptr;
    bool by_node = true;
    if (dist) {
        by_dist = !v->form.lean ? v->d_qdist : !pred ? v->d_qpred : v->d_dist;
        if (!by_dist) {
            const cudaError_t e = hbk::fail_allocation() ? cudaErrorMemoryAllocation
                                                         : cudaMalloc((void**)&v->d_dist, v->n * 4);
            if (e == cudaErrorMemoryAllocation) {
                cudaGetLastError();
                v->d_dist = by_pred = nullptr;
                by_node = false;
            } else {
                VC(v, e, "cudaMalloc");
            }
            by_dist = v->d_dist;
        }
    }
    if (by_dist) VC(v, cudaMemcpyAsync(by_dist, dist, v->n * 4, cudaMemcpyHostToDevice, s), "cudaMemcpyAsync");
    if (by_pred) VC(v, cudaMemcpyAsync(by_pred, pred, v->n * 4, cudaMemcpyHostToDevice, s), "cudaMemcpyAsync");
    VC(v, cudaStreamSynchronize(s), "cudaStreamSynchronize");
    int rc = HB_OK;
    bool wrote = false;
    std::vector<uint32_t> nodes, ps, ds;
    for (size_t i = 0; i < nroots && rc == HB_OK; i++) {
        const uint64_t r = roots[i];
        if (r >= v->n) {
            rc = visit_err(v, HB_ERR_INVALID, "root " + std::to_string(r) + " >= num_nodes");
            break;
        }
        if ((v->host_visited[r >> 5] >> (r & 31)) & 1) continue;  // seq.rs:130: already visited
        hb_visit_stats st{};
        const uint64_t q0 = v->tail;
        rc = visit_levels(v, &r, 1, UINT64_MAX, by_dist, by_pred, st);
        if (!by_node && rc == HB_OK) {
            nodes.resize(st.visited);
            ps.resize(pred ? st.visited : 0);
            ds.resize(dist ? st.visited : 0);
            rc = visit_events(v, q0, st.visited, st.visited, nodes.data(), pred ? ps.data() : nullptr,
                              dist ? ds.data() : nullptr);
            for (uint64_t k = 0; k < st.visited && rc == HB_OK; k++) {
                if (dist) dist[nodes[k]] = ds[k];
                if (pred) pred[nodes[k]] = ps[k];
            }
        }
        wrote = by_node;
        if (rc != HB_OK || i + 1 == nroots) break;
        // what is visited by now, for the next roots: the bitmap, or the few nodes of a small visit
        if (st.visited > words) {
            rc = visit_cuda(v, cudaMemcpyAsync(v->host_visited.data(), v->d_visited, words * 4, cudaMemcpyDeviceToHost, s),
                            "cudaMemcpyAsync");
        } else {
            nodes.resize(st.visited);
            rc = visit_cuda(v, cudaMemcpyAsync(nodes.data(), v->d_queue + q0, st.visited * 4, cudaMemcpyDeviceToHost, s),
                            "cudaMemcpyAsync");
        }
        if (rc == HB_OK) rc = visit_cuda(v, cudaStreamSynchronize(s), "cudaStreamSynchronize");
        if (rc == HB_OK && st.visited <= words)
            for (uint32_t x : nodes) v->host_visited[x >> 5] |= 1u << (x & 31);
    }
    if (wrote) {
        int e = HB_OK;
        if (dist)
            e = visit_cuda(v, cudaMemcpyAsync(dist, by_dist, v->n * 4, cudaMemcpyDeviceToHost, s), "cudaMemcpyAsync");
        if (pred && e == HB_OK)
            e = visit_cuda(v, cudaMemcpyAsync(pred, by_pred, v->n * 4, cudaMemcpyDeviceToHost, s), "cudaMemcpyAsync");
        if (e == HB_OK) e = visit_cuda(v, cudaStreamSynchronize(s), "cudaStreamSynchronize");
        if (rc == HB_OK) rc = e;
    }
    return rc;
}

const char* hb_visit_last_error(const hb_visit* v) { return v ? v->err.c_str() : t_visit_err.c_str(); }

}  // extern "C"
