"""Performance cases of the framework: the calls a user's program makes, over
the sizes, graph kinds and options that the public entry points serve.

    listed()            the cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) inputs and handles a program has in hand before the call
    run(state)          one pass through the public API
    work(case)          bytes and operations a pass cannot do without
    exact(case, seed)   the computed outputs in 64 bits by plain torch

Graphs are drawn on the GPU from the seed alone and handed to the framework as
host CSR arrays, its input format: web-like graphs (Zipf out-degrees, mean 12,
80% of the successors near the source, 20% uniform), R-MAT (0.57, 0.19, 0.19,
0.05) and out-regular uniform graphs, the three kinds of the benchmark.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "webgraph-algo-rs_gb300"))
import hyperball_gb300 as hb  # noqa: E402

NF_ROW = 128
CAP, SHIFT, WINDOW = 100_000, 1.266, 1024  # the web-like generator's defaults


def listed():
    return [
        # HyperBall on a graph of 10^4 nodes: the parity configuration; launches and host round trips
        {"name": "er_10k_m6", "do": "run", "kind": "er", "n": 10_000, "deg": 8, "log2m": 6, "extra": "none"},
        # an ordinary crawl: a handle run on a million-node web graph, all three standard outputs
        {"name": "web_1m_m6", "do": "run", "kind": "web", "n": 1_000_003, "deg": 12, "log2m": 6, "extra": "none"},
        # a large web graph, the headline's kind and counter size
        {"name": "web_33m_m6", "do": "run", "kind": "web", "n": 33_000_001, "deg": 12, "log2m": 6, "extra": "none"},
        # a social-network-like graph with hubs and the larger counters of the R-MAT configuration
        {"name": "rmat_1m_m8", "do": "run", "kind": "rmat", "n": 1 << 20, "deg": 16, "log2m": 8, "extra": "none"},
        # precise counters, node weights and a discounted centrality
        {"name": "er_60k_m10_weights", "do": "run", "kind": "er", "n": 60_001, "deg": 12, "log2m": 10,
         "extra": "weights"},
        # the whole call, graph in host memory to centralities in host memory, log2m 8
        {"name": "call_rmat_3m_m8", "do": "call", "kind": "rmat", "n": 3_000_000, "deg": 16, "log2m": 8,
         "extra": "none"},
        # the whole call without a transpose (standard iterations only) and the derived centralities
        {"name": "call_web_200k_m5", "do": "call", "kind": "web", "n": 200_003, "deg": 12, "log2m": 5,
         "extra": "derived"},
        # a batch of small graphs with mixed counter sizes, run together
        {"name": "batch_128", "do": "batch", "kind": "web", "n": 100_000, "deg": 12, "count": 128},
        # distances from one node of a large web graph
        {"name": "visit_web_4m", "do": "visit", "kind": "web", "n": 4_000_003, "deg": 12, "far": -1},
        # a neighbourhood query: everything within distance 2 of one node
        {"name": "visit_ball_300k", "do": "visit", "kind": "web", "n": 300_007, "deg": 12, "far": 2},
        # exact radius and diameter of a directed graph
        {"name": "sweep_web_260k", "do": "sweep", "kind": "web", "n": 260_003, "deg": 12,
         "level": "radius_diameter"},
        # exact eccentricities of every node of a small symmetric graph
        {"name": "sweep_sym_3k_all", "do": "sweep", "kind": "sym", "n": 3_001, "deg": 4, "level": "all"},
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) | 1


def draw(rng):
    do = rng.choice(["run", "run", "run", "call", "call", "batch", "visit", "visit", "sweep"])
    kind = rng.choice(["web", "web", "rmat", "er"])
    deg = {"web": 12, "rmat": rng.randint(8, 16), "er": rng.randint(4, 16)}[kind]
    if do in ("run", "call"):
        log2m = rng.choice([4, 5, 6, 6, 7, 8, 8, 9, 10])
        # the counters of a drawn graph stay below those of the largest listed case
        n = _size(rng, 2_000, min(20_000_000, (1 << 30) >> log2m) if do == "run" else 3_000_000)
        extra = "none" if do == "call" and kind != "web" else rng.choice(["none", "none", "weights" if do == "run" else "derived"])
        if extra == "weights":
            n = min(n, 500_001)
        return {"do": do, "kind": kind, "n": n, "deg": deg, "log2m": log2m, "extra": extra}
    if do == "batch":
        return {"do": "batch", "kind": kind, "n": _size(rng, 5_000, 100_000), "deg": deg, "count": rng.randint(8, 128)}
    if do == "visit":
        return {"do": "visit", "kind": kind, "n": _size(rng, 20_000, 4_000_000), "deg": deg,
                "far": rng.choice([-1, -1, 1, 2, 3])}
    if rng.random() < 0.4:
        return {"do": "sweep", "kind": "sym", "n": _size(rng, 500, 3_000), "deg": rng.randint(3, 6), "level": "all"}
    return {"do": "sweep", "kind": kind, "n": _size(rng, 10_000, 200_000), "deg": deg,
            "level": rng.choice(["radius_diameter", "diameter", "radius"])}


# ---------------------------------------------------------------------------
# graphs
# ---------------------------------------------------------------------------
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _zipf_table(dev):
    k = torch.arange(1, CAP + 1, dtype=torch.float64, device=dev) + SHIFT
    w = torch.cumsum(k ** -2.1, 0)
    return w / w[-1]


def _csr(src, dst, n):
    """Sorted, duplicate-free and loop-free CSR of the arcs src -> dst."""
    keep = src != dst
    key = torch.unique(src[keep] * n + dst[keep])
    del src, dst, keep
    deg = torch.bincount(key // n, minlength=n)
    off = torch.zeros(n + 1, dtype=torch.int64, device=key.device)
    torch.cumsum(deg, 0, out=off[1:])
    return off, (key % n).to(torch.int32)


def _arcs(case, seed):
    """Device CSR (offsets int64, successors int32) of the case's graph."""
    n, deg, kind, dev = case["n"], case["deg"], case["kind"], _device()
    g = torch.Generator(device=dev)
    g.manual_seed(seed)

    def ints(hi, count):
        return torch.randint(hi, (count,), generator=g, device=dev)

    if kind == "web":
        u = torch.rand(n, generator=g, device=dev, dtype=torch.float64)
        k = torch.searchsorted(_zipf_table(dev), u) + 1
        k = torch.clamp(k, max=min(CAP, n))
        src = torch.repeat_interleave(torch.arange(n, device=dev), k)
        m = src.numel()
        near = torch.rand(m, generator=g, device=dev) < 0.8
        dst = torch.where(near, (src + ints(2 * WINDOW + 1, m) - WINDOW) % n, ints(n, m))
    elif kind == "rmat":
        scale, m = max(1, (n - 1).bit_length()), deg * n
        src = torch.zeros(m, dtype=torch.int64, device=dev)
        dst = torch.zeros(m, dtype=torch.int64, device=dev)
        for _ in range(scale):
            u = torch.rand(m, generator=g, device=dev)
            src = src * 2 + (u >= 0.76)
            dst = dst * 2 + (((u >= 0.57) & (u < 0.76)) | (u >= 0.95))
        inside = (src < n) & (dst < n)
        src, dst = src[inside], dst[inside]
    else:
        src = torch.arange(n, device=dev).repeat_interleave(deg)
        dst = ints(n, n * deg)
    if kind == "sym":
        src, dst = torch.cat([src, dst]), torch.cat([dst, src])
    return _csr(src, dst, n)


def _transpose(off, suc):
    n = off.numel() - 1
    src = torch.repeat_interleave(torch.arange(n, device=off.device), off[1:] - off[:-1])
    return _csr(suc.long(), src, n)


def _host(off, suc, pinned=False):
    """The graph as the framework takes it: host CSR behind a CsrView."""
    o, s = off.cpu(), suc.cpu()
    if pinned and torch.cuda.is_available():
        o, s = o.pin_memory(), s.pin_memory()
    return hb.CsrView(off.numel() - 1, suc.numel(), o.data_ptr(), s.data_ptr(), owner=(o, s))


def _batch_cases(case, seed):
    """Graphs of a batch: sizes log-uniform from 10^3 to n, counters 2^4, 2^6 or 2^8 (the same for every seed)."""
    r = np.random.RandomState(case["n"])
    out = []
    for _ in range(case["count"]):
        n = int(round(math.exp(r.uniform(math.log(1000), math.log(case["n"])))))
        out.append(({"kind": case["kind"], "n": n, "deg": case["deg"]}, int(r.choice([4, 6, 8])), seed * 1000 + len(out)))
    return out


def _weights(case, seed):
    return np.random.RandomState((seed + 1) & 0x7FFFFFFF).randint(1, 4, case["n"]).astype(np.uint64)


def _discount(d):
    return 1.0 / math.log2(1.0 + d)


# ---------------------------------------------------------------------------
# a pass
# ---------------------------------------------------------------------------
def _builder(case, graph, seed):
    if case["extra"] == "weights":
        b = hb.HyperBallBuilder.with_hyper_log_log(graph, None, case["log2m"])
        b.weights(_weights(case, seed), seed=seed)
        b.discount_function(_discount)
    else:
        b = hb.HyperBallBuilder.new(graph, hb.HyperLogLogBuilder(case["n"]).log_2_num_reg(case["log2m"]).build())
    b.sum_of_distances(True).sum_of_inverse_distances(True)
    if case["extra"] != "derived":
        b.transpose_on_device()
    return b


def _vector(n):
    """Page-locked host memory for a per-node result, kept by the program."""
    t = torch.empty(n, dtype=torch.float64)
    return (t.pin_memory() if torch.cuda.is_available() else t).numpy()


def prepare(case, seed):
    s = {"case": case, "seed": seed}
    do, n = case["do"], case["n"]
    if do == "batch":
        parts = _batch_cases(case, seed)
        s["graphs"] = [_host(*_arcs(c, x)) for c, _, x in parts]
        s["batch"] = hb.HyperBallBatch(s["graphs"], [l for _, l, _ in parts], sum_of_distances=True,
                                       sum_of_inverse_distances=True)
        return s
    off, suc = _arcs(case, seed)
    s["graph"] = _host(off, suc, pinned=do == "call")
    if do == "sweep":
        s["transpose"] = None if case["kind"] == "sym" else _host(*_transpose(off, suc))
    elif do == "visit":
        s["root"] = int(np.random.RandomState(seed & 0x7FFFFFFF).randint(n))
        s["visit"] = hb.ParFair(s["graph"])
        s["dist"], s["reached"] = np.full(n, -1, dtype=np.int32), np.zeros(0, dtype=np.uint32)
    else:
        s["out"] = [_vector(n) for _ in range(4)]
        if do == "run":
            s["handle"] = _builder(case, s["graph"], seed).build()
    del off, suc
    if torch.cuda.is_available():
        torch.cuda.empty_cache()  # the framework has a pool of its own
    return s


def _row(nf):
    """A neighbourhood function in a row of fixed length (a run has fewer iterations)."""
    out = np.zeros(NF_ROW)
    out[:len(nf)] = nf
    return out


def _results(h, case, out):
    r = {"nf": _row(h.neighborhood_function()), "sod": h.sum_of_distances(out=out[0]),
         "harmonic": h.harmonic_centralities(out=out[1])}
    if case["extra"] == "weights":
        r["discounted"] = h.discounted_centrality(0, out=out[2])
    elif case["extra"] == "derived":
        r["lin"] = h.lin_centrality(out=out[2])
        r["reachable"] = h.reachable_nodes(out=out[3])
    return r


def run(state):
    case = state["case"]
    do = case["do"]
    if do == "run":
        h = state["handle"]
        h.run_until_done()
        return _results(h, case, state["out"])
    if do == "call":
        with _builder(case, state["graph"], state["seed"]).build() as h:
            h.run_until_done()
            return _results(h, case, state["out"])
    if do == "batch":
        b = state["batch"]
        b.run_until_done()
        each = range(len(b))
        return {"nf": np.stack([_row(b.neighborhood_function(i)) for i in each]),
                "sod": np.concatenate([b.sum_of_distances(i) for i in each]),
                "harmonic": np.concatenate([b.harmonic_centralities(i) for i in each])}
    if do == "visit":
        v = state["visit"]
        v.reset()
        if case["far"] < 0:
            return {"dist": v.visit_each([state["root"]]).view(np.int32)}
        # into the program's own array of distances, where the last query's nodes are cleared first
        dist = state["dist"]
        dist[state["reached"]] = -1
        nodes, _, dists, st = v.par_visit([state["root"]], max_distance=case["far"])
        dist[nodes] = dists
        state["reached"] = nodes
        return {"dist": dist, "visited": st["visited"], "levels": st["levels"], "known_arcs": st["known_arcs"]}
    r = hb.exact_sum_sweep(state["graph"], state["transpose"], level=case["level"])
    out = {k: -1 if r[k] == hb.SWEEP_NONE else int(r[k])
           for k in ("diameter", "radius", "diametral_vertex", "radial_vertex", "radius_iterations",
                     "diameter_iterations", "forward_iterations", "all_iterations")}
    for k in ("forward_eccentricities", "backward_eccentricities"):
        if k in r:
            out[k] = r[k].view(np.int64)
    return out


def _full_sweeps(kind, n):
    """Iterations of a run in units of a pass over every node and arc: a web-like graph's diameter grows with its
    size, the others' hardly."""
    return 0.55 * math.log2(n) if kind == "web" else 5.0


def work(case):
    """A pass over a graph reads 8 bytes a node and 4 an arc; a full HyperBall iteration also reads every
    counter (5-bit registers), writes it and updates the two sums; results leave once."""
    do, n = case["do"], case["n"]
    m = n * case["deg"] * (2 if case["kind"] == "sym" else 1)
    graph = 8 * n + 4 * m
    if do in ("run", "call"):
        w = (1 << case["log2m"]) * 5 / 8
        total = _full_sweeps(case["kind"], n) * (graph + n * (2 * w + 32)) + 16 * n
        return {"bytes": total + (graph if do == "call" else 0), "flops": 0}
    if do == "batch":
        mean = (n - 1000) / math.log(n / 1000)  # of a log-uniform size
        each = _full_sweeps(case["kind"], mean) * ((8 + 4 * case["deg"]) * mean + mean * (2 * 70 + 32)) + 16 * mean
        return {"bytes": case["count"] * each, "flops": 0}
    if do == "visit":
        if case["far"] < 0:
            return {"bytes": graph + 4 * n, "flops": 0}
        nodes = min(n, case["deg"] ** case["far"])
        return {"bytes": 8 * nodes + 4 * nodes * case["deg"], "flops": 0}
    # a visit per sweep, and every node's bounds once per visit
    sweeps = n if case["level"] == "all" else 40
    return {"bytes": float(sweeps) * (graph + 48 * n), "flops": 0}


# ---------------------------------------------------------------------------
# the outputs of a HyperBall run in 64 bits
# ---------------------------------------------------------------------------
_M64 = (1 << 64) - 1


def _hash(x):
    """SipHash-1-3 with zero keys over the 8 bytes of each x (numpy uint64)."""
    def rot(v, b):
        return (v << np.uint64(b)) | (v >> np.uint64(64 - b))

    v0, v1, v2, v3 = (np.full(x.shape, c, dtype=np.uint64) for c in
                      (0x736f6d6570736575, 0x646f72616e646f6d, 0x6c7967656e657261, 0x7465646279746573))

    def rounds(v0, v1, v2, v3, count):
        for _ in range(count):
            v0 = v0 + v1
            v1 = rot(v1, 13) ^ v0
            v0 = rot(v0, 32)
            v2 = v2 + v3
            v3 = rot(v3, 16) ^ v2
            v0 = v0 + v3
            v3 = rot(v3, 21) ^ v0
            v2 = v2 + v1
            v1 = rot(v1, 17) ^ v2
            v2 = rot(v2, 32)
        return v0, v1, v2, v3

    for word in (x, np.uint64(8 << 56)):
        v3 = v3 ^ word
        v0, v1, v2, v3 = rounds(v0, v1, v2, v3, 1)
        v0 = v0 ^ word
    v0, v1, v2, v3 = rounds(v0, v1, v2 ^ np.uint64(0xff), v3, 3)
    return v0 ^ v1 ^ v2 ^ v3


def _initial(n, log2m, weights, seed):
    """Registers of every node's own counter, one byte each."""
    reg = np.zeros((n, 1 << log2m), dtype=np.uint8)

    def add(nodes, values):
        x = _hash(values)
        y = (x >> np.uint64(log2m)) | np.uint64(1 << 30)
        low = y & (~y + np.uint64(1))
        rank = np.log2(low.astype(np.float64)).astype(np.uint8) + 1
        np.maximum.at(reg, (nodes, (x & np.uint64((1 << log2m) - 1)).astype(np.int64)), rank)

    nodes = np.arange(n, dtype=np.uint64)
    if weights is None:
        add(nodes.astype(np.int64), nodes)
        return reg
    # value k of node v: step k of SplitMix64 from seed ^ v * golden ratio
    golden = np.uint64(0x9e3779b97f4a7c15)
    start = np.uint64(seed & _M64) ^ (nodes * golden)
    for k in range(1, int(weights.max()) + 1):
        has = weights >= k
        z = start[has] + np.uint64(k) * golden
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xbf58476d1ce4e5b9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94d049bb133111eb)
        add(np.nonzero(has)[0], z ^ (z >> np.uint64(31)))
    return reg


def _count(reg, log2m):
    """Estimated cardinality of every counter."""
    m = 1 << log2m
    alpha = {4: 0.673, 5: 0.697, 6: 0.709}.get(log2m, 0.7213 / (1 + 1.079 / m))
    out = []
    for part in reg.split(1 << 18):
        h = torch.exp2(-part.double())
        h = torch.where(part == 31, -h, h)  # the reference's 32-bit shift of 1 by 31
        e = alpha * m * m / h.sum(1)
        z = (part == 0).sum(1).double()
        small = (z > 0) & (e < 2.5 * m)
        out.append(torch.where(small, m * torch.log(m / z.clamp(min=1)), e))
    return torch.cat(out)


def _merge(reg, off, suc):
    """Every node's counter merged with its successors' (register-wise maximum), halving each list until one is left."""
    n, new = reg.shape[0], reg.clone()
    deg = off[1:] - off[:-1]
    a, step = 0, max(1, (1 << 28) // reg.shape[1])  # arcs a part
    bounds = off.cpu().numpy()
    while a < n:
        b = max(a + 1, int(np.searchsorted(bounds, bounds[a] + step, side="right")) - 1)
        b = min(b, n)
        d, vals = deg[a:b].clone(), reg[suc[off[a]:off[b]].long()]
        while d.numel() and int(d.max()) > 1:
            first = torch.cumsum(d, 0) - d
            half = (d + 1) // 2
            row = torch.repeat_interleave(torch.arange(b - a, device=d.device), half)
            k = torch.arange(row.numel(), device=d.device) - (torch.cumsum(half, 0) - half)[row]
            i = first[row] + 2 * k
            vals = torch.maximum(vals[i], vals[torch.minimum(i + 1, first[row] + d[row] - 1)])
            d = half
        has = torch.nonzero(d)[:, 0] + a
        new[has] = torch.maximum(new[has], vals)
        a = b
    return new


def _exact_run(case, seed, log2m, extra):
    off, suc = _arcs(case, seed)
    n, dev = case["n"], off.device
    weights = _weights(case, seed) if extra == "weights" else None
    reg = torch.from_numpy(_initial(n, log2m, weights, seed)).to(dev)
    est = _count(reg, log2m)
    nf, t = [torch.tensor(float(n), dtype=torch.float64, device=dev)], 0  # distance 0: every node reaches itself
    sod, harm, disc = (torch.zeros(n, dtype=torch.float64, device=dev) for _ in range(3))
    while t < n:
        new = _merge(reg, off, suc)
        modified = not torch.equal(new, reg)
        reg = new
        post = _count(reg, log2m)
        delta = (post - est).clamp(min=0)
        t += 1
        sod += delta * t
        harm += delta / t
        disc += delta * _discount(t)
        est = post
        nf.append(torch.maximum(est.sum(), nf[-1]))
        if not modified:
            break
    nf = torch.stack(nf).cpu()
    r = {"nf": torch.cat([nf, nf.new_zeros(NF_ROW - len(nf))]), "sod": sod.cpu(), "harmonic": harm.cpu()}
    if extra == "weights":
        r["discounted"] = disc.cpu()
    elif extra == "derived":
        r["lin"] = torch.where(sod == 0, torch.ones_like(sod), est * est / sod).cpu()
        r["reachable"] = est.cpu()
    return r


def exact(case, seed):
    if case["do"] in ("run", "call"):
        # larger graphs take over twenty seconds
        if case["n"] * case["deg"] << case["log2m"] > 6 << 30:
            return None
        return _exact_run(case, seed, case["log2m"], case["extra"])
    if case["do"] == "batch":
        if case["count"] > 24:
            return None
        parts = [_exact_run(c, x, l, "none") for c, l, x in _batch_cases(case, seed)]
        return {"nf": torch.stack([p["nf"] for p in parts]), "sod": torch.cat([p["sod"] for p in parts]),
                "harmonic": torch.cat([p["harmonic"] for p in parts])}
    return None  # whole numbers
