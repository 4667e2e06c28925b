"""The two forms of a visit's arrays: the choice between them on the host, and on
the GPU the lean one, which stands in where the wide one's allocation fails,
against the oracle at the sizes where its paths change."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import test_sweep_steps
import test_visit_levels

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "webgraph-algo-rs_gb300", "csrc")

CHOICE = r"""
#include <cstdio>
#include <initializer_list>
#include "visit_state.h"
using namespace hbl;
int main() {
    int bad = 0, wide = 0, lean = 0;
    const uint64_t G = 1ull << 30, far = 1ull << 40;
    for (uint64_t n : {1ull, 2ull, 100000ull, 400000000ull, 2800000000ull, 4000000000ull, 4026531840ull, 4294967294ull})
        for (uint64_t m : {0ull, 1ull, 7ull, 8ull, 1ull << 20, 1ull << 31, 1ull << 33, 11811160063ull, 30000000000ull,
                           38000000000ull, 70000000000ull})
            for (uint64_t row : {0ull, 0xffffffffull, 1ull << 32})
                for (uint64_t more : {(uint64_t)0, G, G + 1, 20 * G}) {
                    const Form f = choose_form(n, m, row, more, 160 * G);
                    const bool roomy = more <= G || more <= 20 * G;
                    const bool fits = n + m / 8 <= 0xf0000000ull && row < (1ull << 32);
                    if (f.lean == (roomy && fits)) bad++;
                    if (!f.lean && f.lg != 3) bad++;
                    // what a sum of units can reach: a unit a node and one for every 2^lg further arcs
                    if (units(n, m, f.lg) > 0xffffffffull) bad++;
                    // no longer than they have to be
                    if (f.lean && f.lg > 3 && n + (m >> (f.lg - 1)) <= 0xffffffffull && (m >> (f.lg - 1)) <= n) bad++;
                    if (tiles(n, m, f.lg) * 32 < units(n, m, f.lg)) bad++;
                    (f.lean ? lean : wide)++;
                    if (!choose_form(n, m, row, 9 * G, 71 * G).lean) bad++;  // more than its share
                    if (choose_form(n, m, row, 9 * G, 72 * G).lean != !fits) bad++;
                }
    if (!choose_form(400000000ull, 38000000000ull, 95, 0, far).lean) bad++;  // 5.2e9 units
    const uint64_t off[] = {0, 5, 5, 5 + (1ull << 33)};
    if (longest_row(off, 3, off[3]) != 1ull << 33 || longest_row(off, 2, 5) != 0) bad++;
    std::printf("%d wide %d lean %d bad\n", wide, lean, bad);
    return bad || !wide || !lean;
}
"""


def test_choice(tmp_path):
    src, exe = tmp_path / "choice.cpp", tmp_path / "choice"
    src.write_text(CHOICE)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I" + CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


class _Lean:
    """The package, with handles and sweeps made while the first allocation fails."""

    def __init__(self, hb):
        self._hb = hb

    def __getattr__(self, name):
        return getattr(self._hb, name)

    def _failing(self, f, *a, **k):
        self._hb.debug_fail_allocations(0)
        try:
            return f(*a, **k)
        finally:
            self._hb.debug_fail_allocations(-1)

    def ParFair(self, *a, **k):
        return self._failing(self._hb.ParFair, *a, **k)

    def exact_sum_sweep(self, *a, **k):
        return self._failing(self._hb.exact_sum_sweep, *a, **k)


def _er(hb, n, degree):
    return hb.Graph.erdos_renyi(n, degree, 5)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 33, 2_000, 40_000, 524_289])
def test_lean_sizes(hb, oracle, n):
    test_visit_levels.test_sizes(_Lean(hb), oracle, n)


@pytest.mark.gpu
@pytest.mark.parametrize("deg", [1, 8, 9, 257, 16_385, 150_001])
def test_lean_star(hb, oracle, deg):
    test_visit_levels.test_star(_Lean(hb), oracle, deg)


@pytest.mark.gpu
@pytest.mark.parametrize("n,degree", [(300, 15), (300, 16), (300, 299), (3000, 200), (20_000, 100), (600_000, 20)])
@pytest.mark.parametrize("max_distance", [None, 0, 1, 2])
def test_lean_long_units(hb, oracle, n, degree, max_distance):
    """Units of 2^4 to 2^8 arcs, taken eight at a time."""
    test_visit_levels._check(_Lean(hb), oracle, _er(hb, n, degree), [n // 3, 1, n // 3], max_distance)


@pytest.mark.gpu
def test_lean_chain_and_later_visits(hb, oracle):
    """More levels than one launch runs; distances of a second visit, whose queue
    does not begin at 0, and of a part of the events."""
    test_visit_levels.test_chain_and_leaves(_Lean(hb), oracle)
    n = 5000
    g = hb.Graph.from_csr(np.minimum(np.arange(n + 1), n - 1).astype(np.uint64), np.arange(1, n).astype(np.uint32))
    v = _Lean(hb).ParFair(g)
    nodes, _, dists, _ = v.par_visit([3000])
    np.testing.assert_array_equal(nodes, np.arange(3000, n))
    np.testing.assert_array_equal(dists, np.arange(n - 3000))
    nodes, preds, dists, _ = v.par_visit([1000, 0], max_distance=700)
    order = np.argsort(nodes)
    np.testing.assert_array_equal(nodes[order], np.r_[0:701, 1000:1701])
    np.testing.assert_array_equal(dists[order], np.r_[0:701, 0:701])
    v.close()


@pytest.mark.gpu
@pytest.mark.parametrize("lean", [False, True])
def test_distances_by_node_without_room(hb, oracle, lean):
    """hb_visit_each where its arrays by node cannot be allocated."""
    g = hb.Graph.weblike(30_000, cap=3000, window=64, seed=9)
    roots = [5, 17, 29_000, 5] + list(range(100, 200))
    want = oracle.OracleVisit(g.offsets, g.successors).visit_each(roots)
    v = (_Lean(hb) if lean else hb).ParFair(g)
    dist, pred = np.full(30_000, 77, np.uint32), np.full(30_000, 40_000, np.uint32)  # 40,000: no node
    hb.debug_fail_allocations(1)  # the predecessors'
    try:
        v.visit_each(roots, dist, pred)
    finally:
        hb.debug_fail_allocations(-1)
    again, pagain = np.full(30_000, 77, np.uint32), np.full(30_000, 40_000, np.uint32)
    v.reset()
    v.visit_each(roots, again, pagain)  # by node this time
    np.testing.assert_array_equal(dist, again)
    seen = pred != 40_000
    np.testing.assert_array_equal(seen, pagain != 40_000)
    np.testing.assert_array_equal(dist[seen], want[seen])
    assert np.all(dist[~seen] == 77) and seen.sum() > 1000
    up = seen & (dist > 0)
    assert np.all(dist[pred[up]] + 1 == dist[up])
    v.close()


@pytest.mark.gpu
@pytest.mark.parametrize("which", ["dist", "pred", "both"])
@pytest.mark.parametrize("lean", [False, True])
@pytest.mark.parametrize("room", [True, False])
def test_arrays_by_node(hb, oracle, which, lean, room):
    """Distances and predecessors by node stand where the events' do; only the lean
    form needs an allocation, for both, and does without it too. Events after that
    are whole again."""
    n = 30_000
    g = hb.Graph.weblike(n, cap=3000, window=64, seed=9)
    roots = list(range(100, 200)) + [5, 29_000, 5]
    want = oracle.OracleVisit(g.offsets, g.successors).visit_each(roots)
    v = (_Lean(hb) if lean else hb).ParFair(g)
    dist = np.full(n, 50_000, np.uint32) if which != "pred" else None
    pred = np.full(n, 50_000, np.uint32) if which != "dist" else None  # no node
    lib, r = hb.load_library(), np.asarray(roots, dtype=np.uint64)
    if not room:
        hb.debug_fail_allocations(0)
    try:
        rc = lib.hb_visit_each(v._h, r.ctypes.data_as(ctypes.POINTER(ctypes.c_uint64)), len(r),
                               dist.ctypes.data if dist is not None else None,
                               pred.ctypes.data if pred is not None else None, n)
        assert rc == hb.HB_OK
        if not room and not (lean and which == "both"):
            with pytest.raises(hb.HyperBallError):  # nothing was allocated: the failure is still to come
                hb.HyperBallBuilder.new(g, hb.HyperLogLogBuilder(n).log_2_num_reg(4).build()).build()
    finally:
        hb.debug_fail_allocations(-1)
    seen = (dist if dist is not None else pred) != 50_000
    assert seen.sum() > 1000 and not seen.all()
    if dist is not None:
        np.testing.assert_array_equal(dist[seen], want[seen])
    if pred is not None:
        assert np.array_equal(pred != 50_000, seen)
        up = seen & (want > 0)
        assert np.all(want[pred[up]] + 1 == want[up])
    v.reset()
    nodes, preds, dists, _ = v.par_visit([5], max_distance=3)
    on, _, od = oracle.OracleVisit(g.offsets, g.successors).visit([5], 3)
    d = np.full(n, -1, np.int64)
    d[on.astype(np.int64)] = od
    np.testing.assert_array_equal(d[nodes], dists)
    assert len(nodes) == len(on) and np.all(d[preds[dists > 0]] + 1 == dists[dists > 0])
    v.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n,level", [(1, "all"), (2, "all"), (257, "all"), (5_000, "all_forward"),
                                     (40_000, "radius_diameter")])
def test_lean_sweeps(hb, n, level):
    test_sweep_steps.test_sizes(_Lean(hb), n, level)


@pytest.mark.gpu
@pytest.mark.parametrize("n,degree", [(300, 40), (30_000, 17)])
def test_lean_sweeps_long_units(hb, n, degree):
    test_sweep_steps._check(_Lean(hb), _er(hb, n, degree), "radius_diameter")


@pytest.mark.gpu
def test_lean_sweep_symmetric(hb):
    g = _er(hb, 400, 30)
    t = g.transpose()
    rows = [np.union1d(g.successors_of(v), t.successors_of(v)) for v in range(400)]
    s = hb.Graph.from_csr(np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.uint64),
                          np.concatenate(rows).astype(np.uint32))
    want = test_sweep_steps.hbo.sum_sweep(np.asarray(s.offsets), np.asarray(s.successors), level="all")
    got = _Lean(hb).exact_sum_sweep(s, None, level="all")
    for f in test_sweep_steps.FIELDS:
        assert got[f] == want[f], f
    np.testing.assert_array_equal(got["forward_eccentricities"], want["forward_eccentricities"])


@pytest.mark.gpu
def test_sweep_on_a_nearly_full_device(hb):
    """4e6 components where 0.6 GiB are free: 85 bytes a node and 60 a
    component fit, 40 more a node do not."""
    torch = pytest.importorskip("torch")
    n = 4_000_000
    g = hb.Graph.from_csr(np.minimum(np.arange(n + 1), 20).astype(np.uint64), np.arange(1, 21).astype(np.uint32))
    t = g.transpose()
    hb.exact_sum_sweep(g, t, level="diameter")  # what the first sweep of a process brings along
    torch.cuda.empty_cache()
    hb.release_cached_memory(0)
    want = hb.exact_sum_sweep(g, t, level="diameter")
    free = torch.cuda.mem_get_info()[0]
    left = n * (85 + 60) + (48 << 20)
    held = [torch.empty(free - left, dtype=torch.uint8, device="cuda")]
    try:
        got = hb.exact_sum_sweep(g, t, level="diameter")
    finally:
        del held
        torch.cuda.empty_cache()
    for f in ("diameter", "diametral_vertex", "diameter_iterations", "sweeps"):
        assert got[f] == want[f]
