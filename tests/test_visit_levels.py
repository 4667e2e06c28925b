"""GPU tests of the visit's levels at the sizes where their paths change:
levels that one block takes alone and levels of the whole grid, visited bits in
shared and in global memory, nodes of many tiles, long chains, and levels of
nodes without successors."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _csr(hb, rows):
    off = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.uint64)
    suc = np.concatenate(rows).astype(np.uint32) if len(rows) else np.zeros(0, np.uint32)
    return hb.Graph.from_csr(off, suc)


def _check(hb, oracle, g, roots, max_distance=None):
    """Distances, predecessors and counts of one visit against the oracle's sequential visit."""
    v = hb.ParFair(g)
    for _ in range(2):  # the second pass launches as many levels as the first took
        v.reset()
        nodes, preds, dists, st = v.par_visit(roots, max_distance)
        o = oracle.OracleVisit(g.offsets, g.successors)
        on, _, od = o.visit(roots, max_distance)
        want = np.full(g.num_nodes, -1, dtype=np.int64)
        want[on.astype(np.int64)] = od
        got = np.full(g.num_nodes, -1, dtype=np.int64)
        got[nodes] = dists
        np.testing.assert_array_equal(got, want)
        assert len(nodes) == len(on) and np.all(np.diff(dists.astype(np.int64)) >= 0)
        # every arc of an expanded node is an event: Unknown the first time, else Known
        deg = np.diff(np.asarray(g.offsets).astype(np.int64))
        md = g.num_nodes if max_distance is None else max_distance
        far = dists > 0
        assert st["known_arcs"] == deg[nodes[dists < md]].sum() - far.sum() and st["visited"] == len(on)
        assert np.all(want[preds[far]] == dists[far].astype(np.int64) - 1)
        for k in np.nonzero(far)[0][:: max(1, len(nodes) // 500)]:
            assert nodes[k] in g.successors_of(int(preds[k]))
    return st


@pytest.mark.parametrize("n", [1, 2, 31, 33, 2_000, 40_000, 524_288, 524_289, 600_001])
def test_sizes(hb, oracle, n):
    """Tiny graphs (every level one block's), and both sides of the size up to
    which the visited bits stand in shared memory."""
    _check(hb, oracle, hb.Graph.weblike(n, cap=min(n, 5000), window=64, seed=n), [n // 2])


@pytest.mark.parametrize("deg", [1, 7, 8, 9, 255, 256, 257, 4096, 16_383, 16_384, 16_385, 150_001])
def test_star(hb, oracle, deg):
    """A hub's units and tiles around their bounds; the leaves lead back, so the
    level after it is wide and claims nothing."""
    rows = [np.arange(1, deg + 1)] + [np.array([0])] * deg
    st = _check(hb, oracle, _csr(hb, rows), [0])
    assert st["levels"] == 2


def test_chain_and_leaves(hb, oracle):
    """More small levels than one launch runs, then a node whose successors
    have none: a last level without units."""
    n = 3000
    rows = [np.array([v + 1]) for v in range(n - 1)] + [np.arange(n, n + 500)] + [np.zeros(0)] * 500
    st = _check(hb, oracle, _csr(hb, rows), [0])
    assert st["levels"] == n + 1


@pytest.mark.parametrize("max_distance", [0, 1, 2, 5])
def test_filter_and_many_roots(hb, oracle, max_distance):
    g = hb.Graph.rmat(15, 8, seed=3)
    _check(hb, oracle, g, [5, 5, 17, 40, 1000, 17], max_distance)
    _check(hb, oracle, g, list(range(0, g.num_nodes, 3)), max_distance)
