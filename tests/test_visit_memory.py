"""Device memory that a breadth-first visit holds."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _held(make):
    make().close()  # what the first handle of a process brings along
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    h = make()
    held = free - torch.cuda.mem_get_info()[0]
    h.close()
    assert abs(torch.cuda.mem_get_info()[0] - free) <= 2 << 20  # all of it back
    return held


def test_visit_arrays(hb):
    """The successors, 44 bytes a node (its row, its entry, bitmap, queue, predecessor
    and distance), the tiles and a piece of roots; the offsets go when every node's row is known."""
    g = hb.Graph.weblike(4_000_003, seed=1)
    n, m = g.num_nodes, g.num_arcs
    want = 4 * m + 44 * n + n // 8 + (m // 8 + n) // 4 + min(4 * n, 16 << 20)
    assert _held(lambda: hb.ParFair(g)) <= want + (8 << 20)


def test_roots_in_pieces(hb, oracle):
    """More roots than go to the device at once."""
    import numpy as np
    n = (1 << 22) + 5
    g = hb.Graph.from_csr(np.arange(n + 1, dtype=np.uint64), ((np.arange(n) + 1) % n).astype(np.uint32))
    roots = np.arange(0, n, 1)[::-1]
    v = hb.ParFair(g)
    nodes, _, dists, st = v.par_visit(roots)
    assert st["visited"] == n and st["levels"] == 1 and st["known_arcs"] == n
    assert not dists.any() and np.array_equal(np.sort(nodes), np.arange(n))
    v.reset()
    nodes, preds, dists, st = v.par_visit(np.arange(0, n, 2), max_distance=1)
    assert st["visited"] == n and st["levels"] == 2
    assert np.array_equal(np.sort(nodes[dists == 1]), np.arange(1, n, 2)) and np.all(preds[dists == 1] + 1 == nodes[dists == 1])
    v.close()


def test_lean_arrays(hb):
    """Without room for the rows and entries a visit holds no more than its graph and
    24 bytes a node: offsets, queue, predecessors, units, tiles, bitmap and a piece of roots."""
    g = hb.Graph.weblike(4_000_003, seed=1)
    n, m = g.num_nodes, g.num_arcs

    def make():
        hb.debug_fail_allocations(0)
        try:
            return hb.ParFair(g)
        finally:
            hb.debug_fail_allocations(-1)

    want = 4 * m + 20 * n + n // 8 + n // 2 + min(4 * n, 16 << 20)
    assert _held(make) <= min(want + (8 << 20), 4 * m + 24 * n + n // 8 + (8 << 20))
