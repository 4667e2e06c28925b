"""GPU tests of what an iteration runs around its union: the systolic work
lists at the bounds of their tiles, and a batch's statistics at the bounds of
the instances' segments, and the marks of the predecessors of modified nodes."""
import numpy as np
import pytest

from parity import lockstep

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 33, 4096, 32_767, 32_768, 32_769, 65_537])
def test_work_list_tiles(hb, oracle, n):
    """One tile of the bitmaps is 32,768 nodes. A chain (systolic iterations
    that check a few nodes, then one) with nodes of up to 40 arcs in every tile,
    light and medium mixed. Counters and sums as in every lockstep run."""
    rng = np.random.default_rng(n)
    rows = [np.unique(rng.integers(0, n, size=rng.integers(2, 40))) if v % 97 == 0 else np.array([(v + 1) % n])
            for v in range(n)]
    off = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.uint64)
    g = hb.Graph.from_csr(off, np.concatenate(rows).astype(np.uint32))
    lockstep(hb, oracle, g, 4, transpose_on_device=True, buckets=(4, 1024), max_iters=40)


@pytest.mark.parametrize("hubs", [3, 64, 65, 100])
@pytest.mark.parametrize("in_degree", [1023, 1024, 3000])
def test_marks_of_hubs(hb, oracle, hubs, in_degree):
    """Nodes with in-degrees around the bound of what a warp takes alone, up to
    more of them than one block notes; a chain behind them keeps them changing
    while a few thousand nodes change in all."""
    n = 20_000
    chain = list(range(hubs, hubs + 40))
    rows = [[chain[0]] for _ in range(hubs)] + [[c + 1] for c in chain] + [[]] * (n - hubs - 40)
    for v in range(n - in_degree, n):
        rows[v] = list(range(hubs))
    off = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.uint64)
    g = hb.Graph.from_csr(off, np.concatenate([np.asarray(r, dtype=np.uint32) for r in rows]))
    lockstep(hb, oracle, g, 4, transpose_on_device=True)


def test_marks_of_sparse_words(hb, oracle):
    """More nodes than one pass of the warps over single words of the bitmap
    takes, few of them with arcs; the last node is one."""
    n = 10_200_007
    rng = np.random.default_rng(1)
    src = np.unique(np.append(rng.integers(0, n, size=30_000), [0, n - 1]))
    dst = rng.permutation(src)  # long paths over the nodes with arcs
    off = np.zeros(n + 1, dtype=np.uint64)
    off[src + 1] = 1
    g = hb.Graph.from_csr(np.cumsum(off, dtype=np.uint64), dst.astype(np.uint32))
    lockstep(hb, oracle, g, 4, transpose_on_device=True, max_iters=8, check_next=False)


@pytest.mark.parametrize("large", [8191, 8192, 8193, 16_384, 16_385, 70_001])
def test_instance_segments(hb, large):
    """Instances of no node, of one, and around 8,192 (a segment) and its
    multiples, beside each other and not on word bounds: iteration counts and
    registers as alone; sums of the estimates to 1e-12 (their order differs)."""
    e = np.zeros(0, dtype=np.uint32)
    gs = [hb.Graph.from_csr(np.zeros(2, np.uint64), e), hb.Graph.weblike(large, cap=200, window=64, seed=large),
          hb.Graph.from_csr(np.zeros(1, np.uint64), e), hb.Graph.erdos_renyi(large, 3, 7),
          hb.Graph.erdos_renyi(8192, 2, 9), hb.Graph.erdos_renyi(37, 2, 5)]
    b = hb.HyperBallBatch(gs, [5] * len(gs), sum_of_distances=True)
    for _ in range(2):  # the second run replays captured shapes
        b.run_until_done()
        for i, g in enumerate(gs):
            if not g.num_nodes:
                assert b.iterations(i) == 0
                continue
            logic = hb.HyperLogLogBuilder(g.num_nodes).log_2_num_reg(5).build()
            h = hb.HyperBallBuilder.new(g, logic).transpose_on_device(True).sum_of_distances(True).build()
            h.run_until_done()
            assert b.iterations(i) == h.iteration, i
            np.testing.assert_array_equal(b.registers(i), h.registers())
            np.testing.assert_allclose(b.neighborhood_function(i), h.neighborhood_function(), rtol=1e-12)
            np.testing.assert_allclose(b.sum_of_distances(i), h.sum_of_distances(), rtol=1e-12)
            h.close()
    b.close()


@pytest.mark.parametrize("n,cap", [(50, 10), (5000, 10), (60_000, 5000)])
def test_iteration_times(hb, n, cap):
    """The device's times of directly launched and of replayed iterations, with
    and without heavy nodes: the union lies within the iteration, and both
    within the wall time of the run."""
    import time
    g = hb.Graph.weblike(n, cap=cap, window=32, seed=1)
    logic = hb.HyperLogLogBuilder(n).log_2_num_reg(6).build()
    h = hb.HyperBallBuilder.new(g, logic).transpose_on_device(True).build()
    for _ in range(3):
        t0 = time.perf_counter()
        h.run_until_done()
        wall = (time.perf_counter() - t0) * 1e3
        st = h.iteration_stats()
        assert all(0 < s["union_ms"] < s["iteration_ms"] for s in st)
        assert sum(s["iteration_ms"] for s in st) < wall
    h.close()


@pytest.mark.parametrize("log2ms", [[4], [9], [4, 6, 8], [5, 4, 10, 7, 8, 6, 9]])
def test_groups_side_by_side(hb, log2ms):
    """A batch's groups, one for each counter size, with heavy nodes in some and
    runs of different lengths: as alone, first launched and then replayed."""
    gs = [hb.Graph.weblike(9000, cap=3000, window=32, seed=k) if k % 2 else hb.Graph.erdos_renyi(700 * (k + 1), 4, k)
          for k in range(len(log2ms))]
    b = hb.HyperBallBatch(gs, log2ms, sum_of_distances=True)
    for _ in range(3):
        b.run_until_done()
        for i, (g, m) in enumerate(zip(gs, log2ms)):
            logic = hb.HyperLogLogBuilder(g.num_nodes).log_2_num_reg(m).build()
            h = hb.HyperBallBuilder.new(g, logic).transpose_on_device(True).sum_of_distances(True).build()
            h.run_until_done()
            assert b.iterations(i) == h.iteration, i
            np.testing.assert_array_equal(b.registers(i), h.registers())
            np.testing.assert_allclose(b.neighborhood_function(i), h.neighborhood_function(), rtol=1e-12)
            np.testing.assert_allclose(b.sum_of_distances(i), h.sum_of_distances(), rtol=1e-12)
            h.close()
    assert b.stats()["union_ms"] > 0
    b.close()
