"""GPU tests of what an iteration runs around its union: the systolic work
lists at the bounds of their tiles, and a batch's statistics at the bounds of
the instances' segments."""
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
