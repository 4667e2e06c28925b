"""Which standard iterations merge every successor: the share of counters that has
to have changed before grows with the counters."""
import numpy as np
import pytest

from parity import lockstep

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log2m", [4, 7, 8, 9, 10])
def test_shares_on_both_sides(hb, oracle, log2m):
    """Without a transpose: iterations after shares of 1 down to 0, those between a
    quarter and a half among them, each equal to the oracle's."""
    for g in (hb.Graph.weblike(20_000, cap=2000, window=256, seed=4), hb.Graph.rmat(13, 8, seed=2)):
        lockstep(hb, oracle, g, log2m)


def test_long_rows_are_not_merged_for_nothing(hb):
    """At log2m 10 an iteration after which under half of the counters changed leaves
    the others' rows alone: it takes well below one that merges all (0.63 of it; 0.94
    when it merges all itself)."""
    g = hb.Graph.rmat(20, 16, seed=1)
    with hb.HyperBallBuilder.new(g, hb.HyperLogLogBuilder(g.num_nodes).log_2_num_reg(10).build()).union_variant(0).build() as h:
        times = []
        for _ in range(4):
            h.run_until_done()
            st = h.iteration_stats()
            times.append([s["union_ms"] for s in st])
        times = np.min(times, axis=0)
        before = np.array([g.num_nodes] + [s["modified_counters"] for s in st[:-1]]) / g.num_nodes
    some = (before > 0.25) & (before < 0.5)
    assert some.any()
    assert np.all(times[some] < 0.8 * times[1]), (before, times)
