"""GPU tests of ExactSumSweep's steps at the sizes where their kernels can go
wrong: arcs between components around the bounds of an arc tile, and graphs on
both sides of the sizes where the visits' levels change. Every field equals the
oracle's."""
import numpy as np
import pytest

from test_sum_sweep import FIELDS, hbo

pytestmark = pytest.mark.gpu


def _check(hb, g, level):
    t = g.transpose()
    want = hbo.sum_sweep(np.asarray(g.offsets), np.asarray(g.successors), np.asarray(t.offsets),
                         np.asarray(t.successors), level=level)
    got = hb.exact_sum_sweep(g, t, level=level)
    for f in FIELDS:
        assert got[f] == want[f], (f, got[f], want[f])
    for f in ("forward_eccentricities", "backward_eccentricities"):
        assert (f in got) == (f in want), f
        if f in want:
            np.testing.assert_array_equal(got[f], want[f], err_msg=f)


@pytest.mark.parametrize("m", [1, 255, 2047, 2048, 2049, 4096, 6145])
@pytest.mark.parametrize("cross", ["few", "all"])
def test_arcs_between_components(hb, m, cross):
    """A tile is 2,048 arcs. `all`: a chain, each node a component, so that every
    arc crosses; `few`: cycles of 50 nodes joined by one arc each."""
    n = m + 1
    if cross == "all":
        off = np.minimum(np.arange(n + 1), m)
        suc = np.arange(1, n)
    else:
        v = np.arange(m)
        # node v goes on in its cycle; the last arcs of a cycle's end node lead to the next cycle
        nxt = np.where((v % 50 == 49) | (v == m - 1), v - v % 50, v + 1)
        rows = [[int(x)] for x in nxt] + [[]]
        for c in range(49, m - 1, 50):
            rows[c] = sorted({rows[c][0], c + 1})
        off = np.concatenate([[0], np.cumsum([len(r) for r in rows])])
        suc = np.concatenate([np.asarray(r, dtype=np.int64) for r in rows])
    g = hb.Graph.from_csr(off.astype(np.uint64), suc.astype(np.uint32))
    _check(hb, g, "radius_diameter")


@pytest.mark.parametrize("n,level", [(1, "all"), (2, "all"), (255, "all"), (257, "all"), (5_000, "all_forward"),
                                     (40_000, "radius_diameter"), (524_289, "diameter")])
def test_sizes(hb, n, level):
    """One node and a few, both sides of a block's threads, of the graphs whose
    levels one block takes, and more nodes than have their bits in shared memory."""
    _check(hb, hb.Graph.weblike(n, cap=min(n, 3000), window=min(64, n), seed=n), level)
