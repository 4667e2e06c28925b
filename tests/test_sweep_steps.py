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


def _acyclic(hb, n, degree, seed):
    """Every arc leads to a larger node, so that every arc is between components."""
    rng = np.random.RandomState(seed)
    rows = [np.unique(rng.randint(v + 1, n, degree)) if v + 1 < n else np.zeros(0, int) for v in range(n)]
    off = np.concatenate([[0], np.cumsum([len(r) for r in rows])])
    return hb.Graph.from_csr(off.astype(np.uint64), np.concatenate(rows).astype(np.uint32))


def _check_failing(hb, g, fail, fails):
    """The sweep where allocation `fail` fails (0 would be the rows and entries of the
    visits); `fails`: the sweep makes that many."""
    if fail is None:
        return _check(hb, g, "radius_diameter")
    hb.debug_fail_allocations(fail)
    try:
        _check(hb, g, "radius_diameter")
        # what is left of the count fails a handle's creation
        small = hb.Graph.erdos_renyi(100, 3, 1)
        build = hb.HyperBallBuilder.new(small, hb.HyperLogLogBuilder(100).log_2_num_reg(4).build()).build
        if fails:
            build().close()
        else:
            with pytest.raises(hb.HyperBallError):
                build()
    finally:
        hb.debug_fail_allocations(-1)


@pytest.mark.parametrize("n,degree", [(2_000, 1), (2_000, 2), (2_000, 6), (300, 60)])
@pytest.mark.parametrize("fail", [None, 1, 2])
def test_list_of_arcs_between_components(hb, n, degree, fail):
    """Up to two such arcs a node stand in the bounds' arrays; where the list of more
    (1: its sources, 2: its targets) cannot be allocated the host passes over all arcs."""
    _check_failing(hb, _acyclic(hb, n, degree, degree), fail, degree > 2)


@pytest.mark.parametrize("fail", [None, 1, 2, 3, 4, 5])
def test_more_tiles_than_nodes(hb, fail):
    """Arcs between two components, often repeated: the tiles' counts do not fit the bounds' arrays."""
    m = 2048 * 5 + 7
    g = hb.Graph.from_csr(np.array([0, m, m, m], dtype=np.uint64), np.resize([1, 2], m).astype(np.uint32))
    _check_failing(hb, g, fail, True)
