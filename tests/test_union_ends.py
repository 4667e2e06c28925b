"""GPU tests of how the union kernels end a node: the counts of counters with
registers of 30 and 31, medium nodes spread over a team at every counter size,
heavy nodes around the segment bounds, and more heavy items than a grid of
blocks looks at in one pass. The oracle is compared with after every iteration."""
import numpy as np
import pytest

from parity import lockstep

pytestmark = pytest.mark.gpu


def _rank(log2m, seed, node):
    """The register value node's hash gives (Jenkins hash, in Python integers)."""
    mask = (1 << 64) - 1
    a, b, c = (seed + node) & mask, seed, 0x9E3779B97F4A7C13
    for s1, s2, s3 in ((43, 9, 8), (38, 23, 5), (35, 49, 11), (12, 18, 22)):
        a = ((a - b - c) & mask) ^ (c >> s1)
        b = ((b - c - a) & mask) ^ ((a << s2) & mask)
        c = ((c - a - b) & mask) ^ (b >> s3)
    y = (c >> log2m) | (1 << 30)
    return (y & -y).bit_length()


@pytest.mark.parametrize("log2m,seed,node,rank", [
    (4, 246070, 303, 31), (4, 389093, 2427, 30), (6, 246070, 303, 31), (6, 326865, 690, 30),
    (8, 485366, 2798, 31), (8, 981107, 398, 30)])
def test_largest_registers(hb, oracle, log2m, seed, node, rank):
    """A register of 30 or 31 takes the counts out of their fast form (and 31
    into the reference's 32-bit shift), through light, medium and heavy nodes."""
    assert _rank(log2m, seed, node) == rank
    g = hb.Graph.weblike(3000, cap=400, window=256, seed=seed)
    lockstep(hb, oracle, g, log2m, hash_kind=1, seed=seed, transpose_on_device=True, buckets=(3, 24))


@pytest.mark.parametrize("log2m", range(4, 11))
@pytest.mark.parametrize("variant", [0, 6])
def test_medium_teams(hb, oracle, log2m, variant):
    """Medium nodes of 5 to 700 arcs: the team's partial rows are merged and
    spread over its lanes, at every number of chunks per counter."""
    g = hb.Graph.weblike(7001, cap=700, window=128, seed=log2m)
    lockstep(hb, oracle, g, log2m, transpose_on_device=True, buckets=(4, 1024), variant=variant)


@pytest.mark.parametrize("log2m", [4, 6, 7, 10])
def test_heavy_segment_bounds(hb, oracle, log2m):
    """Heavy nodes just below, at and above the bounds of a segment and of a
    split, beside ones of a few arcs."""
    rng = np.random.default_rng(log2m)
    n = 13_000
    sizes = {5: 6143, 900: 6144, 901: 6145, 4000: 8192, 4001: 8193, 12_000: 12_288, 12_999: 12_289, 7: 4096}
    rows = [np.unique(rng.integers(0, n, size=rng.integers(0, 4))) for _ in range(n)]
    for v, d in sizes.items():
        rows[v] = np.sort(rng.choice(n, size=d, replace=False))
    off = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.uint64)
    g = hb.Graph.from_csr(off, np.concatenate(rows).astype(np.uint32))
    lockstep(hb, oracle, g, log2m, transpose_on_device=True, buckets=(2, 3))


def test_heavy_items_beyond_one_pass(hb, oracle):
    """Every node heavy: more items than the blocks of a grid look at in one
    pass, most of them idle in the systolic iterations."""
    g = hb.Graph.erdos_renyi(1_000_000, 1, 3)
    lockstep(hb, oracle, g, 4, transpose_on_device=True, buckets=(0, 0), max_iters=30, check_next=False)
