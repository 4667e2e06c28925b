"""States of a visit's level launches: the ones an ExactSumSweep leaves behind on
a graph whose start has no arcs."""
import numpy as np
import pytest

from test_sum_sweep import FIELDS, hbo

torch = pytest.importorskip("torch")


def _dirty_device_memory():
    """Device memory that later allocations of the library may get, none of it zero."""
    torch.empty(0, device="cuda")
    keep = [torch.full((1 << k,), 0x5b, dtype=torch.uint8, device="cuda") for k in range(9, 26)]
    torch.cuda.synchronize()
    del keep
    torch.cuda.empty_cache()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 100, 70_000])
@pytest.mark.parametrize("symmetric", [False, True])
def test_sweep_without_arcs(hb, n, symmetric):
    """A start without arcs ends its visit before the first level: every launch
    finds an ended state, whatever the memory held before. (70,000 nodes: levels
    of the whole grid.)"""
    _dirty_device_memory()
    off, suc = np.zeros(n + 1, dtype=np.uint64), np.zeros(0, dtype=np.uint32)
    g = hb.Graph.from_csr(off, suc)
    level = "all_forward" if symmetric else "radius_diameter"
    want = hbo.sum_sweep(off, suc, *([] if symmetric else [off, suc]), level=level)
    got = hb.exact_sum_sweep(g, None if symmetric else g, level=level)
    for f in FIELDS:
        assert got[f] == want[f], (f, got[f], want[f])
    if symmetric:
        np.testing.assert_array_equal(got["forward_eccentricities"], want["forward_eccentricities"])
