"""States of a visit's level launches: a block of a launch that reads one while it
is stored over, and the ones an ExactSumSweep leaves behind on a graph whose start
has no arcs."""
import os
import subprocess

import numpy as np
import pytest

from test_sum_sweep import FIELDS, hbo

torch = pytest.importorskip("torch")

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "webgraph-algo-rs_gb300", "csrc")

# every level that a block takes alone, every way its visit can end, and every
# mixture of the words of its state and of the ended one
MIXTURES = r"""
#include <cstdio>
#include <cstring>
#include <initializer_list>
#include "visit_state.h"
using namespace hbl;
int main() {
    static_assert(alignof(State) == 32 && sizeof(State) == 32, "one sector");
    int bad = 0, ends = 0;
    const uint32_t smalls[] = {512, 2048, 16384};
    for (uint32_t small : smalls)
        for (uint32_t units : {1u, 31u, small})
            for (uint32_t d = 1; d <= 4; d++)
                for (uint32_t next : {0u, 1u, small, small + 1, 1u << 20, 0xffffffffu})
                    for (uint32_t max_d : {d, d + 1, 0xffffffffu}) {
                        const State old{7, 20, units, d, d - 1};
                        const State t = advance(old, ((unsigned long long)next << 32) | 90u, max_d);
                        if (t.b != 20 || t.e != 90 || t.d != d + 1 || t.last != d) bad++;
                        if (done(t) != (next == 0 || d + 1 > max_d)) bad++;
                        if (!done(t) && t.units != next) bad++;
                        if (!done(t)) continue;
                        ends++;
                        for (int mask = 0; mask < 32; mask++) {
                            uint32_t w[8], o[8], e[8];
                            std::memcpy(o, &old, 32);
                            std::memcpy(e, &t, 32);
                            for (int k = 0; k < 8; k++) w[k] = (mask >> k) & 1 ? e[k] : o[k];
                            State m;
                            std::memcpy(&m, w, 32);
                            // a block other than the first has nothing to do
                            if (!(done(m) || m.units <= small)) bad++;
                        }
                    }
    for (uint32_t max_d : {0u, 1u, 0xffffffffu})
        if (done(first_level(0, 3, 40000, max_d)) != (max_d == 0)) bad++;
    std::printf("%d %d\n", ends, bad);
    return bad != 0 || ends == 0;
}
"""


def test_mixture_of_states(tmp_path):
    """A visit may end while other blocks of the launch still read the state that
    is stored over: whatever words they get, they have nothing to do."""
    src, exe = tmp_path / "mixtures.cpp", tmp_path / "mixtures"
    src.write_text(MIXTURES)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I" + CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


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
