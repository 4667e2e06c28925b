"""A kernel's dynamic shared memory is allowed on every device that launches it:
the limit belongs to a device, and a first failure is tried again."""
import os
import re
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "webgraph-algo-rs_gb300", "csrc")

ONCE = r"""
#include <thread>
#include <vector>
#include "once_per_device.h"
int main() {
    static hbl::OncePerDevice once;
    int calls[80] = {}, fail = 1;
    auto set = [&](int d) { return once(d, [&] { calls[d]++; return fail; }); };
    if (set(0) != 1 || set(0) != 1 || calls[0] != 2) return 1;  // not kept
    fail = 0;
    if (set(0) || set(0) || calls[0] != 3) return 2;
    if (set(1) || set(1) || calls[1] != 1) return 3;            // another device
    if (set(63) || set(63) || calls[63] != 1) return 4;
    if (set(64) || set(64) || calls[64] != 2 || calls[0] != 3) return 5;
    std::vector<std::thread> ts;
    static hbl::OncePerDevice shared;
    std::atomic<int> n{0};
    for (int t = 0; t < 8; t++) ts.emplace_back([&] { for (int k = 0; k < 1000; k++) shared(5, [&] { n++; return 0; }); });
    for (auto& t : ts) t.join();
    return n >= 1 && n <= 8 ? 0 : 6;
}
"""


def test_once_per_device(tmp_path):
    src, exe = tmp_path / "once.cpp", tmp_path / "once"
    src.write_text(ONCE)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-pthread", "-I" + CSRC, str(src), "-o", str(exe)],
                   check=True)
    assert subprocess.run([str(exe)]).returncode == 0


def test_no_limit_is_kept_for_the_process():
    for name in sorted(os.listdir(CSRC)):
        with open(os.path.join(CSRC, name)) as f:
            text = f.read()
        assert not re.search(r"static\s+(const\s+)?cudaError_t\s+\w+\s*=", text), name


@pytest.mark.gpu
def test_visits_and_sweeps_on_two_devices(hb):
    torch = pytest.importorskip("torch")
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    g = hb.Graph.weblike(40_000, seed=1)
    t = g.transpose()
    got = []
    for device in (0, 1):
        v = hb.ParFair(g, device=device)
        got.append((v.visit_each([7]), hb.exact_sum_sweep(g, t, level="diameter", device=device)["diameter"]))
        v.close()
    np.testing.assert_array_equal(got[0][0], got[1][0])
    assert got[0][1] == got[1][1]
