"""How the host waits for an iteration: a program that asked the device to block
keeps its cores."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

RUN = r"""
import ctypes, sys, time
cu = ctypes.CDLL("libcuda.so.1")
assert cu.cuInit(0) == 0
dev = ctypes.c_int()
assert cu.cuDeviceGet(ctypes.byref(dev), 0) == 0
assert cu.cuDevicePrimaryCtxSetFlags_v2(dev, int(sys.argv[1])) == 0
sys.path.insert(0, sys.argv[2])
import hyperball_gb300 as hb
g = hb.Graph.erdos_renyi(3_000_000, 16, 1)   # below the size whose iterations are timed by events
h = hb.HyperBallBuilder.new(g, hb.HyperLogLogBuilder(g.num_nodes).log_2_num_reg(9).build()).build()
h.run_until_done()
w0, c0 = time.perf_counter(), time.thread_time()
for _ in range(5):
    h.run_until_done()
wall, cpu = time.perf_counter() - w0, time.thread_time() - c0
print(cpu / wall, wall, h.neighborhood_function()[-1])
"""


def _share(flags):
    r = subprocess.run([sys.executable, "-c", RUN, str(flags), os.path.join(REPO, "webgraph-algo-rs_gb300")],
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    return [float(x) for x in r.stdout.split()]


def test_blocking_wait(product_lib):
    """CU_CTX_SCHED_BLOCKING_SYNC (4): iterations of milliseconds cost the calling
    thread a small part of their time (all of it where the host looks for the end)."""
    share, wall, nf = _share(4)
    assert wall > 0.05, wall
    assert share < 0.5, (share, wall)
    assert _share(0)[2] == nf
