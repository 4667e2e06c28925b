"""The page-locked stages of small results: a getter that has none takes its result
through device memory, and many threads' getters agree."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(hb, n=5_000, seed=1):
    g = hb.Graph.erdos_renyi(n, 6, seed)
    h = (hb.HyperBallBuilder.new(g, hb.HyperLogLogBuilder(n).log_2_num_reg(5).build())
         .sum_of_distances(True).sum_of_inverse_distances(True).build())
    h.run_until_done()
    return h


def test_without_a_stage(hb):
    """No stage can be made: the getter does without, and the next one makes it."""
    h = _run(hb)
    hb.release_cached_memory(0)
    hb.debug_fail_allocations(0)
    try:
        first = h.sum_of_distances()
        # the failure was the stage's
        _run(hb, 100).close()
    finally:
        hb.debug_fail_allocations(-1)
    np.testing.assert_array_equal(first, h.sum_of_distances())
    hb.release_cached_memory(0)
    np.testing.assert_array_equal(first, h.sum_of_distances())
    h.close()


def test_more_threads_than_stages(hb):
    hs = [_run(hb, 5_000 + k, k) for k in range(24)]
    want = [(h.sum_of_distances(), h.harmonic_centralities()) for h in hs]
    bad = []

    def get(k):
        for _ in range(50):
            if not (np.array_equal(hs[k].sum_of_distances(), want[k][0])
                    and np.array_equal(hs[k].harmonic_centralities(), want[k][1])):
                bad.append(k)

    ts = [threading.Thread(target=get, args=(k,)) for k in range(len(hs))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad
    for h in hs:
        h.close()
