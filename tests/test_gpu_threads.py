"""Several threads at once, each with graphs of its own."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _in_threads(jobs):
    failed = []

    def guard(job):
        try:
            job()
        except Exception as e:  # noqa: BLE001 -- reported by the test
            failed.append(e)

    ts = [threading.Thread(target=guard, args=(j,)) for j in jobs]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not failed, failed[:3]


def test_builds_with_and_without_weights(gpu):
    """Builds with and without a payload launch the same kernels with different amounts of shared memory."""
    def job(n, weighted, reps=250):
        rng = np.random.default_rng(n)
        s, d = rng.integers(0, n, 3 * n, dtype=np.uint32), rng.integers(0, n, 3 * n, dtype=np.uint32)
        w = rng.integers(1, 9, 3 * n, dtype=np.uint32) if weighted else None
        deg = np.bincount(s, minlength=n)

        def go():
            gpu.lib().eeg_set_device(0)
            for i in range(reps):
                with gpu.VirtualGraph.build(n, s, d, w, K=8, reverse_only=not weighted) as vg:
                    if i % 50 == 0 and weighted:
                        lay = vg.download()
                        assert np.array_equal(np.diff(lay["vstart"].astype(np.int64)), -(-deg // 8))
        return go

    _in_threads([job(500, True), job(700, False), job(5000, True), job(40000, False)])


def test_pagerank_of_small_and_large_graphs(gpu):
    """The sweeps' shared memory follows the number of vertices."""
    def job(n, reps=150):
        rng = np.random.default_rng(n)
        s, d = rng.integers(0, n, 4 * n, dtype=np.uint32), rng.integers(0, n, 4 * n, dtype=np.uint32)
        vg = gpu.VirtualGraph.build(n, s, d, None, K=8, reverse_only=True)

        def go():
            gpu.lib().eeg_set_device(0)
            first = None
            for _ in range(reps):
                x, res = vg.run("pr", "sync_push_td")
                assert res["status"] == gpu.OK
                first = x if first is None else first
                assert np.allclose(x, first, rtol=1e-5)
            vg.close()
        return go

    _in_threads([job(300), job(3000), job(50000)])
