"""Rounds of at most one 32-entry chunk per CTA, where one warp makes the round's reservations itself, and rounds around
that size: paths (one vertex a round), combs (a path with leaves: 2 to 65 claims a round) and hubs, against the oracle
and, bucketed, with and without far vertices."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _comb(length, leaves):
    """A path of hubs, each with leaves: its chunk's claims go past one 32-entry chunk at 32 leaves and up."""
    hubs = np.arange(length) * (leaves + 1)
    s = [hubs[:-1]]
    d = [hubs[1:]]
    for k in range(leaves):
        s.append(hubs)
        d.append(hubs + 1 + k)
    return length * (leaves + 1), np.concatenate(s), np.concatenate(d)


@pytest.mark.parametrize("K", [4, 8, 16])
@pytest.mark.parametrize("leaves", [0, 1, 31, 32, 33, 64, 300, 2000])
def test_paths_and_combs(gpu, leaves, K):
    n, s, d = _comb(max(40, 600 // (leaves + 1)), leaves)
    rng = np.random.default_rng(leaves)
    s, d = np.r_[s, d].astype(np.uint32), np.r_[d, s].astype(np.uint32)
    w = rng.integers(1, 60, s.size, dtype=np.uint32)
    want = {"bfs": oracle.bfs(n, s, d, 0), "sssp": oracle.dijkstra(n, s, d, w, 0)}
    with gpu.VirtualGraph.build(n, s, d, w, K=K) as vg, gpu.VirtualGraph.build(n, s, d, w, K=K, reverse=True) as both:
        for g in (vg, both):
            for cap in (0, n):
                got = g.run("bfs", "sync_push_dd", 0, activity_cap=cap)[0]
                assert np.array_equal(got, want["bfs"])
        for delta in (0, 1, 100, 100000):
            got, _ = vg.run("sssp", "sync_push_dd", 0, delta=delta)
            assert np.array_equal(got, want["sssp"]), delta
        wide = vg.run("sswp", "sync_push_td", 0)[0]
        for delta in (0, 1, 16):
            assert np.array_equal(vg.run("sswp", "sync_push_dd", 0, delta=delta)[0], wide), delta
        assert np.array_equal(vg.run("cc", "async_push_dd")[0], vg.run("cc", "async_push_td")[0])
