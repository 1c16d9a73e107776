"""Round machinery of the persistent traversal at its edges: the warps' append and far buffers (256 and 128
entries) just below, at and above their capacity and many times over it, the queue length that comes with
the round's barrier (also one launch per round), the two halves of a 16-slot part. Whole numbers: equal to
the oracle's, and the activity log equal between the persistent and the one-launch-per-round form."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _fan(leaves, seed=2):
    """Vertex 0 reaches every leaf, heavily (a far vertex when the bucket is narrow); the leaves form a light
    path, so most leaves improve again, one or a few per round."""
    rng = np.random.default_rng(seed)
    i = np.arange(1, leaves + 1, dtype=np.uint32)
    s = np.concatenate((np.zeros(leaves, np.uint32), i[:-1]))
    d = np.concatenate((i, i[1:]))
    w = np.concatenate((rng.integers(500, 1000, leaves), rng.integers(1, 8, leaves - 1))).astype(np.uint32)
    return leaves + 1, s, d, w


@pytest.mark.parametrize("K", [4, 8, 16])
@pytest.mark.parametrize("leaves", [31, 127, 128, 129, 255, 256, 257, 20000])
def test_fan(gpu, leaves, K):
    n, s, d, w = _fan(leaves)
    if leaves > 1000:  # a short path: the number of rounds stays small
        keep = np.r_[np.arange(leaves), leaves + np.arange(0, leaves - 1, 2)]
        s, d, w = s[keep], d[keep], w[keep]
    want = {"bfs": oracle.bfs(n, s, d, 0), "sssp": oracle.dijkstra(n, s, d, w, 0), "sswp": oracle.widest(n, s, d, w, 0)}
    with gpu.VirtualGraph.build(n, s, d, w, K=K) as vg:
        for algo, deltas in (("bfs", (0,)), ("sssp", (0, 1, 100)), ("sswp", (0, 1, 100))):
            for delta in deltas:
                got, _ = vg.run(algo, "sync_push_dd", 0, delta=delta)
                assert np.array_equal(got, want[algo]), (algo, delta)
                got, _ = vg.run(algo, "sync_push_dd", 0, delta=delta, host_loop=leaves < 200)
                assert np.array_equal(got, want[algo]), (algo, delta, "host loop")
        if leaves < 200:
            _, _, a1 = vg.run("bfs", "sync_push_dd", 0, activity_cap=64)
            _, _, a2 = vg.run("bfs", "sync_push_dd", 0, activity_cap=64, host_loop=True)
            assert np.array_equal(a1, a2) and a1[0] == leaves


@pytest.mark.parametrize("algo", ["sssp", "sswp", "cc"])
@pytest.mark.parametrize("degree", [7, 8, 9, 15, 16, 17, 33])
def test_wide_parts(gpu, algo, degree):
    """Degrees around the part size at K = 16: rows whose second half is empty, partly and wholly used."""
    rng = np.random.default_rng(degree)
    n = 600
    s = np.repeat(np.arange(n, dtype=np.uint32), degree)
    d = rng.integers(0, n, s.size).astype(np.uint32)
    w = rng.integers(1, 64, s.size).astype(np.uint32)
    with gpu.VirtualGraph.build(n, s, d, w, K=16) as vg:
        for variant in ("async_push_dd", "async_push_td", "sync_push_td"):
            got, _ = vg.run(algo, variant, 3)
            assert np.array_equal(got, oracle.expected(algo, variant, n, s, d, w, 3)), variant


@pytest.mark.parametrize("K", [4, 8, 16])
@pytest.mark.parametrize("b", [1, 31, 257, 3000])
def test_push_after_the_first_pull_round(gpu, b, K):
    """BFS's first pull round only counts its claims' parts; when a push round follows, the queue is collected
    from the levels. Vertex 0 reaches 4000 vertices with many parts, b of them lead on (too few to pull
    again: 12 b < n), the first through a vertex of more than 32 parts; two more levels follow. The
    vertices are numbered at random, so the ones collected lie anywhere."""
    a, rng = 4000, np.random.default_rng(b)
    n = 1 + a + 3 * b + 12 * b + 1003
    A, B, C, D = 1 + np.arange(a), 1 + a + np.arange(b), 1 + a + b + np.arange(b), 1 + a + 2 * b + np.arange(b)
    pairs = [(np.zeros(a), A), (np.repeat(A, 9), np.zeros(9 * a)), (A[:b], B), (B, C),
             (np.full(40 * K + 3, B[0]), C[np.arange(40 * K + 3) % b]), (C, D)]
    name = rng.permutation(n)
    s, d = (name[np.concatenate([p[i] for p in pairs]).astype(np.int64)].astype(np.uint32) for i in (0, 1))
    src = int(name[0])
    want = oracle.bfs(n, s, d, src)
    with gpu.VirtualGraph.build(n, s, d, None, K=K, reverse=True) as vg:
        got, res, act = vg.run("bfs", "sync_push_dd", src, activity_cap=16)
        assert np.array_equal(got, want) and res["pull_rounds"] >= 1
        ref, res2, act2 = vg.run("bfs", "sync_push_dd", src, activity_cap=16, bfs_push_only=True)
        assert np.array_equal(ref, want) and res2["pull_rounds"] == 0 and np.array_equal(act, act2)
