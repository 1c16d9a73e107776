"""The cluster size a batch picks when none is given, and its working memory: bounded by what 4 CTAs per query need or a
sixteenth of the device, and 4 when the choice does not fit."""
import numpy as np
import pytest

from tests import alloc_fail

pytestmark = pytest.mark.gpu


def test_a_large_graph_bounds_the_choice(gpu):
    """900 queries on a small graph alone would take one CTA each; with 21 M vertices beside it that is 25 GB of scratch."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(0)
    n, big = 1000, 5 << 22
    s, d, w = (rng.integers(1 if i == 2 else 0, n, 5000, dtype=np.uint32) for i in range(3))
    with gpu.VirtualGraph.build(n, s, d, w) as a, gpu.VirtualGraph.build(big, s, d, w) as b:
        queries = [(0, "sssp", int(s[i])) for i in range(900)]
        with gpu.Batch([a]) as batch:
            batch.set_queries(queries)
            assert batch.config()[0] == 1
        with gpu.Batch([a, b]) as batch:
            before = torch.cuda.mem_get_info()
            words = batch.set_queries(queries + [(1, "bfs", int(s[0]))])
            used = before[0] - torch.cuda.mem_get_info()[0]
            assert used <= max(before[1] / 16, 76 * 4 * (big + 2 * a.info()["num_parts"])) * 1.1, used
            out = torch.empty(words, dtype=torch.int32, device="cuda")
            batch.run(out.data_ptr())
            got = out.cpu().numpy().view(np.uint32)
        for i in (0, 1, 450, 899):
            assert np.array_equal(got[i * n:(i + 1) * n], a.run("sssp", "sync_push_dd", int(s[i]))[0])
        assert np.array_equal(got[900 * n:], b.run("bfs", "sync_push_dd", int(s[0]))[0])


def test_four_when_the_choice_does_not_fit(gpu, tmp_path):
    alloc_fail.run(tmp_path, """
rng = np.random.default_rng(0)
n = 1 << 18
s, d, w = (rng.integers(1 if i == 2 else 0, 1000, 5000, dtype=np.uint32) for i in range(3))
with E.VirtualGraph.build(n, s, d, w) as g, E.Batch([g]) as b:
    queries = [(0, "sssp", int(s[i])) for i in range(900)]
    b.set_queries(queries)
    assert b.config()[0] == 1, b.config()
    fail(200 << 20, 1 << 40)  # the stamps of 304 clusters: 319 MB; of 76: 80
    b.set_queries(queries)
    assert failed() == 1 and b.config()[0] == 4, (failed(), b.config())
    try:
        b.set_queries(queries, 1)  # the caller's own choice stays an error
        raise SystemExit("no error")
    except E.EEGError:
        pass
    b.set_queries(queries)
    fail(1, 0)
    b.set_queries(queries[:3], 4)
""")
