"""The cluster size a batch picks when none is given: few large queries, many small ones, none at all, one;
every query equals a single run."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale,graphs,per_graph,expect", [(18, 2, 2, 8), (10, 60, 12, 1), (13, 40, 4, None)])
def test_chosen_cluster_size(gpu, scale, graphs, per_graph, expect):
    torch = pytest.importorskip("torch")
    n = 1 << scale
    vgs = []
    for i in range(graphs):
        s, d, w = gpu.gen_rmat(scale, 8 + i % 9, seed=100 + i)
        vgs.append(gpu.VirtualGraph.build(n, s, d, w, K=(4, 8, 16)[i % 3]))
    queries = [(i, ("bfs", "sssp", "sswp")[(i + j) % 3], vgs[i].info()["max_degree_vertex"])
               for i in range(graphs) for j in range(per_graph)]
    with gpu.Batch(vgs) as b:
        words = b.set_queries(queries)
        out = torch.empty(words, dtype=torch.int32, device="cuda")
        b.run(out.data_ptr())
        assert b.config()[0] in (1, 2, 4, 8) and expect in (None, b.config()[0])
        host = out.cpu().numpy().view(np.uint32)
        for i, (g, algo, src) in enumerate(queries):
            if i % 7 == 0 or i == len(queries) - 1:
                want, _ = vgs[g].run(algo, "sync_push_dd", src)
                assert np.array_equal(host[i * n:(i + 1) * n], want), (i, algo)
        assert b.set_queries([]) == 0
        assert b.set_queries(queries[:1]) == n
        b.run(out.data_ptr())
        assert np.array_equal(out[:n].cpu().numpy().view(np.uint32), host[:n])
    for v in vgs:
        v.close()
