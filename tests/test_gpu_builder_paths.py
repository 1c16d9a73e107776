"""The build's two forms (buckets of 2048 vertices; sparse graphs sorted down to the vertex) on both sides of the line
between them, with edge indices, both directions of each edge, page-locked input, hubs and buckets of many tiles.
Whole numbers: equal to a stable sort in numpy. Transposed parts: through PageRank, run to the end (a relative L1 bound
of 1e-7 says little about single vertices of a graph that leaks most of its mass), which a wrong or missing in-edge
changes by far more than the 1e-5 allowed for FP32's rounding."""
import numpy as np
import pytest

from tests.test_gpu_builder import _check, _edges

pytestmark = pytest.mark.gpu
N20, N22 = 1 << 20, 1 << 22


# (n, m): the last row of each group is on the buckets' side
@pytest.mark.parametrize("n,m,kind", [
    (N20 + 1, 700_000, "random"), (N20 + 1, 700_000, "one"), (N20 + 3, 786_434, "skew"), (N20 + 3, 786_436, "skew"),
    (N22, 3_145_727, "random"), (N22, 3_145_728, "random"),
    (N22 + 1, 6_291_457, "skew"), (N22 + 1, 6_291_458, "skew"), (N22 + 2, 100_000, "ends"),
    (300, 300_000, "one"), (5000, 400_000, "ends"), (2048, 140_000, "random")])
def test_forms(gpu, n, m, kind):
    torch = pytest.importorskip("torch")
    K = (4, 8, 16)[m % 3]
    s, d, w = _edges(n, m, kind)
    with gpu.VirtualGraph.build(n, s, d, w, K=K) as vg:
        _check(vg, n, s, d, w, K)
    # edge indices: the weights are gathered by them
    pinned = [torch.from_numpy(a.view(np.int32)).pin_memory().numpy().view(np.uint32) for a in (s, d, w)]
    with gpu.VirtualGraph.build(n, *pinned, K=K, edge_ids=True) as vg:
        _check(vg, n, s, d, w, K)
    half = m // 2  # both directions of each edge: m arcs again
    s, d, w = s[:half], d[:half], w[:half]
    both = np.concatenate((s, d)), np.concatenate((d, s)), np.concatenate((w, w))
    for a in ((s, d, w), [p[:half] for p in pinned]):
        with gpu.VirtualGraph.build(n, *a, K=K, symmetrize=True, edge_ids=True) as vg:
            _check(vg, n, *both, K)


@pytest.mark.parametrize("n,m", [(N20 + 1, 500_000), (N22 + 1, 500_000), (N22 + 1, 7_000_000), (3000, 500_000)])
@pytest.mark.parametrize("mode", ["reverse", "reverse_only", "symmetrize"])
def test_transposed_parts(gpu, n, m, mode):
    sp = pytest.importorskip("scipy.sparse")
    s, d, _ = _edges(n, m // 2 if mode == "symmetrize" else m, "skew")
    with gpu.VirtualGraph.build(n, s, d, None, K=8, **{mode: True}) as vg:
        x, res = vg.run("pr", "sync_push_td", pr_tolerance=1e-15)
    assert res["status"] == gpu.OK
    if mode == "symmetrize":
        s, d = np.concatenate((s, d)), np.concatenate((d, s))
    A = sp.csr_matrix((0.85 / np.bincount(s, minlength=n).astype(float)[s], (d, s)), (n, n))
    want = f = np.full(n, 0.15)
    while (f / want).max() > 1e-12:
        f = A @ f
        want = want + f
    assert np.abs(x / want - 1).max() <= 1e-5


@pytest.mark.parametrize("n,m", [(3000, 20_000), (N22 + 1, 300_000), (N22 + 1, 7_000_000)])
@pytest.mark.parametrize("bad", [0, 1])
def test_bad_endpoints_of_both_directions_and_pinned_input(gpu, n, m, bad):
    torch = pytest.importorskip("torch")
    e = _edges(n, m, "random")
    e[bad][m - 3] = n
    pinned = [torch.from_numpy(a.view(np.int32)).pin_memory().numpy().view(np.uint32) for a in e]
    for a in (e, pinned):
        for kw in ({}, {"symmetrize": True}, {"reverse": True}, {"edge_ids": True}):
            with pytest.raises(gpu.EEGError):
                gpu.VirtualGraph.build(n, *a, K=8, **kw)
