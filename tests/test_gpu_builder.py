"""The GPU build of the virtual graph against a stable sort in numpy, at the sizes where its passes change:
vertex counts around a bucket (2048) and around one and two partition passes (2^22), edge counts around a
tile (8192), one vertex owning every edge, empty buckets, sorted and random input order, host, page-locked
and device arrays. The layout is whole numbers: equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _layout(n, owner, nb, w, K):
    order = np.argsort(owner, kind="stable")
    deg = np.bincount(owner, minlength=n).astype(np.int64)
    parts = (deg + K - 1) // K
    vstart = np.concatenate(([0], np.cumsum(parts)))
    first = np.concatenate(([0], np.cumsum(deg)))[:-1]
    o = owner[order].astype(np.int64)
    slot = vstart[o] * K + (np.arange(o.size) - first[o])
    vcol = np.full(vstart[-1] * K, 0xFFFFFFFF, np.uint32)
    vw = np.zeros(vstart[-1] * K, np.uint32)
    vcol[slot] = nb[order]
    vw[slot] = w[order]
    return deg, vstart, np.repeat(np.arange(n), parts), vcol, vw


def _check(vg, n, s, d, w, K):
    deg, vstart, vowner, vcol, vw = _layout(n, s, d, w, K)
    got = vg.download()
    assert np.array_equal(got["outdeg"], deg)
    assert np.array_equal(got["vstart"], vstart)
    assert np.array_equal(got["vowner"], vowner)
    assert np.array_equal(got["vcol"].ravel(), vcol)
    assert np.array_equal(got["vw"].ravel(), vw)
    inf = vg.info()
    assert inf["max_out_degree"] == deg.max(initial=0)
    if deg.max(initial=0):
        assert inf["max_degree_vertex"] == int(deg.argmax())


def _edges(n, m, kind, seed=1):
    rng = np.random.default_rng(seed)
    s = rng.integers(0, n, m, dtype=np.uint32)
    if kind == "one":
        s[:] = n // 2
    elif kind == "sorted":
        s.sort()
    elif kind == "skew":
        s = (s.astype(np.float64) / n) ** 4 * n
        s = s.astype(np.uint32)
    elif kind == "ends":
        s = np.where(rng.random(m) < 0.5, 0, n - 1).astype(np.uint32)
    return s, rng.integers(0, n, m, dtype=np.uint32), rng.integers(1, 64, m, dtype=np.uint32)


@pytest.mark.parametrize("kind", ["random", "sorted", "skew", "one", "ends"])
@pytest.mark.parametrize("n,m", [(1, 3), (2, 5), (5, 1), (2047, 8191), (2048, 8192), (2049, 8193), (4097, 40000),
                                 (70001, 16384), (1 << 20, 300001), (1 << 22, 70000), ((1 << 22) + 1, 70001),
                                 (9_000_001, 200003)])
def test_layout(gpu, n, m, kind):
    torch = pytest.importorskip("torch")
    K = {0: 4, 1: 8, 2: 16}[(n + m) % 3]
    s, d, w = _edges(n, m, kind)
    with gpu.VirtualGraph.build(n, s, d, w, K=K) as vg:
        _check(vg, n, s, d, w, K)
    pinned = [torch.from_numpy(a.view(np.int32)).pin_memory().numpy().view(np.uint32) for a in (s, d, w)]
    with gpu.VirtualGraph.build(n, *pinned, K=K) as vg:
        _check(vg, n, s, d, w, K)
    # device arrays at an address that is not 16-byte aligned, both directions of each edge
    dev = [torch.from_numpy(np.concatenate((np.zeros(1, np.int32), a.view(np.int32)))).cuda()[1:] for a in (s, d, w)]
    torch.cuda.synchronize()
    with gpu.VirtualGraph.build_device(n, m, *[t.data_ptr() for t in dev], K=K, symmetrize=True) as vg:
        _check(vg, n, np.concatenate((s, d)), np.concatenate((d, s)), np.concatenate((w, w)), K)


@pytest.mark.parametrize("bad", ["source", "target"])
def test_bad_endpoints_are_refused(gpu, bad):
    s, d, w = _edges(3000, 9000, "random")
    (s if bad == "source" else d)[8500] = 3000
    with pytest.raises(gpu.EEGError):
        gpu.VirtualGraph.build(3000, s, d, w, K=8)
