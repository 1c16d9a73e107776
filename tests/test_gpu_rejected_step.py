"""A long step of the adjoint that its estimate allows and its outcome does not: the L1 norm of a residual can grow there
(every leaf of a hub takes the hub's), which the measurement before the step does not see. Such a run goes on with plain
sweeps. A cycle carries most of the residual; a pulse travels down a path and reaches 2000 leaves' hub in the sweep of
the step when the path has three edges (by a model in 64 bits), before or after it with two or four."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C", [1, 3, 64])
@pytest.mark.parametrize("length", [2, 3, 4])
def test_adjoint(gpu, length, C):
    sp = pytest.importorskip("scipy.sparse")
    cycle, leaves = 50, 2000
    hub, last = cycle, cycle + length
    n = last + 1 + leaves
    s = np.r_[np.arange(cycle), np.arange(hub, last), np.arange(last + 1, n)]
    d = np.r_[(np.arange(cycle) + 1) % cycle, np.arange(hub + 1, last + 1), np.full(leaves, hub)]
    g = np.zeros((n, C), np.float32)
    g[:cycle] = 1.0
    g[last] = 0.02 * cycle
    A = sp.csr_matrix((np.full(s.size, 0.85), (s, d)), (n, n))
    want = f = g.astype(np.float64)
    while np.abs(f).max() > 1e-18:
        f = A @ f
        want = want + f
    with gpu.VirtualGraph.build(n, s.astype(np.uint32), d.astype(np.uint32), None, K=8, reverse=True, edge_ids=True) as vg:
        with gpu.PPR(vg, C) as p:
            p.set_weights(np.ones(s.size, np.float32))
            p.forward(np.full((n, C), 1.0 / n, np.float32), x_out=False)
            out, res = p.adjoint(g, outputs=("dt",))
    assert (res["iterations"] > 45) == (length == 3), res["iterations"]
    # d/(1-d) ||f||_1 <= tol ||L||_1 over all columns, and FP32 sums of a few terms
    off = np.abs(out["dt"].astype(np.float64) / 0.15 - want)
    assert off.sum() <= 2e-7 * np.abs(want).sum() + 3e-7 * np.abs(want).sum()
