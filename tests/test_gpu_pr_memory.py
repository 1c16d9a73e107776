"""PageRank where the residual form's array does not fit: plain sweeps, as with a sweep cap."""
import pytest

from tests import alloc_fail

pytestmark = pytest.mark.gpu


def test_without_the_residual_form(gpu, tmp_path):
    """The partial sums and ranks (also 8 bytes per vertex) are there from a capped run."""
    alloc_fail.run(tmp_path, """
n = 1 << 15
s, d, _ = E.gen_rmat(15, 16, seed=4)
def graph(): return E.VirtualGraph.build(n, s, d, None, K=8, reverse_only=True)
with graph() as vg:
    want, full = vg.run("pr", "sync_push_td")
with graph() as vg:
    plain, capped = vg.run("pr", "sync_push_td", max_iterations=500)
    assert capped["status"] == E.OK and capped["iterations"] > 3 * full["iterations"]
    fail(8 * n, 8 * n)
    x, res = vg.run("pr", "sync_push_td")
    assert failed() == 1, sizes()
    assert res["status"] == E.OK and res["iterations"] == capped["iterations"]
    assert np.abs(x - want).sum() <= 1e-6 * want.sum()
""")
