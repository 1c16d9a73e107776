"""Data-driven PageRank where its extras do not fit: without private targets, and without long steps."""
import pytest

from tests import alloc_fail

pytestmark = pytest.mark.gpu

GRAPH = """
n = 1 << 15
s, d, _ = E.gen_rmat(15, 16, seed=4)
def graph(): return E.VirtualGraph.build(n, s, d, None, K=8)
def run(vg, **kw):
    x, res = vg.run("pr", "sync_push_dd", **kw)
    assert res["status"] == E.OK
    return x, res
with graph() as vg:
    want, full = run(vg)
    P = vg.info()["num_parts"]
"""


def test_without_private_targets(gpu, tmp_path):
    alloc_fail.run(tmp_path, GRAPH + """
with graph() as vg:
    fail(4 * P * 8, 4 * P * 8)
    x, res = run(vg)
    assert failed() == 1, sizes()
    assert np.abs(x - want).sum() <= 1e-6 * want.sum()
    x, _ = run(vg)  # settled: not asked for again
    assert failed() == 1
    assert np.abs(x - want).sum() <= 1e-6 * want.sum()
""")


def test_without_long_steps(gpu, tmp_path):
    """The values, residuals and amounts are there from a run with a threshold; the two arrays that long steps add are
    refused."""
    alloc_fail.run(tmp_path, GRAPH + """
with graph() as vg:
    run(vg, pr_accuracy=1e-6)
    fail(8 * n, 8 * n)
    x, res = run(vg)
    assert failed() == 1, sizes()
    assert res["iterations"] > 2 * full["iterations"]  # the queue's rounds
    assert np.abs(x - want).sum() <= 1e-6 * want.sum()
""")


def test_the_queue_is_not_asked_for_by_long_steps(gpu, tmp_path):
    alloc_fail.run(tmp_path, GRAPH + """
with graph() as vg:
    fail(1, 0)
    run(vg)
    assert 4 * P not in sizes(), sizes()
    run(vg, pr_accuracy=1e-6)
    assert 4 * P in sizes(), sizes()
""")
