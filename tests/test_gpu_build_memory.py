"""What a build asks the device's memory for: a page-locked list read in place where its copy does not fit, and two sets
of partitioned edges however many passes there are."""
import pytest

from tests import alloc_fail

pytestmark = pytest.mark.gpu


def test_symmetrised_page_locked_input_without_a_copy(gpu, tmp_path):
    torch = pytest.importorskip("torch")  # noqa: F841 -- the child pins with it
    alloc_fail.run(tmp_path, """
import torch
n, m = 70001, 300007
rng = np.random.default_rng(1)
e = [rng.integers(1 if i == 2 else 0, n if i < 2 else 60, m, dtype=np.uint32) for i in range(3)]
pinned = [torch.from_numpy(a.view(np.int32)).pin_memory().numpy().view(np.uint32) for a in e]
with E.VirtualGraph.build(n, *e, K=8, symmetrize=True) as vg:
    want = vg.download()
for lo, hi, count in ((1, 0, 0), (12 * m, 12 * m, 1)):
    fail(lo, hi)
    with E.VirtualGraph.build(n, *pinned, K=8, symmetrize=True) as vg:
        got = vg.download()
    assert failed() == count, sizes()
    assert all(np.array_equal(got[k], want[k]) for k in want)
fail(12 * m, 12 * m)
try:  # pageable input has to be copied
    E.VirtualGraph.build(n, *e, K=8, symmetrize=True)
    raise SystemExit("no error")
except E.EEGError:
    pass
""")


def test_two_sets_of_edges(gpu, tmp_path):
    alloc_fail.run(tmp_path, """
n, m = (1 << 22) + 5, 500003  # sorted by vertex in three passes
rng = np.random.default_rng(1)
s, d = rng.integers(0, n, m, dtype=np.uint32), rng.integers(0, n, m, dtype=np.uint32)
fail(1, 0)
with E.VirtualGraph.build(n, s, d, None, K=8) as vg:
    pass
assert sizes().count(4 * m) == 6, sizes()  # owners, neighbours and weights, twice
""")
