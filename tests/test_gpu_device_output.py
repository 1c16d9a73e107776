"""Traversal results left on the GPU: the run's last kernel writes the caller's array, in 16-byte stores where it is
aligned for them and word by word elsewhere; memory that is not this device's own goes through a copy. Equal to the
host's, and nothing beside the array is written."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
RUNS = [("bfs", "sync_push_dd"), ("sssp", "sync_push_dd"), ("sswp", "async_push_td"), ("cc", "async_push_dd")]
GUARD = 0x5A5A5A5A


def _graph(gpu, n):
    rng = np.random.default_rng(n)
    m = 3 * n
    e = rng.integers(0, n, m, dtype=np.uint32), rng.integers(0, n, m, dtype=np.uint32), rng.integers(1, 60, m, dtype=np.uint32)
    return gpu.VirtualGraph.build(n, *e, K=8), int(e[0][0])


@pytest.mark.parametrize("offset", [0, 1, 2, 3, 4, 7])
@pytest.mark.parametrize("n", [1, 3, 4, 5, 1023, 2048, 2049, 100003])
def test_alignments_and_tails(gpu, n, offset):
    torch = pytest.importorskip("torch")
    vg, src = _graph(gpu, n)
    with vg:
        for algo, variant in RUNS:
            out = torch.full((n + 16,), GUARD, dtype=torch.int32, device="cuda")
            torch.cuda.synchronize()
            want, ref = vg.run(algo, variant, src)
            _, res = vg.run(algo, variant, src, out_device_ptr=out.data_ptr() + 4 * offset)
            got = out.cpu().numpy().view(np.uint32)
            assert np.array_equal(got[offset:offset + n], want)
            assert (np.r_[got[:offset], got[offset + n:]] == GUARD).all()
            assert (res["reached_vertices"], res["reached_edges"]) == (ref["reached_vertices"], ref["reached_edges"])


def test_managed_memory(gpu):
    vg, src = _graph(gpu, 5001)
    p = C.c_void_p()
    assert gpu.lib().eeg_managed_alloc(C.c_size_t(4 * 5001), C.byref(p)) == gpu.OK
    try:
        with vg:
            for algo, variant in RUNS:
                want, _ = vg.run(algo, variant, src)
                vg.run(algo, variant, src, out_device_ptr=p.value)
                assert np.array_equal(np.ctypeslib.as_array(C.cast(p, C.POINTER(C.c_uint32)), (5001,)), want)
    finally:
        gpu.lib().eeg_managed_free(p)


def test_iteration_cap_writes_what_it_has(gpu):
    torch = pytest.importorskip("torch")
    n = 3000  # a path: two rounds reach two vertices past the source
    s = np.arange(n - 1, dtype=np.uint32)
    with gpu.VirtualGraph.build(n, s, s + 1, None, K=4) as vg:
        want, ref = vg.run("bfs", "sync_push_dd", 0, max_iterations=2, check=False)
        out = torch.full((n,), GUARD, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        _, res = vg.run("bfs", "sync_push_dd", 0, max_iterations=2, check=False, out_device_ptr=out.data_ptr())
    assert ref["status"] == res["status"] == gpu.ERR_ITER_CAP
    assert want[:3].tolist() == [0, 1, 2] and (want[3:] >= gpu.DIST_INFINITY).all()
    assert np.array_equal(out.cpu().numpy().view(np.uint32), want)


def test_a_run_that_gives_up_leaves_the_array(gpu):
    torch = pytest.importorskip("torch")
    s, d, w = gpu.gen_rmat(20, 16, seed=1, wmin=1, wmax=63)
    out = torch.full((1 << 20,), GUARD, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    gave_up = 0
    with gpu.VirtualGraph.build(1 << 20, s, d, w, K=8) as vg:
        for variant in ("async_push_td", "sync_push_td", "async_push_td"):
            out.fill_(GUARD)
            torch.cuda.synchronize()
            _, res = vg.run("sssp", variant, int(s[0]), timeout_us=1, check=False, out_device_ptr=out.data_ptr())
            if res["status"] == gpu.ERR_TIMEOUT:
                gave_up += 1
                assert bool((out == GUARD).all())
    assert gave_up, "no wait ran out under a 1 us limit"
