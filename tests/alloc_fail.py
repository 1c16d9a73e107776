"""The library with a fake of the device allocator's failures: its objects linked again with cudaMalloc and cudaMallocAsync
wrapped, in a package of its own for a child process. Nothing fails on the GPU: the wrapped call returns the error."""
import os
import subprocess
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]

SHIM = r"""
#include <stddef.h>
typedef int err;
extern err __real_cudaMalloc(void**, size_t);
extern err __real_cudaMallocAsync(void**, size_t, void*);
static size_t lo = 1, hi = 0;
static long failed = 0, calls = 0;
static size_t sizes[4096];
static int refused(size_t n) {
    if (calls < 4096) sizes[calls] = n;
    ++calls;
    if (n < lo || n > hi) return 0;
    ++failed;
    return 1;
}
err __wrap_cudaMalloc(void** p, size_t n) { return refused(n) ? 2 : __real_cudaMalloc(p, n); }
err __wrap_cudaMallocAsync(void** p, size_t n, void* s) { return refused(n) ? 2 : __real_cudaMallocAsync(p, n, s); }
void shim_fail(size_t from, size_t to) { lo = from; hi = to; failed = 0; calls = 0; }
long shim_failed(void) { return failed; }
long shim_calls(void) { return calls; }
size_t shim_size(long i) { return sizes[i]; }
"""


def run(tmp_path, script):
    """Run `script` in a child process whose eegraph_gb300 (E) is the wrapped library; fail(lo, hi) makes allocations of
    lo to hi bytes fail, failed() counts them, sizes() lists what was asked for since."""
    from eegraph_gb300 import _build

    pkg = tmp_path / "eegraph_gb300"
    (pkg / "_lib").mkdir(parents=True)
    for f in (ROOT / "eegraph_gb300").glob("*.py"):
        (pkg / f.name).write_text(f.read_text())
    (tmp_path / "shim.c").write_text(SHIM)
    subprocess.run(["gcc", "-O1", "-fPIC", "-c", str(tmp_path / "shim.c"), "-o", str(tmp_path / "shim.o")], check=True)
    objs = [str(_build.OBJ / (Path(s).stem + ".o")) for s in _build.CU_SOURCES + _build.CPP_SOURCES]
    subprocess.run([_build.NVCC, "-shared", "-o", str(pkg / "_lib" / "libeegraph.so"), *objs, str(tmp_path / "shim.o"),
                    *_build.GENCODE, "-cudart", "static", "-Xlinker", "--wrap=cudaMalloc", "-Xlinker", "--wrap=cudaMallocAsync",
                    "-ldl", "-lpthread", "-lrt"], check=True)
    head = ("import ctypes as C\nimport numpy as np\nimport eegraph_gb300 as E\nL = E.lib()\nL.eeg_set_device(0)\n"
            "L.shim_size.restype = C.c_size_t\n"
            "def fail(lo, hi): L.shim_fail(C.c_size_t(lo), C.c_size_t(hi))\n"
            "def failed(): return L.shim_failed()\n"
            "def sizes(): return [L.shim_size(C.c_long(i)) for i in range(min(L.shim_calls(), 4096))]\n")
    r = subprocess.run([sys.executable, "-c", head + script], env={**os.environ, "PYTHONPATH": str(tmp_path)},
                       cwd=str(tmp_path), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    return r.stdout
