"""The barrier that ends a traversal's round, in a kernel of its own: a CTA that gives up ends the waits of CTAs that
have gone on to another round's word. Two CTAs, every wait bounded; nothing faults or hangs."""
import ctypes as C
import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]

SOURCE = r"""
#include "traverse.cuh"
using namespace eeg;
struct Out { uint32_t first, second; unsigned long long waited; };
__global__ void two(unsigned long long* w, BarrierWords* bw, uint64_t brief, uint64_t patient, Out* out) {
    __shared__ uint32_t len;
    const uint64_t t0 = global_timer_ns();
    // CTA 0 waits for CTA 1 at the first word and gives up; CTA 1 is already at the second
    const bool ok = blockIdx.x == 0 ? trav::round_barrier(&w[0], bw, brief, &len) : trav::round_barrier(&w[1], bw, patient, &len);
    if (threadIdx.x == 0) {
        if (blockIdx.x == 0) out->first = ok;
        else { out->second = ok; out->waited = global_timer_ns() - t0; }
    }
}
extern "C" int run(unsigned long long brief, unsigned long long patient, Out* host) {
    unsigned char* d = nullptr;
    if (cudaMalloc((void**)&d, 4096) != cudaSuccess || cudaMemset(d, 0, 4096) != cudaSuccess) return -1;
    unsigned long long* w = (unsigned long long*)d;
    BarrierWords* bw = (BarrierWords*)(d + 1024);
    Out* out = (Out*)(d + 2048);
    uint64_t b = brief, p = patient;
    void* args[] = {&w, &bw, &b, &p, &out};
    if (cudaLaunchCooperativeKernel((const void*)two, dim3(2), dim3(64), args, 0, 0) != cudaSuccess) return -2;
    const bool ok = cudaMemcpy(host, out, sizeof(Out), cudaMemcpyDeviceToHost) == cudaSuccess;
    BarrierWords h;
    const bool ok2 = cudaMemcpy(&h, bw, sizeof(h), cudaMemcpyDeviceToHost) == cudaSuccess;
    cudaFree(d);
    return ok && ok2 ? (int)h.status : -3;
}
"""


class Out(C.Structure):
    _fields_ = [("first", C.c_uint32), ("second", C.c_uint32), ("waited", C.c_uint64)]


def test_giving_up_reaches_every_round(gpu, tmp_path):
    from eegraph_gb300 import _build

    (tmp_path / "two.cu").write_text(SOURCE)
    subprocess.run([_build.NVCC, *_build.GENCODE, "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-I", str(_build.CSRC),
                    str(tmp_path / "two.cu"), "-o", str(tmp_path / "two.so")], check=True, capture_output=True)
    lib = C.CDLL(str(tmp_path / "two.so"))
    o = Out()
    status = lib.run(C.c_ulonglong(1_000_000), C.c_ulonglong(1_000_000_000), C.byref(o))
    assert status == 1, status  # DEV_TIMEOUT: the first CTA's millisecond ran out
    assert (o.first, o.second) == (0, 0)
    assert o.waited < 100_000_000, o.waited  # not its own second
