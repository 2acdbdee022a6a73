"""Side streams (csrc/qsv_side.cpp) over a fake CUDA runtime, on the host: what a failed call leaves behind."""
import ctypes
import os
import subprocess

import pytest

from qsv_b200 import build

# counts live streams and events, fails the call that is told to, and keeps the last error as the runtime does
FAKE = r"""
#include <cuda_runtime.h>
#include <cstdint>
#include "qsv_side.h"
static int live_streams = 0, live_events = 0, made = 0, fail_at = -1, device = 0;
static cudaError_t last = cudaSuccess;
static cudaError_t step() {
    if (made++ == fail_at) return last = cudaErrorMemoryAllocation;
    return cudaSuccess;
}
extern "C" {
cudaError_t cudaGetDevice(int *d) { *d = device; return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
    const cudaError_t e = step();
    if (e == cudaSuccess) { *s = (cudaStream_t)(uintptr_t)(0x1000 + made); live_streams++; }
    return e;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *v, unsigned) {
    const cudaError_t e = step();
    if (e == cudaSuccess) { *v = (cudaEvent_t)(uintptr_t)(0x2000 + made); live_events++; }
    return e;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { live_streams--; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { live_events--; return cudaSuccess; }
void fake_reset(int fail, int dev) { made = 0; fail_at = fail; device = dev; last = cudaSuccess; }
int fake_made() { return made; }
int fake_live() { return live_streams + live_events; }
int fake_last() { return (int)last; }
void *take() { return qsv::side_take(); }
void give(void *s) { qsv::side_give((qsv::SideStreams *)s); }
}
"""


@pytest.fixture(scope="module")
def side(tmp_path_factory):
    d = tmp_path_factory.mktemp("side")
    src, so = d / "fake.cpp", d / "side.so"
    src.write_text(FAKE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-I", os.path.join(build.cuda_root(), "include"),
                    "-I", build.CSRC, "-o", str(so), str(src), os.path.join(build.CSRC, "qsv_side.cpp")],
                   check=True, timeout=300)
    lib = ctypes.CDLL(str(so))
    lib.take.restype = ctypes.c_void_p
    lib.give.argtypes = [ctypes.c_void_p]
    return lib


def test_a_failed_call_leaves_no_error_and_no_streams(side):
    side.fake_reset(-1, 0)
    s = side.take()
    calls = side.fake_made()
    assert s and calls > 0
    side.give(s)
    for k in range(calls):
        before = side.fake_live()
        side.fake_reset(k, 1 + k)                # a device of its own: nothing is left over from an earlier turn
        assert side.take() is None
        assert side.fake_last() == 0, f"call {k} left its error for the next launch to report"
        assert side.fake_live() == before
