"""Side streams (csrc/qsv_side.cpp) over a fake CUDA runtime, on the host: what a failed call leaves behind, which
streams they can be tied to while something is being captured, and that sets are made once, kept and bounded."""
import ctypes
import os
import subprocess

import pytest

from qsv_b200 import build

# counts live streams and events, fails the call that is told to, and keeps the last error as the runtime does
FAKE = r"""
#include <cuda_runtime.h>
#include <cstdint>
#include <map>
#include "qsv_side.h"
static int live_streams = 0, live_events = 0, made = 0, fail_at = -1, device = 0;
static cudaError_t last = cudaSuccess;
static std::map<cudaStream_t, int> captures;     // graph each captured stream belongs to (-1: cannot be asked)
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
cudaError_t cudaStreamGetCaptureInfo(cudaStream_t s, cudaStreamCaptureStatus *st, unsigned long long *id, cudaGraph_t *,
                                     const cudaGraphNode_t **, size_t *) {
    const auto c = captures.find(s);
    if (c != captures.end() && c->second < 0) return last = cudaErrorStreamCaptureImplicit;
    *st = c == captures.end() ? cudaStreamCaptureStatusNone : cudaStreamCaptureStatusActive;
    *id = c == captures.end() ? 0 : c->second;
    return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus *st) {
    *st = captures.count(s) ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
void fake_capture(void *s, int graph) { if (graph) captures[(cudaStream_t)s] = graph; else captures.erase((cudaStream_t)s); }
void *side_stream(void *s, int k) { return ((qsv::SideStreams *)s)->stream[k]; }
int joins(void *s, int count, void *stream) { return qsv::side_joins((qsv::SideStreams *)s, count, (cudaStream_t)stream); }
void fake_reset(int fail, int dev) { made = 0; fail_at = fail; device = dev; last = cudaSuccess; }
int fake_made() { return made; }
int fake_live() { return live_streams + live_events; }
int fake_last() { return (int)last; }
int kept() { return qsv::kSideKept; }
void *take() { return qsv::side_take(); }
void give(void *s) { qsv::side_give((qsv::SideStreams *)s); }
}
"""


@pytest.fixture(scope="module")
def side(tmp_path_factory):
    d = tmp_path_factory.mktemp("side")
    src, so = d / "fake.cpp", d / "side.so"
    src.write_text(FAKE)
    # -Bsymbolic: the fake's calls, also in a process that has a CUDA runtime in its global scope
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-Wl,-Bsymbolic",
                    "-I", os.path.join(build.cuda_root(), "include"), "-I", build.CSRC, "-o", str(so), str(src),
                    os.path.join(build.CSRC, "qsv_side.cpp")], check=True, timeout=300)
    lib = ctypes.CDLL(str(so))
    lib.take.restype = ctypes.c_void_p
    lib.give.argtypes = [ctypes.c_void_p]
    lib.kept.restype = ctypes.c_int
    lib.side_stream.restype = ctypes.c_void_p
    lib.side_stream.argtypes = [ctypes.c_void_p, ctypes.c_int]
    lib.fake_capture.argtypes = [ctypes.c_void_p, ctypes.c_int]
    lib.joins.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p]
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


def test_streams_in_another_capture_are_not_joined(side):
    side.fake_reset(-1, 0)
    s = side.take()
    caller, last = 0x77, side.side_stream(s, 2)
    assert side.joins(s, 3, caller)
    side.fake_capture(caller, 5)
    assert side.joins(s, 3, caller)              # free side streams join the caller's capture
    side.fake_capture(last, 5)
    assert side.joins(s, 3, caller)              # and are in it at its next launch
    side.fake_capture(caller, 0)
    assert not side.joins(s, 3, caller) and side.joins(s, 2, caller)
    side.fake_capture(caller, 6)
    assert not side.joins(s, 3, caller)
    side.fake_capture(last, 0)
    side.fake_capture(caller, -1)
    assert not side.joins(s, 1, caller) and side.fake_last() == 0
    side.fake_capture(caller, 0)
    side.give(s)


def test_sets_are_handed_out_again_and_bounded(side):
    side.fake_reset(-1, 20)                      # a device of its own
    start = side.fake_live()
    s = side.take()
    one = side.fake_live() - start
    side.give(s)
    side.fake_reset(-1, 20)
    for _ in range(50):
        s = side.take()
        side.give(s)
    assert side.fake_made() == 0 and side.fake_live() - start == one
    # never the same set twice at a time; not another device's
    some = [side.take() for _ in range(2 * side.kept())]
    assert len(set(some)) == len(some)
    for s in some:
        side.give(s)
    assert side.fake_live() - start == side.kept() * one
    side.fake_reset(-1, 21)
    other = side.take()
    assert other and side.fake_made() > 0        # (its address may be that of a destroyed set)
    side.give(other)


def test_captured_sets_stay_until_their_capture_ends(side):
    side.fake_reset(-1, 22)
    start = side.fake_live()
    held = side.take()
    one = side.fake_live() - start
    side.fake_capture(side.side_stream(held, 1), 9)
    side.give(held)
    s = side.take()
    assert s != held
    some = [s] + [side.take() for _ in range(side.kept())]
    assert held not in some
    for s in some:
        side.give(s)
    assert side.fake_live() - start == side.kept() * one
    side.fake_capture(side.side_stream(held, 1), 0)
    got = [side.take() for _ in range(side.kept())]
    assert held in got and side.fake_live() - start == side.kept() * one
    for s in got:
        side.give(s)
