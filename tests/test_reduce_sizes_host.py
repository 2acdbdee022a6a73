"""The grid of the FP64 reductions (csrc/qsv_reduce.h), host side: it depends on the qubit count alone, covers the
state, keeps its partials inside the scratch that callers are told to bring, and fits the fixed one."""
import os
import subprocess

from qsv_b200 import build, engine

SRC = r"""
#include <cstdio>
#include "qsv_reduce.h"
int main() {
    for (int n = 10; n <= 34; n++) {
        const qsv::ReduceGrid g = qsv::reduce_grid(n);       // (no other argument: not the device's SM count)
        std::printf("%d %lld %d %lld\n", n, (long long)g.blocks, g.nout, qsv::reduce_room(n));
    }
}
"""


def test_reduction_grid(tmp_path):
    src, exe = tmp_path / "grid.cpp", tmp_path / "grid"
    src.write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-I", build.CSRC, "-o", str(exe), str(src)], check=True, timeout=120)
    rows = [[int(x) for x in ln.split()] for ln in
            subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=60).stdout.splitlines()]
    assert [r[0] for r in rows] == list(range(10, 35))
    L = engine.load()
    for n, blocks, nout, room in rows:
        assert 1 <= blocks and blocks * nout <= room
        assert room * 8 <= L.qsv_reduce_scratch_bytes(n) and room <= 32768
        chunks = 1 << max(0, n - 13)
        assert blocks <= chunks
        # one chunk a block: its 13 bits are enough; chunks in turn: all bits
        assert (nout == 14 and blocks == chunks) or nout == n + 1
        if n >= 24:
            assert blocks == min(592, room // (n + 1))


def test_reductions_take_no_sm_count():
    text = open(os.path.join(build.CSRC, "qsv_aux.cu")).read()
    for name in ("launch_reduce_t", "launch_reduce", "launch_reduce_noalloc"):
        head = text[text.index(f"cudaError_t {name}("):]
        assert "nsm" not in head[:head.index("{")]
