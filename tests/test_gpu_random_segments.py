"""Sweep kernels on random segments, value for value against the oracle: every window size, windows whose
qubits fall into one to many runs (each staging form), every matrix kind, targets and controls in every slot."""
import os
import sys

import numpy as np
import pytest

from qsv_b200 import compile_circuit, engine, isa
from qsv_b200.generators import random_layer
from oracle import oracle as orc

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from random_segments import random_segment, random_state  # noqa: E402

pytestmark = pytest.mark.gpu

# (n, k, passes, ops): one tile of each size; one to a few tiles; many tiles with scattered high qubits
SHAPES = [(10, 10, 3, 20), (11, 11, 3, 20), (12, 12, 3, 20), (13, 12, 4, 16), (14, 8, 6, 12), (17, 9, 12, 6),
          (19, 12, 12, 8), (20, 7, 16, 4), (21, 12, 10, 10)]


@pytest.mark.parametrize("dtype", ["c64", "c128"])
@pytest.mark.parametrize("shape", SHAPES)
def test_random_segments_exact(shape, dtype):
    torch = pytest.importorskip("torch")
    n, k, passes, ops = shape
    old = engine.set_jit("off")
    try:
        for seed in range(4):
            seg = random_segment(n, k, passes, ops, 100 * n + seed, dtype)
            x = random_state(n, seed, dtype)
            t = torch.from_numpy(x.copy()).cuda()
            engine.run_segment(t, seg)
            torch.cuda.synchronize()
            assert engine.device_status() == 0
            ref = orc.run_segment(x.copy(), seg)
            assert np.array_equal(t.cpu().numpy(), ref), f"n={n} k={k} seed={seed}"
    finally:
        engine.set_jit(old)


@pytest.mark.parametrize("mode", ["eager", "coarse"])
@pytest.mark.parametrize("shape", [(10, 10, 2, 20), (12, 12, 2, 20), (13, 12, 2, 20), (17, 9, 8, 6), (19, 12, 4, 8)])
def test_random_segments_specialised_exact(shape, mode):
    torch = pytest.importorskip("torch")
    n, k, passes, ops = shape
    segs = [random_segment(n, k, passes, ops, 7 * n)]
    # one U3 (real first entry) on every qubit: targets in every slot, lane bits among them
    layer, _, _ = compile_circuit(random_layer(n, 2, n), n, min(n, 12))
    segs += [p for what, p in layer]
    x = random_state(n, n)
    old = engine.set_jit(mode)
    try:
        for seg in segs:
            engine.jit_prepare(seg, n)
            before = engine.jit_info()["jit_launches"]
            t = torch.from_numpy(x.copy()).cuda()
            engine.run_segment(t, seg)
            torch.cuda.synchronize()
            assert engine.device_status() == 0
            assert engine.jit_info()["jit_launches"] > before
            x = orc.run_segment(x.copy(), seg)
            assert np.array_equal(t.cpu().numpy(), x)
    finally:
        engine.set_jit(old)


@pytest.mark.parametrize("dtype", ["c64", "c128"])
@pytest.mark.parametrize("lanes", [0, 1, 2])
@pytest.mark.parametrize("n", [11, 12, 13])
def test_most_phases(n, lanes, dtype):
    """96 ops whose targets never repeat within a phase: as many phases as a sweep can need, whatever the knob."""
    torch = pytest.importorskip("torch")
    k = min(n, 12)
    seg = random_segment(n, k, 2, 48, n, dtype).copy()
    words = isa.OP_WORDS_C128 if dtype == "c128" else isa.OP_WORDS
    at = isa.HDR_WORDS
    for p in range(2):
        seg[at:at + 8] = [0, 0, 0, 48, 0, 0, 0, 0]
        at += isa.PASS_WORDS
        for o in range(48):
            rec = seg[at:at + words]
            mats = rec[8:].view(np.float64 if dtype == "c128" else np.float32)
            mats[:8] = mats[8:] = [0.6, 0.1, 0.3, -0.5, -0.3, -0.5, 0.6, -0.1]        # dense: needs a slot
            rec[1], rec[2] = 3 + (5 * o) % (k - 3), 0
            at += words
    x = random_state(n, n, dtype)
    old = engine.set_jit("off")
    engine.set_phase_lanes(lanes)
    try:
        t = torch.from_numpy(x.copy()).cuda()
        engine.run_segment(t, seg)
        torch.cuda.synchronize()
        assert engine.device_status() == 0
        assert np.array_equal(t.cpu().numpy(), orc.run_segment(x.copy(), seg))
    finally:
        engine.set_phase_lanes(1)
        engine.set_jit(old)
