"""A whole-circuit batch of several qubit counts, launched on one stream while its launch on another stream is being
captured: the capture is left alone, and both launches give the oracle's values."""
import numpy as np
import pytest

from qsv_b200 import compile_circuit, engine
from qsv_b200.generators import random_layer_ccx
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def test_launch_beside_a_capture():
    torch = pytest.importorskip("torch")
    ns = (10, 12, 13, 12)
    batch = engine.SmallBatch()
    segs, states = [], []
    rng = np.random.default_rng(4)
    xs = [(rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)).astype(np.complex64) for n in ns]
    for i, n in enumerate(ns):
        prog, _, _ = compile_circuit(random_layer_ccx(n, 4, i), n, n)
        segs.append([seg for _, seg in prog])
        states.append(torch.from_numpy(xs[i].copy()).cuda())
        batch.add(states[-1], segs[-1])
    batch.upload()
    torch.cuda.synchronize()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=a, capture_error_mode="thread_local"):
        batch.launch(a)
        batch.launch(b)              # not captured: runs now
        batch.launch(a)              # again into the same capture
    b.synchronize()
    refs = [x.copy() for x in xs]

    def check(times):
        for i, st in enumerate(states):
            for _ in range(times):
                for seg in segs[i]:
                    refs[i] = orc.run_segment(refs[i], seg)
            assert np.array_equal(st.cpu().numpy(), refs[i]), f"circuit {i}"

    check(1)
    g.replay()                       # two launches
    torch.cuda.synchronize()
    check(2)
    assert engine.device_status() == 0
