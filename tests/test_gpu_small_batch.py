"""Whole-circuit batches whose qubit counts run side by side: the launch is ordered after the caller's earlier work
and before its later work on the same stream, on a stream of the caller's and inside a graph capture, for one and
for several counts; values equal the oracle's."""
import numpy as np
import pytest

from qsv_b200 import compile_circuit, engine
from qsv_b200.generators import random_layer_ccx
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns", [(12,), (10, 13), (10, 11, 12, 13, 13, 10)])
@pytest.mark.parametrize("graph", [False, True])
def test_side_by_side(ns, graph):
    torch = pytest.importorskip("torch")
    s = torch.cuda.Stream()
    refs, states = [], []
    batch = engine.SmallBatch()
    with torch.cuda.stream(s):
        for i, n in enumerate(ns):
            prog, _, _ = compile_circuit(random_layer_ccx(n, 3 + i, i), n, n)
            x = np.zeros(1 << n, dtype=np.complex64)
            x[0] = 1
            for _, seg in prog:
                x = orc.run_segment(x, seg)
            refs.append(x)
            states.append(torch.empty(1 << n, dtype=torch.complex64, device="cuda"))
            batch.add(states[-1], [seg for _, seg in prog])
        batch.upload()

        def once():
            for st in states:
                engine.zero_state(st)
            batch.launch()
            return [st.clone() for st in states]

        outs = once()
        if graph:
            s.synchronize()
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=s):
                outs = once()
            for _ in range(3):
                g.replay()
    torch.cuda.synchronize()
    assert engine.device_status() == 0
    for out, ref in zip(outs, refs):
        assert np.array_equal(out.cpu().numpy(), ref)
