"""A phase leaves the amplitudes it does not select alone, bit for bit: also an infinity, a NaN and the sign of a zero
that sit beside a selected amplitude in the same 16-byte slot (target or control on tile bit 0)."""
import numpy as np
import pytest

from qsv_b200 import engine, isa

pytestmark = pytest.mark.gpu

N = 12
ANGLE = 0.7


def _segment(t, c, dtype):
    c128 = dtype == "c128"
    fl = np.zeros(16, dtype=np.float64 if c128 else np.float32)
    p = np.exp(1j * ANGLE)
    fl[[0, 8]] = 1.0
    fl[6:8] = fl[14:16] = [p.real, p.imag]
    if c is not None:
        fl[6:8] = [1.0, 0.0]
    return np.concatenate([
        np.array([isa.MAGIC, N, 1, N, isa.DTYPE_C128 if c128 else isa.DTYPE_C64, 0, 0, 0, 0, 0, 0, 1, 0, 0, 0, 0,
                  isa.OP_MUX2, t, 0 if c is None else 1 << c, 0, 0, 0, 0, 0], dtype=np.int32), fl.view(np.int32)])


@pytest.mark.parametrize("mode,dtype", [("off", "c64"), ("batch", "c64"), ("eager", "c64"), ("off", "c128")])
def test_phase_leaves_unselected_amplitudes(mode, dtype):
    torch = pytest.importorskip("torch")
    real = np.float64 if dtype == "c128" else np.float32
    rng = np.random.default_rng(2)
    i = np.arange(1 << N)
    old = engine.set_jit("eager" if mode == "eager" else "off")
    try:
        pairs = [(t, c) for t in (0, 1, 6, 11) for c in (None, 0, 3, 10) if t != c]
        for t, c in pairs[::3] if mode == "eager" else pairs:
            seg = _segment(t, c, dtype)
            picked = ((i >> t) & 1 == 1) & ((i >> c) & 1 == 1 if c is not None else True)
            x = rng.standard_normal((1 << N, 2)).astype(real)
            odd = np.array([[np.inf, 1], [-1, -np.inf], [np.nan, 2], [-0.0, -3], [3, -0.0], [-0.0, -0.0]], dtype=real)
            x[~picked] = odd[np.arange((~picked).sum()) % len(odd)]
            d = torch.from_numpy(x.copy()).cuda()
            s = torch.view_as_complex(d)
            if mode == "batch":
                b = engine.SmallBatch()
                b.add(s, [seg])
                b.upload()
                b.launch()
            else:
                engine.run_segment(s, seg)
            torch.cuda.synchronize()
            y = d.cpu().numpy()
            word = np.uint64 if dtype == "c128" else np.uint32
            assert np.array_equal(y[~picked].view(word), x[~picked].view(word)), (t, c)
            # one product of two rounded factors and a sum per part: 4 units in the last place of the largest term
            z = (x[picked, 0].astype(np.float64) + 1j * x[picked, 1]) * np.exp(1j * ANGLE)
            assert np.max(np.abs(y[picked, 0] + 1j * y[picked, 1] - z)) < 4 * np.finfo(real).eps * np.abs(x[picked]).max()
        assert engine.device_status() == 0
    finally:
        engine.set_jit(old)
