"""FP64 reductions, chunk probabilities and the Born sampler at the edges of their kernels' ranges: one block and
many, one chunk per block and grids that take chunks in turn, chunk sizes on both sides of the warp form, states
that start between two 16-byte boundaries, shots that do not fill a block. Reductions against NumPy in FP64
(relative 1e-12 of the total: at most 2^23 terms, each rounded to 2^-53, summed in trees of depth below 64);
samples must lie where the exact cumulative sums put them, to 1e-12 of the total."""
import numpy as np
import pytest

from qsv_b200 import engine

pytestmark = pytest.mark.gpu


def _state(torch, n, dtype, seed, offset=0):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    x[rng.random(1 << n) < 0.3] = 0                     # amplitudes that must never be drawn
    x = x.astype(np.complex128 if dtype == "c128" else np.complex64)
    buf = torch.zeros((1 << n) + offset, dtype=torch.from_numpy(x).dtype, device="cuda")
    buf[offset:] = torch.from_numpy(x).cuda()
    return x, buf[offset:]


def _probs(x):
    x = x.astype(np.complex128)
    return x.real ** 2 + x.imag ** 2


@pytest.mark.parametrize("dtype,offset", [("c64", 0), ("c64", 1), ("c128", 0)])
@pytest.mark.parametrize("n", [10, 12, 13, 14, 17, 22, 23])
def test_reduction(n, dtype, offset):
    torch = pytest.importorskip("torch")
    x, t = _state(torch, n, dtype, n, offset)
    p = _probs(x)
    z = engine.reduce_f64(t).cpu().numpy()
    ref = [p.sum()] + [p.reshape(-1, 2, 1 << q)[:, 0].sum() - p.reshape(-1, 2, 1 << q)[:, 1].sum() for q in range(n)]
    assert np.max(np.abs(z - np.array(ref))) <= 1e-12 * ref[0]


@pytest.mark.parametrize("dtype,offset", [("c64", 0), ("c64", 1), ("c128", 0)])
@pytest.mark.parametrize("n,bits", [(10, 0), (14, 7), (14, 8), (18, 12), (18, 13), (18, 14), (20, 20)])
def test_chunk_probabilities(n, bits, dtype, offset):
    torch = pytest.importorskip("torch")
    x, t = _state(torch, n, dtype, n + bits, offset)
    p = _probs(x)
    got = engine.chunk_probs_f64(t, bits).cpu().numpy()
    assert np.max(np.abs(got - p.reshape(-1, 1 << bits).sum(axis=1))) <= 1e-12 * p.sum()


@pytest.mark.parametrize("dtype,offset", [("c64", 0), ("c64", 1), ("c128", 0)])
@pytest.mark.parametrize("n,shots", [(10, 1), (11, 7), (13, 9), (20, 1000), (25, 300)])
def test_samples(n, shots, dtype, offset):
    torch = pytest.importorskip("torch")
    x, t = _state(torch, n, dtype, 3 * n, offset)
    p = _probs(x)
    cdf = np.cumsum(p)
    u = np.random.default_rng(n).random(shots)
    u[0] = 0.0
    got = engine.sample_f64(t, u).cpu().numpy()
    draw, tol = u * cdf[-1], 1e-12 * cdf[-1]
    assert np.all(cdf[got] >= draw - tol) and np.all(cdf[got] - p[got] <= draw + tol)
    assert np.all(p[got] > 0)
