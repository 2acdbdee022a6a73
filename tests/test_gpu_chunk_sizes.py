"""Chunk probabilities (qsv_chunk_probs_f64) at the sizes where the work per chunk changes hands: a block per chunk below
256 amplitudes, a warp up to 8 KiB, a block with eight loads per thread and turn above, whole states in one chunk."""
import numpy as np
import pytest

from qsv_b200 import engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
@pytest.mark.parametrize("n,bits", [(10, 0), (10, 7), (10, 8), (10, 9), (12, 10), (13, 11), (14, 12), (13, 13), (17, 17),
                                    (18, 9), (18, 10), (18, 11), (18, 12)])
def test_chunk_sums(n, bits, dtype, offset):
    import torch
    rng = np.random.default_rng(n * 40 + bits)
    x = (rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)).astype(dtype)
    whole = torch.zeros((1 << n) + offset, dtype=getattr(torch, dtype), device="cuda")
    state = whole[offset:]                       # offset 1: complex64 off the 16-byte boundary
    state.copy_(torch.from_numpy(x))
    got = engine.chunk_probs_f64(state, bits).cpu().numpy()
    p = x.real.astype(np.longdouble) ** 2 + x.imag.astype(np.longdouble) ** 2
    want = p.reshape(-1, 1 << bits).sum(axis=1)
    # terms of one sign: a rounding per product and sum, at most 2^bits / 32 sums one after the other and a tree
    bound = ((1 << bits) / 32 + 16) * 2.0 ** -53
    assert got.shape == want.shape and np.max(np.abs(got - want) / want) <= bound
