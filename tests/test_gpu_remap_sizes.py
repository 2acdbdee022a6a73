"""The permutation kernel at the edges of its tiles: states of one tile and fewer bits than a tile asks for, both
element types, permutations that keep, exchange, rotate and reverse the low bits; exact (pure data movement)."""
import numpy as np
import pytest

from qsv_b200 import engine

pytestmark = pytest.mark.gpu


def _perms(n, rng):
    yield list(range(n))
    yield list(range(n))[::-1]
    yield list(range(1, n)) + [0]
    yield [n - 1] + list(range(n - 1))
    p = list(range(n))
    p[2], p[n - 1] = p[n - 1], p[2]
    yield p
    for _ in range(3):
        yield [int(x) for x in rng.permutation(n)]


@pytest.mark.parametrize("dtype", ["c64", "c128"])
@pytest.mark.parametrize("n", [10, 11, 12, 13, 17, 21])
def test_remap_exact(n, dtype):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    x = np.arange(1 << n).astype(np.complex128 if dtype == "c128" else np.complex64) * (1 - 2j)
    src = torch.from_numpy(x).cuda()
    y = np.arange(1 << n)
    for perm in _perms(n, rng):
        dst = torch.empty_like(src)
        engine.remap(src, dst, perm)
        index = np.zeros(1 << n, dtype=np.int64)
        for j in range(n):
            index |= ((y >> j) & 1) << perm[j]
        assert np.array_equal(dst.cpu().numpy(), x[index]), perm
