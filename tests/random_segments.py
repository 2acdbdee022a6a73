"""Random QSV2 segments for the engine's tests: passes over random windows (so that a tile's qubits fall into
one to many runs), targets and controls anywhere in the window, and every matrix kind the engine has a code
path for (dense, dense with a real first entry, diagonal, phase, exchange, identity; as one matrix, under
controls, and as a general choice between two matrices)."""
import numpy as np

from qsv_b200 import isa


def _unitary(rng):
    q, _ = np.linalg.qr(rng.standard_normal((2, 2)) + 1j * rng.standard_normal((2, 2)))
    return q


def _matrix(rng, kind):
    if kind == "dense":
        return _unitary(rng)
    if kind == "real00":
        m = _unitary(rng)
        return m * (abs(m[0, 0]) / m[0, 0])
    if kind == "diag":
        return np.diag(np.exp(1j * rng.uniform(0, 2 * np.pi, 2)))
    if kind == "phase":
        return np.diag([1.0, np.exp(1j * rng.uniform(0, 2 * np.pi))])
    if kind == "swap":
        return np.array([[0, 1], [1, 0]], dtype=complex)
    return np.eye(2, dtype=complex)


KINDS = ["dense", "real00", "diag", "phase", "swap", "ident"]


def random_segment(n, k, passes, ops, seed, dtype="c64", max_high=4):
    rng = np.random.default_rng(seed)
    words = [np.array([isa.MAGIC, n, passes, k, isa.DTYPE_C128 if dtype == "c128" else isa.DTYPE_C64, 0, 0, 0],
                      dtype=np.int32)]
    for _ in range(passes):
        m = int(rng.integers(0, min(max_high, k - 3, n - k + 1) + 1)) if n > k else 0
        h = sorted(int(x) for x in rng.choice(np.arange(k - m, n), m, replace=False)) if m else []
        slots = h + [0] * (4 - len(h))
        words.append(np.array([m, slots[0], slots[1], ops, slots[2], slots[3], 0, 0], dtype=np.int32))
        for _ in range(ops):
            # high window qubits and the lowest qubits are where layouts differ: draw them often
            t = int(rng.choice([rng.integers(k), rng.integers(min(k, 7)), k - 1 - rng.integers(max(1, m))]))
            nctrl = int(rng.choice([0, 0, 1, 1, 2, 3]))
            others = [b for b in range(k) if b != t]
            cmask = sum(1 << int(b) for b in rng.choice(others, nctrl, replace=False))
            m1 = _matrix(rng, rng.choice(KINDS))
            # no controls: one matrix; under controls: mostly identity elsewhere, sometimes a second matrix
            m0 = m1 if not cmask else (np.eye(2) if rng.integers(4) else _matrix(rng, rng.choice(KINDS)))
            fl = np.empty(16, dtype=np.float64 if dtype == "c128" else np.float32)
            for i, mat in enumerate((m0, m1)):
                fl[8 * i:8 * i + 8:2] = np.asarray(mat).reshape(-1).real
                fl[8 * i + 1:8 * i + 8:2] = np.asarray(mat).reshape(-1).imag
            words.append(np.concatenate([np.array([isa.OP_MUX2, t, cmask, 0, 0, 0, 0, 0], dtype=np.int32),
                                         fl.view(np.int32)]))
    return np.concatenate(words)


def random_state(n, seed, dtype="c64"):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    return (x / np.linalg.norm(x)).astype(np.complex128 if dtype == "c128" else np.complex64)
