"""Every matrix kind of an op, in every place its target and its control can take in a sweep, value for value against
the oracle.

An op of a QSV2 segment chooses between two matrices. The kinds here are the ones a kernel has code of its own for
(dense, dense with a real first entry, diagonal, phase, exchange, identity); a target can sit on tile bit 0 (inside a
16-byte slot), on a register bit or on a lane bit, a control on any of those or on a warp bit. In every pair of places
each kind is applied under the control alone, as the first of two matrices and as the second. The segments are made
until the sweep plan shows every combination, so that none is left to chance; kernels specialised to their exact
structure, the interpreter and the whole-circuit batch kernel run all of them, kernels of their coarse structure (which
knows dense ops and exchanges only) every third."""
import numpy as np
import pytest

from qsv_b200 import engine, isa
from oracle import oracle as orc

N = 12                      # one tile of 2^12 amplitudes: tile bit = qubit
OPS = 32
KINDS = ["dense", "real00", "diag", "phase", "swap", "ident"]


def _matrix(rng, kind):
    q, _ = np.linalg.qr(rng.standard_normal((2, 2)) + 1j * rng.standard_normal((2, 2)))
    if kind == "dense":
        return q
    if kind == "real00":
        m = q * (q[0, 0].conj() / abs(q[0, 0]))
        m[0, 0] = m[0, 0].real
        return m
    if kind == "diag":
        return np.diag(np.exp(1j * rng.uniform(0, 2 * np.pi, 2)))
    if kind == "phase":
        return np.diag([1.0, np.exp(1j * rng.uniform(0, 2 * np.pi))])
    return np.array([[0, 1], [1, 0]], dtype=complex) if kind == "swap" else np.eye(2, dtype=complex)


def _segment(rng, ops):
    """ops: (target, control or None, kind of M0, kind of M1)."""
    words = [np.array([isa.MAGIC, N, 1, N, isa.DTYPE_C64, 0, 0, 0, 0, 0, 0, len(ops), 0, 0, 0, 0], dtype=np.int32)]
    for t, c, k0, k1 in ops:
        m0 = _matrix(rng, k0)
        m1 = m0 if c is None else _matrix(rng, k1)
        fl = np.empty(16, dtype=np.float32)
        for i, m in enumerate((m0, m1)):
            fl[8 * i:8 * i + 8:2] = m.reshape(-1).real
            fl[8 * i + 1:8 * i + 8:2] = m.reshape(-1).imag
        words += [np.array([isa.OP_MUX2, t, 0 if c is None else 1 << c, 0, 0, 0, 0, 0], dtype=np.int32),
                  fl.view(np.int32)]
    return np.concatenate(words)


def _roles(seg):
    """Per op: where its target and its control (if any) sit in the plan of the one sweep."""
    (sw,) = engine.plan_segment(seg, N)
    out = []
    for ph in sw["phases"]:
        role = {0: "comp"}
        role.update({b: "reg" for b in ph["reg_bits"]})
        role.update({b: "lane" for b in ph["lane_bits"] + ph["lane_lo"]})
        role.update({b: "warp" for b in ph["warp_bits"]})
        for o in sw["ops"][ph["op_begin"]:ph["op_end"]]:
            at = "comp" if o["slot"] == 0 else "reg" if o["slot"] < 7 else "lane"
            out.append((at, role[o["cmask"].bit_length() - 1] if o["cmask"] else None))
    return out


def _wanted():
    # (first, second matrix): under the control alone; a choice of two, each kind once on either side
    pairs = [("ident", k) for k in KINDS[:-1]]
    pairs += [("dense", k) for k in KINDS] + [(k, "dense") for k in KINDS[1:-1]] + [("diag", "swap"), ("swap", "ident")]
    want = {}
    for t in ("comp", "reg", "lane"):
        want[t, None] = [(k, k) for k in KINDS]
        for c in ("comp", "reg", "lane", "warp"):
            if (t, c) != ("comp", "comp"):
                want[t, c] = list(pairs)
    return want


def segments():
    """Segments in whose plans every combination of _wanted() occurs."""
    want, segs, seed = _wanted(), [], 0

    def give(ops):
        """ops with kinds that their places still lack, and which of them have such kinds."""
        left = {place: list(kinds) for place, kinds in want.items()}
        out, new = [], []
        for op, place in zip(ops, _roles(_segment(rng, ops))):
            new.append(bool(left.get(place)))
            out.append(op[:2] + (left[place].pop() if new[-1] else ("dense", "dense")))
        return out, new

    while any(want.values()):
        assert seed < 500, "the segments no longer cover every combination"
        rng = np.random.default_rng(seed)
        seed += 1
        some = [0] + [int(b) for b in rng.choice(np.arange(1, N), 7, replace=False)]
        ops = []
        for _ in range(OPS):
            t = int(rng.choice(some))
            c = None if rng.integers(8) == 0 else int(rng.choice([b for b in range(N) if b != t]))
            ops.append((t, c, "dense", "dense"))
        # the places follow from targets and controls alone: lay out, and leave out ops whose places lack no kind (the
        # rest is laid out anew)
        ops, new = give(ops)
        while any(new) and not all(new):
            fewer, fresh = give([op for op, x in zip(ops, new) if x])
            if sum(fresh) < 0.8 * sum(new):
                break
            ops, new = fewer, fresh
        if sum(new) < min(16, sum(map(len, want.values())) / 4):
            continue
        segs.append(_segment(rng, ops))
        for op, place in zip(ops, _roles(segs[-1])):
            if op[2:] in want.get(place, ()):
                want[place].remove(op[2:])
    return segs


def test_every_combination_is_planned():
    assert len(segments()) >= 4


@pytest.mark.gpu
@pytest.mark.timeout(900)
@pytest.mark.parametrize("mode", ["eager", "coarse", "off", "batch"])
def test_matrix_kinds_exact(mode):
    torch = pytest.importorskip("torch")
    segs = segments()[::3 if mode == "coarse" else 1]
    rng = np.random.default_rng(5)
    x = (rng.standard_normal(1 << N) + 1j * rng.standard_normal(1 << N)).astype(np.complex64)
    x /= np.float32(np.linalg.norm(x))
    old = engine.set_jit("off" if mode == "batch" else mode)
    try:
        if mode in ("eager", "coarse"):
            before = engine.jit_info()["jit_launches"]
            for seg in segs:
                engine.jit_prepare(seg, N)
        for i, seg in enumerate(segs):
            t = torch.from_numpy(x.copy()).cuda()
            if mode == "batch":
                b = engine.SmallBatch()
                b.add(t, [seg])
                b.upload()
                b.launch()
            else:
                engine.run_segment(t, seg)
            torch.cuda.synchronize()
            assert engine.device_status() == 0
            assert np.array_equal(t.cpu().numpy(), orc.run_segment(x.copy(), seg)), f"segment {i}"
        if mode in ("eager", "coarse"):
            assert engine.jit_info()["jit_launches"] - before == len(segs)
    finally:
        engine.set_jit(old)
