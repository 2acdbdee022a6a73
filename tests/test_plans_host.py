"""The sweep plans that qsv_plan_segment and qsv_plan_interp list, host side: the tensor-map boxes of every sweep hold
exactly its tiles, and the interpreter's phases place every op where its slot and control split say."""
import numpy as np
import pytest

import qsv_b200 as q
from qsv_b200 import engine, generators as gen

SKIP, UNI_DIAG, CTRL_DIAG1, MUX, CTRL_DIAG1_SEL = 0, 2, 5, 7, 9
CTRL = 1
DIAG1 = 4
SLOT_COMP, SLOT_REG0, SLOT_BASE, SLOT_LANE0 = 0, 1, 7, 8


def spread(x, bits):
    """Bit i of x on bit bits[i]."""
    out = np.zeros_like(x)
    for i, b in enumerate(bits):
        out |= ((x >> i) & 1) << b
    return out


def box_addresses(sw, n, T):
    """The state index of every shared-memory position of tile T, by its boxes: each dim's coordinate takes the next
    bits of T above the box; with xbits the last dim spans window bits too, which select one of the boxes."""
    xbits, rank = sw["tma_xbits"], sw["tma_rank"]
    boxbits = sw["kw"] - xbits
    assert boxbits == sum(sw["tdim_box"]) and xbits <= min(5, len(sw["H"])) and (xbits == 0 or rank == 5)
    p = np.arange(1 << sw["kw"], dtype=np.int64)
    box, e = p >> boxbits, p & ((1 << boxbits) - 1)
    addr, start, t = np.zeros_like(p), 0, T
    for d in range(rank):
        f, w = sw["tdim_free"][d], sw["tdim_box"][d]
        if d == 4 and xbits:
            c = np.full_like(p, t << w)
            for i in range(xbits):
                h = sw["H"][len(sw["H"]) - xbits + i] - start
                c = ((c >> h) << (h + 1)) | (((box >> i) & 1) << h) | (c & ((1 << h) - 1))
        else:
            c = np.full_like(p, (t & ((1 << f) - 1)) << w)
        addr += (c + (e & ((1 << w) - 1))) << start
        e >>= w
        t >>= f
        start += f + w
    assert start == n
    return addr


CIRCUITS = [
    (10, 8, lambda: gen.random_layer(10, 4, 1)),
    (11, 9, lambda: gen.random_layer_ccx(11, 3, 2)),
    (13, 12, lambda: gen.qft(13)),
    (16, 12, lambda: gen.zoo(16, 5)),
    (17, 12, lambda: gen.rqc(17, 6, 3)),
    (18, 12, lambda: gen.random_layer_ccx(18, 6, 5)),
    (22, 12, lambda: gen.random_layer_ccx(22, 5, 7)),
    (30, 12, lambda: gen.random_layer_ccx(30, 3, 9)),
]


def plans(n, k, maker):
    prog, _, _ = q.compile_circuit(maker(), n, k)
    for kind, seg in prog:
        if kind == "segment":
            yield engine.plan_segment(seg, n), engine.plan_interp(seg, n)


@pytest.mark.parametrize("n,k,maker", CIRCUITS)
def test_boxes_hold_the_tiles(n, k, maker):
    rng = np.random.default_rng(n)
    for spec, interp in plans(n, k, maker):
        for sw in spec + interp:
            if not sw["tma_rank"]:
                assert sw["tma_xbits"] == 0
                continue
            free = [b for b in range(n) if b not in sw["window"]]
            ntiles = 1 << len(free)
            for T in {0, ntiles - 1, *(int(x) for x in rng.integers(0, ntiles, 3))}:
                want = spread(np.arange(1 << sw["kw"], dtype=np.int64), sw["window"]) | int(spread(np.int64(T), free))
                assert np.array_equal(box_addresses(sw, n, T), want)


def test_windows_of_many_runs_have_several_boxes():
    """(Otherwise the test above would not see them.)"""
    assert any(sw["tma_xbits"] for spec, interp in plans(*CIRCUITS[-1]) for sw in spec + interp)


@pytest.mark.parametrize("n,k,maker", CIRCUITS)
def test_interpreter_places_every_op(n, k, maker):
    for spec, interp in plans(n, k, maker):
        assert len(spec) == len(interp)
        for sp, sw in zip(spec, interp):
            kw = sw["kw"]
            assert (sw["lo"], sw["H"], kw) == (sp["lo"], sp["H"], sp["kw"]) and len(sw["ops"]) == len(sp["ops"])
            at = 0
            for ph in sw["phases"]:
                assert ph["op_begin"] == at
                at = ph["op_end"]
                assert len(ph["reg_bits"]) == (3 if kw >= 12 else 2)
                lanes = ph["lane_lo"] + ph["lane_bits"]
                assert sorted([0] + lanes + ph["reg_bits"] + ph["warp_bits"]) == list(range(kw))
                # conflict-free 16-byte accesses: lane bits 0-2 on tile bits 1-3, or on 1+l / 4+l in a swizzled tile
                for l, b in enumerate(ph["lane_lo"]):
                    assert b == 1 + l or (sw["swizzled"] and b == 4 + l)
                for o in range(ph["op_begin"], ph["op_end"]):
                    op, so = sw["ops"][o], sp["ops"][o]
                    assert (op["tbit"], op["cmask"], op["kind"]) == (so["tbit"], so["cmask"], so["kind"])
                    assert np.array_equal(op["m0"], so["m0"]) and np.array_equal(op["m1"], so["m1"])
                    t, slot = op["tbit"], op["slot"]
                    if t == 0:
                        assert slot == SLOT_COMP
                    elif t in ph["reg_bits"]:
                        assert slot == SLOT_REG0 + ph["reg_bits"].index(t)
                    elif t in lanes:
                        assert slot == SLOT_LANE0 + lanes.index(t)
                    else:                        # a warp bit: only for ops that act on each amplitude alone
                        assert slot == SLOT_BASE
                        assert (op["variant"] in (SKIP, UNI_DIAG, CTRL_DIAG1, CTRL_DIAG1_SEL) or
                                (op["variant"] == MUX and op["kind"] == CTRL and op["cls1"] == DIAG1))
                    assert op["cm_reg"] == sum(((op["cmask"] >> b) & 1) << i for i, b in enumerate(ph["reg_bits"]))
                    assert op["cm_thr"] == op["cmask"] & ~(1 | sum(1 << b for b in ph["reg_bits"]))
            assert at == len(sw["ops"])
