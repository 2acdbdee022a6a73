"""The work this framework's users have it do, as cases that can be timed and compared.

Every case goes through a public entry point and is described by plain values (kind, sizes, element type,
options). ``prepare`` makes what a user's program holds before the call, from the seed alone; ``run`` is one
pass; ``exact`` is the same result in 64 bits, from plain torch.

Kinds:
  circuit   a compiled circuit on a resident device state: ``engine.zero_state``, then every segment of the
            program with ``engine.run_segment`` (as ``precision.run_state`` and the benchmark do). ``jit`` is
            the specialised-kernel mode the program runs under: "eager" (kernels of its exact structures are
            prepared once, as for a circuit that is run over and over), "coarse" (kernels shared by every
            circuit of a family), "off" (no kernel was made for it: the first run of any circuit, and circuits
            whose structures never repeat). complex128 circuits have no specialised kernels.
  remap     ``engine.remap``: a random permutation of all index bits into a second state.
  reduce    ``engine.reduce_f64``: norm and every <Z_q> of a state.
  sample    ``engine.sample_f64``: Born-rule samples of a state.
  batch     ``batch.BatchRunner``: many circuits per replay of one captured CUDA graph, with their reductions
            and a sample of final states read back to the host.
  small     ``engine.SmallBatch``: circuits of 10..13 qubits, each run whole by one thread block.
  runtime   ``runtime.SVRuntime.run``: from a host circuit to counts and the final state on the host,
            compilation included (the latency of a single small request).

Circuit families: ``rl`` (a U3 on every qubit, then a CX brickwork), ``rqc`` (one of rx, ry, rz, t, h on every
qubit, then a CZ brickwork), ``ccx`` (U3s, a CZ brickwork and Toffolis on random triples), ``vqe`` (ry rz on
every qubit and a CX ladder) and ``qft`` (of a random product state).
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    """This repository's package (its directory has dashes in its name) as ``qsv_b200``."""
    if "qsv_b200" not in sys.modules:
        pkg = os.path.join(ROOT, "u55c-statevector-30q_b200")
        spec = importlib.util.spec_from_file_location("qsv_b200", os.path.join(pkg, "__init__.py"),
                                                      submodule_search_locations=[pkg])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["qsv_b200"] = mod
        spec.loader.exec_module(mod)
    return importlib.import_module("qsv_b200")


_package()
from qsv_b200 import batch as _batch  # noqa: E402
from qsv_b200 import engine as _engine  # noqa: E402
from qsv_b200 import runtime as _runtime  # noqa: E402
from qsv_b200.circuit import Circuit  # noqa: E402
from qsv_b200.compiler import compile_circuit  # noqa: E402

TWO_PI = 2 * math.pi
K = 12                      # tile exponent of the compiled streams (the runtime's default)


# ------------------------------------------------------------------------------------------------ cases
def listed():
    return [
        # the 30-qubit random-layer circuit the benchmark is quoted on, run repeatedly (kernels prepared)
        dict(name="rl30", kind="circuit", family="rl", n=30, depth=24, dtype="c64", jit="eager"),
        # a transform of a prepared state: controlled phases between all pairs of qubits
        dict(name="qft28", kind="circuit", family="qft", n=28, depth=1, dtype="c64", jit="eager"),
        # random circuits of one family, a new one each time, through the family's shared kernels
        dict(name="rqc28", kind="circuit", family="rqc", n=28, depth=10, dtype="c64", jit="coarse"),
        # the first run of a circuit: nothing was prepared for it
        dict(name="rqc27_first", kind="circuit", family="rqc", n=27, depth=10, dtype="c64", jit="off"),
        # the largest circuits of a mixed batch or a service: Toffolis anywhere, structures never repeat
        dict(name="ccx24_first", kind="circuit", family="ccx", n=24, depth=20, dtype="c64", jit="off"),
        # the FP64 path of precision studies
        dict(name="ccx27_c128", kind="circuit", family="ccx", n=27, depth=8, dtype="c128", jit="off"),
        # bringing a state to logical qubit order
        dict(name="remap29", kind="remap", n=29, dtype="c64"),
        # observables of a large state
        dict(name="reduce30", kind="reduce", n=30, dtype="c64"),
        # counts from a large state
        dict(name="sample28", kind="sample", n=28, dtype="c64", shots=1024),
        # a mixed batch of small and middling circuits per graph replay
        dict(name="batch", kind="batch", count=48, n_min=10, n_max=20, depth_min=5, depth_max=40),
        # many small circuits in one launch
        dict(name="small", kind="small", count=128, n_min=10, n_max=13, depth_min=5, depth_max=40),
        # one small request from a host circuit to counts: latency
        dict(name="runtime16", kind="runtime", family="rqc", n=16, depth=10, dtype="c64", shots=1024),
    ]


def draw(rng):
    """One more case of the ranges the listed ones stand for: the smallest states to 29 qubits (28 in
    complex128), every family, element type and kernel mode."""
    kind = rng.choice(["circuit", "circuit", "circuit", "remap", "reduce", "sample", "batch", "small", "runtime"])
    dtype = rng.choice(["c64", "c64", "c128"])
    if kind == "circuit":
        family = rng.choice(["rl", "rqc", "ccx", "vqe", "qft"])
        jit = "off" if dtype == "c128" else rng.choice(["eager", "off", "off"] if family in ("rl", "qft")
                                                       else ["coarse", "off", "off"] if family in ("rqc", "vqe")
                                                       else ["off"])
        n = rng.randint(10, 29 if dtype == "c64" else 28)
        depth = 1 if family == "qft" else max(2, int(round(math.exp(rng.uniform(math.log(2), math.log(24))))))
        if jit == "off" or dtype == "c128":
            depth = min(depth, max(2, 24 >> max(0, n - 26)))
        return dict(kind=kind, family=family, n=n, depth=depth, dtype=dtype, jit=jit)
    if kind in ("remap", "reduce"):
        return dict(kind=kind, n=rng.randint(10, 29), dtype=dtype)
    if kind == "sample":
        return dict(kind=kind, n=rng.randint(10, 29), dtype=dtype,
                    shots=int(round(math.exp(rng.uniform(math.log(1), math.log(16384))))))
    if kind == "runtime":
        return dict(kind=kind, family=rng.choice(["rl", "rqc", "ccx", "vqe", "qft"]), n=rng.randint(4, 20),
                    depth=rng.randint(2, 12), dtype=dtype, shots=rng.choice([1, 100, 1024, 4096]))
    lo = rng.randint(10, 12)
    hi = rng.randint(lo, 13 if kind == "small" else 20)
    count = int(round(math.exp(rng.uniform(math.log(1), math.log(128 if kind == "small" else 48)))))
    dlo = rng.randint(2, 20)
    return dict(kind=kind, count=count, n_min=lo, n_max=hi, depth_min=dlo, depth_max=dlo + rng.randint(0, 20))


# --------------------------------------------------------------------------------------------- circuits
def _gates(family, n, depth, seed):
    """The circuit's gates: [(name, qubits, params)]."""
    rng = np.random.default_rng([int(seed) & 0x7FFFFFFF, n, depth])
    out = []
    if family == "qft":
        for q in range(n):
            out.append(("ry", (q,), (float(rng.uniform(0, TWO_PI)),)))
        for j in reversed(range(n)):
            out.append(("h", (j,), ()))
            for k in reversed(range(j)):
                out.append(("cp", (k, j), (math.pi / 2 ** (j - k),)))
        return out
    for layer in range(depth):
        for q in range(n):
            a, b, c = (float(x) for x in rng.uniform(0, TWO_PI, 3))
            if family == "rqc":
                g = ("rx", "ry", "rz", "t", "h")[int(rng.integers(5))]
                out.append((g, (q,), (a,) if g[0] == "r" else ()))
            elif family == "vqe":
                out.append(("ry", (q,), (a,)))
                out.append(("rz", (q,), (b,)))
            else:
                out.append(("u", (q,), (a, b, c)))
        if family == "vqe":
            out += [("cx", (q, q + 1), ()) for q in range(n - 1)]
        else:
            two = "cx" if family == "rl" else "cz"
            out += [(two, (q, q + 1), ()) for q in range(layer % 2, n - 1, 2)]
        if family == "ccx":
            for _ in range(n // 4):
                out.append(("ccx", tuple(int(x) for x in rng.choice(n, 3, replace=False)), ()))
    return out


def _circuit(n, gates):
    qc = Circuit(n)
    for name, qs, ps in gates:
        qc.append(name, qs, ps)
    return qc


def _batch_members(case, seed):
    rng = np.random.default_rng([case["count"], case["n_min"], case["n_max"]])      # sizes belong to the case
    ns = rng.integers(case["n_min"], case["n_max"] + 1, case["count"])
    ds = rng.integers(case["depth_min"], case["depth_max"] + 1, case["count"])
    return [(int(n), _gates("ccx", int(n), int(d), int(seed) * 1000 + i)) for i, (n, d) in enumerate(zip(ns, ds))]


def _torch_dtype(case):
    return torch.complex128 if case.get("dtype") == "c128" else torch.complex64


def _random_state(case, seed):
    """A normalised random state (Gaussian amplitudes, as random circuits give)."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    real = torch.float64 if case["dtype"] == "c128" else torch.float32
    x = torch.empty(2 << case["n"], dtype=real, device="cuda")
    x.normal_(generator=g)
    x.mul_(1.0 / math.sqrt(2 << case["n"]))
    return torch.view_as_complex(x.view(-1, 2))


def _permutation(case, seed):
    return [int(x) for x in np.random.default_rng([int(seed) & 0x7FFFFFFF, 77]).permutation(case["n"])]


def _uniforms(case, seed):
    return np.random.default_rng([int(seed) & 0x7FFFFFFF, 78]).random(case["shots"])


# ------------------------------------------------------------------------------------------ prepare, run
def prepare(case, seed):
    kind = case["kind"]
    if kind == "circuit":
        n = case["n"]
        prog, fmap, _ = compile_circuit(_circuit(n, _gates(case["family"], n, case["depth"], seed)), n, min(K, n),
                                        dtype=case["dtype"])
        _engine.set_jit(case["jit"])
        segments = [payload for what, payload in prog if what == "segment"]
        if len(segments) != len(prog) or fmap != list(range(n)):
            raise RuntimeError("the circuit needs remaps")
        if case["jit"] != "off":
            for seg in segments:
                _engine.jit_prepare(seg, n)
        return dict(kind=kind, segments=segments, state=_engine.new_state(n, dtype=case["dtype"]))
    if kind == "remap":
        src = _random_state(case, seed)
        return dict(kind=kind, src=src, dst=torch.empty_like(src), perm=_permutation(case, seed))
    if kind == "reduce":
        return dict(kind=kind, state=_random_state(case, seed), scratch=_engine.new_scratch(case["n"]))
    if kind == "sample":
        return dict(kind=kind, state=_random_state(case, seed), scratch=_engine.new_scratch(case["n"]),
                    uniforms=torch.from_numpy(_uniforms(case, seed)).cuda())
    if kind == "runtime":
        _engine.set_jit("off")       # a request too small and too rare for kernels of its own
        rt = _runtime.SVRuntime(dtype=case["dtype"])
        qc = _circuit(case["n"], _gates(case["family"], case["n"], case["depth"], seed))
        return dict(kind=kind, rt=rt, qc=qc, shots=case["shots"], seed=int(seed))
    members = _batch_members(case, seed)
    _engine.set_jit("off")
    if kind == "batch":
        runner = _batch.BatchRunner(autotune=False)
        plan = runner.prepare([_circuit(n, g) for n, g in members], sample_fraction=0.05)
        runner.capture(plan)
        return dict(kind=kind, runner=runner, plan=plan)
    arena = torch.zeros(sum(1 << n for n, _ in members), dtype=torch.complex64, device="cuda")
    small, starts, at = _engine.SmallBatch(), [], 0
    for n, g in members:
        prog, _, _ = compile_circuit(_circuit(n, g), n, n)
        small.add(arena[at:at + (1 << n)], [payload for _, payload in prog])
        starts.append(at)
        at += 1 << n
    small.upload()
    return dict(kind=kind, small=small, arena=arena, starts=torch.tensor(starts, device="cuda"))


def run(state):
    kind = state["kind"]
    if kind == "circuit":
        st = state["state"]
        _engine.zero_state(st)
        for seg in state["segments"]:
            _engine.run_segment(st, seg)
        return st
    if kind == "remap":
        _engine.remap(state["src"], state["dst"], state["perm"])
        return state["dst"]
    if kind == "reduce":
        return _engine.reduce_f64(state["state"], scratch=state["scratch"])
    if kind == "sample":
        return _engine.sample_f64(state["state"], state["uniforms"], state["scratch"])
    if kind == "runtime":
        r = state["rt"].run(state["qc"], shots=state["shots"], seed=state["seed"])
        found = np.full((2, state["shots"]), -1, dtype=np.int64)        # (outcome, count), then -1
        found[:, :len(r["counts"])] = list(r["counts"].keys()), list(r["counts"].values())
        return dict(state=r["state"], counts=found)
    if kind == "batch":
        z, states = state["runner"].run(state["plan"])
        return dict(z=np.concatenate([np.concatenate([[norm], zq]) for norm, zq in z]),
                    states=[states[i] for i in sorted(states)])
    arena = state["arena"]
    arena.zero_()
    arena.index_fill_(0, state["starts"], 1.0)
    state["small"].launch()
    return arena


# ------------------------------------------------------------------------------------------------- work
_FLOPS = {"u": 14, "h": 14, "rx": 14, "ry": 14, "rz": 6, "t": 3, "cp": 1.5, "cx": 0, "cz": 0.25, "ccx": 0}


def _circuit_flops(n, gates):
    """Real operations on the amplitudes: a complex 2x2 product is 14 per amplitude, a phase 6 per amplitude it
    touches, an exchange none."""
    return float(sum(_FLOPS[name] for name, _, _ in gates)) * 2.0 ** n


def work(case):
    kind = case["kind"]
    if kind in ("batch", "small"):
        ns = [(case["n_min"] + case["n_max"]) / 2] * case["count"]
        spread = range(case["n_min"], case["n_max"] + 1)
        amps = case["count"] * sum(2.0 ** n for n in spread) / len(spread)
        depth = (case["depth_min"] + case["depth_max"]) / 2
        return dict(bytes=8 * amps, flops=amps * depth * 14 * sum(ns) / len(ns))
    n, amp = case["n"], 16 if case["dtype"] == "c128" else 8
    if kind in ("circuit", "runtime"):
        gates = _gates(case["family"], n, case["depth"], 1)
        return dict(bytes=amp * 2.0 ** n, flops=_circuit_flops(n, gates))
    if kind == "remap":
        return dict(bytes=2 * amp * 2.0 ** n, flops=0)
    return dict(bytes=amp * 2.0 ** n, flops=(3 + (n if kind == "reduce" else 0)) * 2.0 ** n)


# ------------------------------------------------------------------------------------------------ exact
def _matrix(name, params):
    if name == "u":
        th, ph, la = params
        c, s = math.cos(th / 2), math.sin(th / 2)
        return [[c, -np.exp(1j * la) * s], [np.exp(1j * ph) * s, np.exp(1j * (ph + la)) * c]]
    if name == "h":
        r = 1 / math.sqrt(2)
        return [[r, r], [r, -r]]
    if name == "t":
        return [[1, 0], [0, np.exp(0.25j * math.pi)]]
    c, s = math.cos(params[0] / 2), math.sin(params[0] / 2)
    if name == "rx":
        return [[c, -1j * s], [-1j * s, c]]
    if name == "ry":
        return [[c, -s], [s, c]]
    return [[complex(c, -s), 0], [0, complex(c, s)]]         # rz


def _simulate(n, gates, device):
    """The circuit's state from |0...0>, gate by gate in complex128."""
    v = torch.zeros(1 << n, dtype=torch.complex128, device=device)
    v[0] = 1.0

    def part(bits):
        """The amplitudes whose qubits have the values of `bits`, as a strided view."""
        shape, index, top = [], [], n
        for q in sorted(bits, reverse=True):
            shape += [1 << (top - 1 - q), 2]
            index += [slice(None), bits[q]]
            top = q
        return v.view(shape + [1 << top])[tuple(index)]

    for name, qs, ps in gates:
        if name == "cp":
            part({qs[0]: 1, qs[1]: 1}).mul_(complex(math.cos(ps[0]), math.sin(ps[0])))
        elif name == "cz":
            part({qs[0]: 1, qs[1]: 1}).neg_()
        elif name in ("cx", "ccx"):
            on = {q: 1 for q in qs[:-1]}
            a, b = part({**on, qs[-1]: 0}), part({**on, qs[-1]: 1})
            keep = a.clone()
            a.copy_(b)
            b.copy_(keep)
        else:
            m = _matrix(name, ps)
            a, b = part({qs[0]: 0}), part({qs[0]: 1})
            if m[0][1] == 0 and m[1][0] == 0:
                a.mul_(complex(m[0][0]))
                b.mul_(complex(m[1][1]))
            else:
                new = a * complex(m[0][0])
                new.add_(b, alpha=complex(m[0][1]))
                b.mul_(complex(m[1][1]))
                b.add_(a, alpha=complex(m[1][0]))
                a.copy_(new)
    return v


def _moments(v, n):
    """[sum |a|^2, <Z_0>, ..., <Z_{n-1}>] in float64."""
    p = v.real.double().square() + v.imag.double().square()
    out = [float(p.sum())]
    for q in range(n):
        w = p.view(-1, 2, 1 << q)
        out.append(float(w[:, 0].sum() - w[:, 1].sum()))
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "circuit":
        if case["n"] > 28:
            return None                                     # over about 20 seconds, and a state of its own size
        return _simulate(case["n"], _gates(case["family"], case["n"], case["depth"], seed), "cuda")
    if kind == "remap":
        x, perm = _random_state(case, seed), _permutation(case, seed)
        n = case["n"]
        # bit j of the result's index is bit perm[j] of the source's, moved a bit at a time
        order = list(range(n))                              # order[j]: source bit at index bit j of x
        for j in range(n):
            i = order.index(perm[j])
            if i != j:                                      # exchange index bits i and j
                w = x.view(-1, 2, 1 << (i - 1 - j), 2, 1 << j)
                keep = w[:, 0, :, 1].clone()
                w[:, 0, :, 1] = w[:, 1, :, 0]
                w[:, 1, :, 0] = keep
                order[i], order[j] = order[j], order[i]
        return x if case["dtype"] == "c128" or n > 28 else x.to(torch.complex128)
    if kind == "reduce":
        return torch.tensor(_moments(_random_state(case, seed), case["n"]), dtype=torch.float64)
    if kind == "sample":
        return None                                         # whole numbers: compared with each other
    if kind == "runtime":
        v = _simulate(case["n"], _gates(case["family"], case["n"], case["depth"], seed), "cuda")
        return dict(state=v, counts=None)
    members = _batch_members(case, seed)
    states = [_simulate(n, g, "cuda") for n, g in members]
    if kind == "small":
        return torch.cat(states)
    return dict(z=np.concatenate([_moments(v, n) for v, (n, _) in zip(states, members)]), states=None)
