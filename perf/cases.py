"""The workloads this engine is timed on: what a user of the package runs, through its public calls.

A case is a dict of plain values; ``prepare`` builds the circuit and the device state a program has
in hand before the call, ``run`` makes the call, ``exact`` restates the result in FP64 with plain
torch, and ``work`` counts the bytes and operations the result cannot do without. ``call`` names the
way the engine is entered:

* ``plan``: a reusable ``Plan`` replayed on a resident state (parameter sweeps, repeated circuits).
  ``start`` is ``zero`` (``init_basis`` before every run) or ``gauss`` (a random normalised state
  that is transformed in place).
* ``execute``: one-shot ``B200Backend.execute`` of a host circuit, then its probabilities.
* ``apply``: the trait's gate-by-gate ``apply``.
* ``batch``: a reusable batch of uneven small circuits, ``<Z_0>`` of each.
* ``readout``: norm, several ``<Z_mask>`` and measurement shots of a resident state.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from rustatevec_b200 import B200Backend, Circuit, DenseGate, Plan
from rustatevec_b200 import PLAN_GREEDY, PLAN_LEARNED
from rustatevec_b200 import _lib as L
from rustatevec_b200 import tuning

PLANNERS = {"greedy": PLAN_GREEDY, "learned": PLAN_LEARNED}


def listed():
    return [
        # the inner loop of a variational run: a small layered ansatz replayed on the default
        # options, with one read-out; bound by launches, not by memory
        {"name": "ansatz12-f64-plan", "call": "plan", "circuit": "ansatz", "n": 12, "depth": 4, "dtype": "f64",
         "planner": "greedy", "k": 4, "start": "zero", "z": True},
        # a script that runs one circuit once and looks at its probabilities
        {"name": "random18-f32-execute", "call": "execute", "circuit": "random", "n": 18, "depth": 10, "dtype": "f32",
         "planner": "greedy", "k": 4},
        # the trait's default execute loop: one kernel per gate, unfused
        {"name": "layer24-f32-apply", "call": "apply", "circuit": "ansatz", "n": 24, "depth": 1, "dtype": "f32"},
        # greedy fusion at a wide cap on a dense complex128 state of an odd size
        {"name": "random25-f64-greedy5", "call": "plan", "circuit": "random", "n": 25, "depth": 6, "dtype": "f64",
         "planner": "greedy", "k": 5, "start": "gauss", "z": False},
        # random brickwork on the reference's own method (fuse at its default width) in both precisions
        {"name": "brick28-f32-greedy4", "call": "plan", "circuit": "brickwork", "n": 28, "depth": 6, "dtype": "f32",
         "planner": "greedy", "k": 4, "start": "zero", "z": False},
        {"name": "brick27-f64-greedy4", "call": "plan", "circuit": "brickwork", "n": 27, "depth": 5, "dtype": "f64",
         "planner": "greedy", "k": 4, "start": "zero", "z": False},
        # the headline: 30-qubit depth-20 brickwork, tensor cores and the learned planner
        {"name": "brick30-f32-learned", "call": "plan", "circuit": "brickwork", "n": 30, "depth": 20, "dtype": "f32",
         "planner": "learned", "k": 6, "start": "zero", "z": False},
        # the same method on a state that is not much larger than L2, odd qubit count and depth
        {"name": "brick23-f32-learned", "call": "plan", "circuit": "brickwork", "n": 23, "depth": 7, "dtype": "f32",
         "planner": "learned", "k": 6, "start": "zero", "z": False},
        # QFT of a random state
        {"name": "qft30-f32-learned", "call": "plan", "circuit": "qft", "n": 30, "depth": 1, "dtype": "f32",
         "planner": "learned", "k": 6, "start": "gauss", "z": False},
        # QAOA MaxCut on a random 3-regular graph, complex128
        {"name": "qaoa29-f64-learned", "call": "plan", "circuit": "qaoa", "n": 29, "depth": 2, "dtype": "f64",
         "planner": "learned", "k": 6, "start": "zero", "z": False},
        # uneven small circuits in one persistent kernel
        {"name": "batch384-f32", "call": "batch", "circuit": "ansatz", "n": 20, "depth": 12, "count": 384,
         "dtype": "f32"},
        # what is asked of a final state
        {"name": "readout27-f64", "call": "readout", "n": 27, "shots": 20000, "masks": 4, "dtype": "f64"},
    ]


def draw(rng):
    def size(lo, hi):
        return rng.randint(lo, hi)

    dtype = rng.choice(["f32", "f64"])
    wide = dtype == "f64"
    what = rng.choice(["small", "execute", "apply", "greedy", "greedy", "learned", "learned", "qft", "qaoa", "batch",
                       "readout"])
    if what == "small":
        return {"call": "plan", "circuit": rng.choice(["ansatz", "random"]), "n": size(8, 16), "depth": size(2, 8),
                "dtype": dtype, "planner": "greedy", "k": size(2, 5), "start": "zero", "z": True}
    if what == "execute":
        return {"call": "execute", "circuit": rng.choice(["ansatz", "random", "brickwork"]), "n": size(10, 21),
                "depth": size(3, 12), "dtype": dtype, "planner": "greedy", "k": 4}
    if what == "apply":
        return {"call": "apply", "circuit": rng.choice(["ansatz", "random", "brickwork"]), "n": size(12, 26),
                "depth": size(1, 3), "dtype": dtype}
    if what == "greedy":
        return {"call": "plan", "circuit": rng.choice(["random", "brickwork", "ansatz"]),
                "n": size(18, 26 if wide else 28), "depth": size(2, 6), "dtype": dtype, "planner": "greedy",
                "k": size(2, 5 if wide else 6), "start": rng.choice(["zero", "gauss"]), "z": False}
    if what == "learned":
        return {"call": "plan", "circuit": "brickwork", "n": size(18, 30), "depth": size(3, 20), "dtype": "f32",
                "planner": "learned", "k": 6, "start": "zero", "z": False}
    if what == "qft":
        return {"call": "plan", "circuit": "qft", "n": size(17, 28 if wide else 30), "depth": 1, "dtype": dtype,
                "planner": "learned", "k": 6, "start": "gauss", "z": False}
    if what == "qaoa":
        return {"call": "plan", "circuit": "qaoa", "n": size(18, 28), "depth": size(1, 4), "dtype": dtype,
                "planner": "learned", "k": 6, "start": "zero", "z": False}
    if what == "batch":
        return {"call": "batch", "circuit": "ansatz", "n": size(14, 20), "depth": size(4, 12),
                "count": int(round(math.exp(rng.uniform(math.log(16), math.log(384))))), "dtype": dtype}
    return {"call": "readout", "n": size(14, 27 if wide else 28), "shots": size(1000, 100000), "masks": size(1, 6),
            "dtype": dtype}


# ------------------------------------------------------------------ circuits, as lists of (matrix, qubits)
_R2 = math.sqrt(0.5)
_H = np.array([[_R2, _R2], [_R2, -_R2]], dtype=np.complex128)
_FIXED = [_H, np.array([[0, 1], [1, 0]], dtype=np.complex128), np.array([[0, -1j], [1j, 0]]),
          np.diag([1, -1]).astype(np.complex128), np.diag([1, 1j]), np.diag([1, complex(_R2, _R2)]),
          0.5 * np.array([[1 + 1j, 1 - 1j], [1 - 1j, 1 + 1j]])]
# two-qubit matrices: row/column index bit j is qubit j of the pair, the control first
_CX = np.eye(4, dtype=np.complex128)[[0, 3, 2, 1]]
_CZ = np.diag([1, 1, 1, -1]).astype(np.complex128)
_SWAP = np.eye(4, dtype=np.complex128)[[0, 2, 1, 3]]


def _rx(t):
    c, s = math.cos(t / 2), math.sin(t / 2)
    return np.array([[c, -1j * s], [-1j * s, c]])


def _ry(t):
    c, s = math.cos(t / 2), math.sin(t / 2)
    return np.array([[c, -s], [s, c]], dtype=np.complex128)


def _rz(t):
    return np.diag([complex(math.cos(t / 2), -math.sin(t / 2)), complex(math.cos(t / 2), math.sin(t / 2))])


def _cphase(t):
    return np.diag([1, 1, 1, complex(math.cos(t), math.sin(t))])


def _rzz(t):
    a, b = complex(math.cos(t / 2), -math.sin(t / 2)), complex(math.cos(t / 2), math.sin(t / 2))
    return np.diag([a, b, b, a])


def _su2(g):
    a, b, c, d = (lambda v: v / np.linalg.norm(v))(g.standard_normal(4))
    return np.array([[complex(a, b), complex(c, d)], [complex(-c, d), complex(a, -b)]])


def _ansatz(n, depth, g):
    ops = []
    for _ in range(depth):
        for q in range(n):
            ops += [(_rz(g.uniform(0, 2 * math.pi)), (q,)), (_ry(g.uniform(0, 2 * math.pi)), (q,))]
        ops += [(_CX, (i, i + 1)) for i in range(n - 1)]
    return ops


def _random(n, depth, g):
    """``depth * n`` gates over the one- and two-qubit gate set."""
    ops = []
    for _ in range(depth * n):
        q, kind, t = int(g.integers(n)), int(g.integers(15)), g.uniform(0, 2 * math.pi)
        if kind < 7:
            ops.append((_FIXED[kind], (q,)))
        elif kind < 11:
            ops.append(((_rx(t), _ry(t), _rz(t), np.diag([1, complex(math.cos(t), math.sin(t))]))[kind - 7], (q,)))
        else:
            q2 = (q + 1 + int(g.integers(n - 1))) % n
            ops.append(((_CX, _CZ, _SWAP, _rzz(t))[kind - 11], (q, q2)))
    return ops


def _brickwork(n, depth, g):
    ops = []
    for layer in range(depth):
        ops += [(_su2(g), (q,)) for q in range(n)]
        ops += [(_CZ, (i, i + 1)) for i in range(layer % 2, n - 1, 2)]
    return ops


def _qft(n, depth, g):
    ops = []
    for j in range(n):
        ops.append((_H, (j,)))
        ops += [(_cphase(math.pi / 2 ** (k - j)), (k, j)) for k in range(j + 1, n)]
    return ops + [(_SWAP, (j, n - 1 - j)) for j in range(n // 2)]


def _qaoa(n, depth, g):
    """MaxCut on a random 3-regular graph (odd ``n``: node 0 has degree 4)."""
    while True:
        stubs = np.array([v for v in range(n) for _ in range(3 + (v == 0 and n % 2))])
        pairs = g.permutation(stubs).reshape(-1, 2)
        edges = {(int(min(p)), int(max(p))) for p in pairs}
        if len(edges) == len(pairs) and all(a != b for a, b in edges):
            break
    ops = [(_H, (q,)) for q in range(n)]
    for _ in range(depth):
        gamma, beta = g.uniform(0, math.pi), g.uniform(0, math.pi / 2)
        ops += [(_rzz(-gamma), e) for e in sorted(edges)] + [(_rx(2 * beta), (q,)) for q in range(n)]
    return ops


_CIRCUITS = {"ansatz": _ansatz, "random": _random, "brickwork": _brickwork, "qft": _qft, "qaoa": _qaoa}


def _ops(case, seed):
    return _CIRCUITS[case["circuit"]](case["n"], case["depth"], np.random.default_rng(seed))


def _batch_ops(case, seed):
    """``count`` circuits of 10..n qubits and 4..depth layers. The sizes are the case's own (a seed of their
    own), the angles the seed's: one program's circuits keep their shapes while the parameters change."""
    shape, g = np.random.default_rng(case["count"]), np.random.default_rng(seed)
    out = []
    for _ in range(case["count"]):
        n, d = int(shape.integers(10, case["n"] + 1)), int(shape.integers(4, case["depth"] + 1))
        out.append((n, _ansatz(n, d, g)))
    return out


def _circuit(n, ops):
    c = Circuit(n)
    for m, q in ops:
        c.push(DenseGate(len(q), m), q)
    return c


# ------------------------------------------------------------------ the engine's side
_BACKENDS = {}


def _backend(dtype):
    """One backend (context and stream) per precision, as a program keeps it, with the cost model installed."""
    if dtype not in _BACKENDS:
        tuning.load()
        _BACKENDS[dtype] = B200Backend(0, precision=dtype)
    return _BACKENDS[dtype]


class _Buffer:
    """A state's device array for torch; keeps the state alive."""

    def __init__(self, state, ptr, wide):
        self.state = state
        self.__cuda_array_interface__ = {"shape": (1 << state.n,), "typestr": "<f8" if wide else "<f4",
                                         "data": (ptr, False), "version": 3}


def _views(state, dtype):
    re, im = C.c_void_p(), C.c_void_p()
    L.check(L.lib().qsvb_state_info(state.handle, None, None, C.byref(re), C.byref(im)))
    return {"re": torch.as_tensor(_Buffer(state, re.value, dtype == "f64"), device="cuda"),
            "im": torch.as_tensor(_Buffer(state, im.value, dtype == "f64"), device="cuda")}


def _gauss(n, seed, dtype):
    """A random state: i.i.d. complex Gaussian amplitudes, normalised, in the state's precision."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    t = torch.float64 if dtype == "f64" else torch.float32
    re = torch.randn(1 << n, generator=g, device="cuda", dtype=t)
    im = torch.randn(1 << n, generator=g, device="cuda", dtype=t)
    s = 1.0 / math.sqrt(2.0 * (1 << n))
    return re.mul_(s), im.mul_(s)


def _masks(case, seed):
    g = np.random.default_rng(seed)
    return [int(g.integers(1, 1 << case["n"])) for _ in range(case["masks"])]


class _Batch:
    def __init__(self, be, circuits):
        self.be, self.packed = be, L.PackedBatch(circuits)
        self.handle = C.c_void_p()
        L.check(L.lib().qsvb_batch_create(be.ctx, self.packed.ptr(), self.packed.count, be.dtype, 0, 0,
                                          C.byref(self.handle)))

    def run(self):
        z0 = np.empty(self.packed.count)
        L.check(L.lib().qsvb_batch_run(self.be.ctx, self.handle, z0.ctypes.data_as(C.POINTER(C.c_double)), None, None,
                                       None))
        return z0

    def __del__(self):
        L.lib().qsvb_batch_free(self.be.ctx, self.handle)


def prepare(case, seed):
    be = _backend(case["dtype"])
    s = {"case": case, "be": be}
    if case["call"] == "batch":
        s["batch"] = _Batch(be, [_circuit(n, ops) for n, ops in _batch_ops(case, seed)])
        return s
    n = case["n"]
    if case["call"] == "execute":
        be.opts = L.make_opts(PLANNERS[case["planner"]], case["k"])
        s["circuit"] = _circuit(n, _ops(case, seed))
        return s
    state = s["state"] = be.alloc(n)
    s["out"] = _views(state, case["dtype"])
    be.init_basis(state, 0)
    be.synchronize()
    if case["call"] == "readout" or case.get("start") == "gauss":
        re, im = _gauss(n, seed, case["dtype"])
        s["out"]["re"].copy_(re)
        s["out"]["im"].copy_(im)
        torch.cuda.synchronize()
    if case["call"] == "readout":
        s["masks"], s["seed"] = _masks(case, seed), seed
    elif case["call"] == "apply":
        s["gates"] = [(DenseGate(len(q), m), q) for m, q in _ops(case, seed)]
    else:
        s["plan"] = Plan(be, _circuit(n, _ops(case, seed)), L.make_opts(PLANNERS[case["planner"]], case["k"]))
    return s


def run(s):
    case, be = s["case"], s["be"]
    call = case["call"]
    if call == "plan":
        if case["start"] == "zero":
            be.init_basis(s["state"], 0)
        s["plan"].run(s["state"])
        if case["z"]:
            return dict(s["out"], z=be.expectation_z(s["state"], 1))
        return s["out"]
    if call == "apply":
        be.init_basis(s["state"], 0)
        for gate, qubits in s["gates"]:
            be.apply(s["state"], gate, qubits)
        return s["out"]
    if call == "execute":
        return {"p": be.probabilities(be.execute(s["circuit"]))}
    if call == "batch":
        return {"z": s["batch"].run()}
    state = s["state"]
    return {"norm": be.norm_sqr(state), "z": [be.expectation_z(state, m) for m in s["masks"]],
            "shots": be.sample_device(state, case["shots"], s["seed"]).astype(np.int64)}


# ------------------------------------------------------------------ bytes and operations
def _flops(n, ops):
    total = 0.0
    for m, q in ops:
        d = len(m)
        if np.count_nonzero(m - np.diag(np.diag(m))) == 0:  # a complex product where the entry is not 1
            total += 6.0 * np.count_nonzero(np.diag(m) != 1) / d
        elif np.count_nonzero(m) > d:  # (permutations move amplitudes and compute nothing)
            total += 14.0
    return float(total * (1 << n))


def work(case):
    size = 8 if case["dtype"] == "f64" else 4
    if case["call"] == "batch":
        return {"bytes": 8.0 * case["count"], "flops": sum(_flops(n, ops) for n, ops in _batch_ops(case, 0))}
    state = 2.0 * size * (1 << case["n"])
    if case["call"] == "readout":
        return {"bytes": state + 8.0 * case["shots"], "flops": 4.0 * (1 << case["n"])}
    moved = state
    if case["call"] == "execute":
        moved = state / 2  # the probabilities
    elif case.get("start") == "gauss":
        moved = 2 * state
    return {"bytes": moved, "flops": _flops(case["n"], _ops(case, 0))}


# ------------------------------------------------------------------ FP64 values in plain torch
def _windows(ops, k):
    """Groups of gates on at most k qubits, each group free of the qubits of the gates it goes before."""
    while ops:
        qs, blocked, take, rest = set(), set(), [], []
        for op in ops:
            s = set(op[1])
            if s & blocked or len(qs | s) > k:
                blocked |= s
                rest.append(op)
            else:
                qs |= s
                take.append(op)
        yield sorted(qs), take
        ops = rest


def _product(qs, ops):
    """The matrix of ``ops`` in order on the qubits ``qs`` (index bit j is qs[j])."""
    k = len(qs)
    u = np.eye(1 << k, dtype=np.complex128).reshape([2] * k + [-1])  # axis k-1-j is bit j
    for m, q in ops:
        axes = [k - 1 - qs.index(x) for x in reversed(q)]
        u = np.tensordot(m.reshape([2] * (2 * len(q))), u, axes=(list(range(len(q), 2 * len(q))), axes))
        u = np.moveaxis(u, list(range(len(q))), axes)
    return u.reshape(1 << k, 1 << k)


def _simulate(n, ops, psi=None):
    if psi is None:
        psi = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
        psi[0] = 1.0
    for qs, group in _windows(ops, min(6, n)):
        u = torch.from_numpy(np.ascontiguousarray(_product(qs, group))).cuda()
        shape, top, where = [], n, []
        for q in reversed(qs):  # the highest qubit first
            shape += [1 << (top - 1 - q), 2]
            where.append(len(shape) - 1)
            top = q
        shape.append(1 << top)
        order = where + [d for d in range(len(shape)) if d not in where]
        view = psi.view(shape).permute(order)
        new = u @ view.reshape(1 << len(qs), -1)
        view.copy_(new.view([shape[d] for d in order]))
        del new
    return psi


def exact(case, seed):
    if case["call"] == "batch":
        z = []
        for n, ops in _batch_ops(case, seed):
            p = torch.view_as_real(_simulate(n, ops)).square().sum(1).view(-1, 2).sum(0)
            z.append(p[0] - p[1])
        return {"z": torch.stack(z)}
    n = case["n"]
    start = None
    if case["call"] == "readout" or case.get("start") == "gauss":
        start = torch.complex(*(x.double() for x in _gauss(n, seed, case["dtype"])))
    if case["call"] == "readout":
        p = torch.view_as_real(start).square().sum(1)
        i = torch.arange(1 << n, device="cuda")
        z = []
        for m in _masks(case, seed):
            odd = i & m
            for shift in (16, 8, 4, 2, 1):
                odd = odd ^ (odd >> shift)
            z.append(float((p * (1 - 2 * (odd & 1))).sum()))
        return {"norm": float(p.sum()), "z": z, "shots": None}
    psi = _simulate(n, _ops(case, seed), start)
    if case["call"] == "execute":
        return {"p": torch.view_as_real(psi).square().sum(1)}
    out = {"re": psi.real, "im": psi.imag}
    if case.get("z"):
        p = torch.view_as_real(psi).square().sum(1).view(-1, 2).sum(0)
        out["z"] = float(p[0] - p[1])
    return out
