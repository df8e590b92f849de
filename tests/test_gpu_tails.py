"""Diagonals carried by dense sweeps, in every form of the kernels that carry them: gate bits with and without
the three lowest state bits, tables, tables that act only where some bits are 1, sign flips, several diagonals
joined in one tail, up to six qubits; and amplitudes that are not finite."""
import numpy as np
import pytest

from rustatevec_b200 import Plan, PLAN_AS_GIVEN, PLAN_GREEDY, ENGINE_CUDA_CORE
from rustatevec_b200 import _lib as L
from rustatevec_b200 import gate as G
from rustatevec_b200.circuit import Circuit

from helpers import max_abs_diff, numpy_run

pytestmark = pytest.mark.gpu
UNIT = {"f64": 2.0 ** -53, "f32": 2.0 ** -24}
LOW = {"none": [], "0": [0], "1": [1], "2": [2], "01": [0, 1], "02": [0, 2], "12": [1, 2]}


def unitary(k, rng):
    z = rng.normal(size=(1 << k, 1 << k)) + 1j * rng.normal(size=(1 << k, 1 << k))
    return np.linalg.qr(z)[0]


def diagonal(m, rng, kind):
    """phases; phases that act only where the lowest bit is 1; signs."""
    d = rng.choice([-1.0, 1.0], size=1 << m) if kind == "signs" else np.exp(1j * rng.uniform(0, 2 * np.pi, size=1 << m))
    d = d.astype(np.complex128)
    d[-1] = -1.0 if kind == "signs" else d[-1]
    if kind == "control":
        d[::2] = 1.0
    return np.diag(d)


def random_state(n, rng, precision):
    psi = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    return (psi / np.linalg.norm(psi)).astype(np.complex128 if precision == "f64" else np.complex64)


def run(be, st, c, psi, planner):
    # (a width cap of 1 leaves the gates apart)
    plan = Plan(be, c, L.make_opts(planner, 1, ENGINE_CUDA_CORE))
    be.upload(st, psi.real, psi.imag)
    plan.run(st)
    return be.download(st).as_complex(), [s["carried"] for s in plan.sweeps()]


def gate_qubits(n, k, low, rng):
    return LOW[low] + sorted((3 + rng.choice(n - 3, size=k - len(LOW[low]), replace=False)).tolist())


# 11 qubits: one group a warp; 20, 21 and 22: several, and the complex64 kernel for k <= 4
@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("low", list(LOW))
@pytest.mark.parametrize("k,n", [(2, 11), (4, 11), (6, 11), (2, 21), (3, 22), (4, 22), (5, 20), (6, 20)])
def test_tail_of_every_kind_in_every_form(be64, be32, precision, low, k, n):
    """The two sweeps' own bits: a tail is applied in the order and the rounding of a sweep of its own."""
    be = be64 if precision == "f64" else be32
    rng = np.random.default_rng(1000 * k + 10 * n + list(LOW).index(low))
    qs = gate_qubits(n, k, low, rng)
    rest = [q for q in range(n) if q not in qs]
    psi = random_state(n, rng, precision)
    st = be.alloc(n)
    for kind, m in (("phases", 2), ("phases", 6), ("control", 3), ("signs", 2), ("signs", 5), ("signs", 6)):
        # the lowest free qubits (vector elements, lanes) and one far one, then some of the gate's own
        dq = ([rest[0], rest[-1]] + qs[:2] + rest[1:3])[:m]
        c = Circuit(n)
        c.push(G.DenseGate(k, unitary(k, rng)), qs)
        c.push(G.DenseGate(m, diagonal(m, rng, kind)), dq)
        want, given = run(be, st, c, psi, PLAN_AS_GIVEN)
        got, carried = run(be, st, c, psi, PLAN_GREEDY)
        assert given == [False, False] and carried == [False, True]
        assert np.array_equal(want, got), (kind, m, qs, dq)
    st.free()


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("low", ["none", "0", "2", "12"])
@pytest.mark.parametrize("k,n", [(2, 11), (3, 22), (4, 22), (5, 20)])
def test_joined_tails(be64, be32, precision, low, k, n):
    """Two and three diagonals that leave the gate's qubits join in one tail while they act on at most six qubits;
    one that would make seven stays a sweep. A joined table is a product of unit factors rounded once, so it and
    its multiplication, and the separate tables and multiplications, are each off by at most 4 u of an amplitude
    below 1: 8 u for one and two (three) diagonals 8 u (12 u) apart, on top of the dense sums' bound."""
    be = be64 if precision == "f64" else be32
    rng = np.random.default_rng(100 * k + n + list(LOW).index(low))
    qs = gate_qubits(n, k, low, rng)
    rest = [q for q in range(n) if q not in qs]
    psi = random_state(n, rng, precision)
    st = be.alloc(n)
    for kinds, dqs, want_carried in (
            (("phases", "phases"), ([rest[0], qs[0], rest[-1]], [rest[1], qs[1], rest[2]]), [True, True]),
            (("control", "signs", "phases"), ([rest[0], qs[0]], [rest[0], rest[3]], [qs[-1], rest[1]]), [True] * 3),
            (("signs", "signs"), ([rest[0], qs[0]], [rest[-1], qs[1], rest[0]]), [True, True]),
            (("signs", "signs"), ([rest[0], qs[0], rest[1]], [rest[-1], qs[1], rest[2]]), [True, True]),
            (("phases", "phases"), ([rest[0], qs[0], rest[1], rest[2]], [rest[-1], qs[1], rest[3]]), [True, False])):
        c = Circuit(n)
        c.push(G.DenseGate(k, unitary(k, rng)), qs)
        for kind, dq in zip(kinds, dqs):
            c.push(G.DenseGate(len(dq), diagonal(len(dq), rng, kind)), dq)
        want, _ = run(be, st, c, psi, PLAN_AS_GIVEN)
        got, carried = run(be, st, c, psi, PLAN_GREEDY)
        assert carried == [False] + want_carried
        assert max_abs_diff(want, got) <= 20 * UNIT[precision], (kinds, qs, dqs)
        if all(kind == "signs" for kind in kinds):  # signs are exact either way
            assert np.array_equal(want, got)
        if n < 20:
            assert max_abs_diff(numpy_run(c, psi), got) <= (2 ** (k + 1) + 24) * UNIT[precision]
    st.free()


def not_finite(psi):
    return set(np.flatnonzero(~(np.isfinite(psi.real) & np.isfinite(psi.imag))).tolist())


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("planner,n", [(PLAN_GREEDY, 11), (PLAN_GREEDY, 22), (L.PLAN_TILE, 16)])
def test_amplitudes_that_are_not_finite(be64, be32, precision, value, planner, n):
    """An infinite or undefined amplitude stays so (whether a sign flip or a skipped factor of 1 took the place of
    a product or not), reaches the amplitudes that a gate mixes it with, and no others."""
    be = be64 if precision == "f64" else be32
    rng = np.random.default_rng(n)
    at = 5 + (1 << (n - 2))
    c = Circuit(n)
    c.push(G.DenseGate(3, unitary(3, rng)), [1, 4, n - 1]) if planner == PLAN_GREEDY else c.h(4)
    if planner != PLAN_GREEDY:
        c.rx(9, 0.4)
    c.push(G.DenseGate(2, diagonal(2, rng, "signs")), [4, n - 2])
    c.push(G.DenseGate(2, diagonal(2, rng, "control")), [2, 4])
    c.cphase(1, n - 1, 0.7)
    c.push(G.DenseGate(2, diagonal(2, rng, "phases")), [4, 7])
    psi = random_state(n, rng, precision)
    clean = numpy_run(c, psi)
    st = be.alloc(n)
    for part in (1, 1j):
        bad = psi.copy()
        bad[at] = complex(value, 0.5) if part == 1 else complex(0.5, value)
        mixed = (1 << 1, 1 << 4, 1 << (n - 1)) if planner == PLAN_GREEDY else (1 << 4, 1 << 9)
        reach = {at}
        for b in mixed:
            reach |= {i ^ b for i in reach}
        be.upload(st, bad.real, bad.imag)
        Plan(be, c, L.make_opts(planner, 1, ENGINE_CUDA_CORE)).run(st)
        got = be.download(st)
        got = got.re.astype(np.float64) + 1j * np.where(np.isfinite(got.im), got.im, 0) + np.where(np.isfinite(got.im), 0, np.nan)
        assert not_finite(got) == reach
        ok = np.array([i for i in range(1 << n) if i not in reach]) if n < 20 else np.setdiff1d(np.arange(1 << n), list(reach))
        assert max_abs_diff(clean[ok], got[ok]) <= 100 * UNIT[precision]
    st.free()
