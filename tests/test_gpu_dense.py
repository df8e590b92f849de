"""Dense CUDA-core sweeps at every size class of their launch rule: states with fewer columns than one
matrix-instruction tile, one column group a warp, several groups a warp, and gate bits low, high,
spread and in descending order.

Tolerance: each output is a sum of 2^(k+1) products whose absolute values add up to at most
|row| |x| <= 1 (unitary row, normalised state), so with unit roundoff u the sum is off by at most
2^(k+1) u, plus u for the rounding of the matrix and of the input each and one for the store."""
import numpy as np
import pytest

from rustatevec_b200 import Plan, PLAN_AS_GIVEN, PLAN_GREEDY, ENGINE_CUDA_CORE
from rustatevec_b200 import _lib as L
from rustatevec_b200 import gate as G
from rustatevec_b200.circuit import Circuit

from helpers import max_abs_diff, numpy_run

pytestmark = pytest.mark.gpu
UNIT = {"f64": 2.0 ** -53, "f32": 2.0 ** -24}


def unitary(k, rng):
    z = rng.normal(size=(1 << k, 1 << k)) + 1j * rng.normal(size=(1 << k, 1 << k))
    return np.linalg.qr(z)[0]


def placements(n, k, rng):
    spread = sorted(rng.choice(n, size=k, replace=False).tolist())
    out = [list(range(k)), list(range(n - k, n)), spread, spread[::-1]]
    if n >= k + 3:  # the bits around a 16-byte vector, a 32-byte sector and a warp's row
        out += [[0] + list(range(n - k + 1, n)), [1] + list(range(n - k + 1, n)), [2] + list(range(n - k + 1, n)),
                list(range(1, k + 1)), list(range(2, k + 2)), [0, 2] + list(range(n - k + 2, n)),
                [1, 2] + list(range(n - k + 2, n)), [0, 1] + list(range(n - k + 2, n))]
    return out


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("k", [2, 3, 4, 5, 6])
@pytest.mark.parametrize("n", [6, 8, 9, 10, 11, 13, 17, 21])
def test_dense_sweep_every_size_class(be64, be32, precision, k, n):
    be = be64 if precision == "f64" else be32
    rng = np.random.default_rng(100 * k + n)
    qsets = placements(n, k, rng)
    if n >= 17:  # the large states: one launch class, every placement once across the sizes
        qsets = qsets[:3] + [qsets[3 + n % (len(qsets) - 3)]]
    st = be.alloc(n)
    for qs in qsets:
        if len(set(qs)) < k:
            continue
        psi = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
        psi = (psi / np.linalg.norm(psi)).astype(np.complex128 if precision == "f64" else np.complex64)
        c = Circuit(n)
        c.push(G.DenseGate(k, unitary(k, rng)), qs)
        plan = Plan(be, c, L.make_opts(PLAN_AS_GIVEN, k, ENGINE_CUDA_CORE))
        assert plan.stats()["by_kind"] == {"dense": 1}
        be.upload(st, psi.real, psi.imag)
        plan.run(st)
        err = max_abs_diff(numpy_run(c, psi), be.download(st).as_complex())
        assert err <= (2 ** (k + 1) + 4) * UNIT[precision], (qs, err)
    st.free()


def diagonal(m, rng, controls=0, signs=False):
    """A random diagonal (of signs, or of phases) on m qubits that acts only where the lowest `controls`
    bits are 1."""
    d = rng.choice([-1.0, 1.0], size=1 << m) if signs else np.exp(1j * rng.uniform(0, 2 * np.pi, size=1 << m))
    d = d.astype(np.complex128)
    d[-1] = -1.0 if signs else d[-1]
    d[(np.arange(1 << m) & ((1 << controls) - 1)) != (1 << controls) - 1] = 1.0
    return np.diag(d)


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("k,n", [(2, 5), (2, 11), (3, 11), (4, 11), (5, 11), (6, 11), (2, 21), (3, 22), (4, 22), (5, 20)])
def test_diagonal_carried_by_a_dense_sweep(be64, be32, precision, k, n):
    """A dense sweep that multiplies by the following diagonal gives the two sweeps' own bits (to rounding
    where the diagonal went into the matrix); with a second diagonal moved back past a sweep on other
    qubits, the circuit is right to rounding."""
    be = be64 if precision == "f64" else be32
    rng = np.random.default_rng(10 * k + n)
    st = be.alloc(n)
    qsets = placements(n, k, rng)
    for i, qs in enumerate(qsets if n < 17 else qsets[::4]):
        if len(set(qs)) < k:
            continue
        m = 1 + (i + k) % 5
        psi = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
        psi = (psi / np.linalg.norm(psi)).astype(np.complex128 if precision == "f64" else np.complex64)
        c = Circuit(n)
        c.push(G.DenseGate(k, unitary(k, rng)), qs)
        inside = i % 3 == 2  # on the dense gate's own qubits: multiplied into its matrix
        dq = rng.permutation(qs)[:m].tolist() if inside else rng.choice(n, size=m, replace=False).tolist()
        m = len(dq)
        inside = set(dq) <= set(qs)
        c.push(G.DenseGate(m, diagonal(m, rng, controls=i % 2, signs=i % 4 >= 2)), dq)
        got = []
        for planner in (PLAN_AS_GIVEN, PLAN_GREEDY):  # (a width cap of 1 leaves the gates apart)
            plan = Plan(be, c, L.make_opts(planner, 1, ENGINE_CUDA_CORE))
            assert plan.stats()["by_kind"] == {"dense": 1, "diag": 1}
            be.upload(st, psi.real, psi.imag)
            plan.run(st)
            got.append(be.download(st).as_complex())
        if inside:
            assert max_abs_diff(got[0], got[1]) <= 2 * (2 ** (k + 1) + 8) * UNIT[precision], (qs, dq)
        else:
            assert np.array_equal(got[0], got[1]), (qs, dq)
        rest = [q for q in range(n) if q not in qs][:2]
        c.push(G.DenseGate(2, unitary(2, rng)), rest)
        c.push(G.DenseGate(2, diagonal(2, rng)), [qs[0], qs[-1]])
        be.upload(st, psi.real, psi.imag)
        Plan(be, c, L.make_opts(PLAN_GREEDY, 1, ENGINE_CUDA_CORE)).run(st)
        err = max_abs_diff(numpy_run(c, psi), be.download(st).as_complex())
        assert err <= (2 ** (k + 1) + 2 ** 3 + 20) * UNIT[precision], (qs, m, err)
    st.free()


@pytest.mark.parametrize("planner", [L.PLAN_GREEDY, L.PLAN_WINDOW, L.PLAN_LEARNED, PLAN_AS_GIVEN])
def test_dry_run_reports_what_the_plan_reports(be32, planner):
    import ctypes as C
    from rustatevec_b200.circuits import brickwork
    c, opts = brickwork(22, 4, 1), L.make_opts(planner, 4, ENGINE_CUDA_CORE)
    pc, st = L.PackedCircuit(c), L.PlanStats()
    L.check(L.lib().qsvb_plan_dry_run(pc.ref(), be32.dtype, C.byref(opts), C.byref(st)))
    assert Plan(be32, c, opts).stats() == st.to_dict()


def test_profile_runs_what_the_plan_runs(be64):
    """A carried diagonal is marked, takes no time of its own and is part of its dense sweep's: profiling launches
    every sweep twice (reps = 1 and a warm-up), which for one launched sweep is two runs of the plan."""
    rng = np.random.default_rng(2)
    n = 11
    c = Circuit(n)
    c.push(G.DenseGate(3, unitary(3, rng)), [2, 5, 6])
    c.push(G.DenseGate(2, diagonal(2, rng)), [5, 9])
    psi = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    apart = L.make_opts(PLAN_GREEDY, 1)
    apart.diagonals_apart = 1
    st = be64.alloc(n)
    got = []
    for opts in (L.make_opts(PLAN_GREEDY, 1), apart):
        plan = Plan(be64, c, opts)
        for step in (lambda: plan.profile(st, 1), lambda: (plan.run(st), plan.run(st))):
            be64.upload(st, psi.real, psi.imag)
            secs = step()
            got.append((be64.download(st).as_complex(), secs, [s["carried"] for s in plan.sweeps()], plan.launches()))
    (prof, secs, carried, launches), (runs, *_), (prof_apart, secs_apart, carried_apart, two), (runs_apart, *_) = got
    assert carried == [False, True] and launches == 1 and secs[0] > 0 and secs[1] == 0
    assert carried_apart == [False, False] and two == 2 and (secs_apart > 0).all()
    assert np.array_equal(prof, runs) and np.array_equal(runs, runs_apart)
    assert not np.array_equal(prof_apart, runs_apart)  # (there the dense sweep ran twice, then the diagonal)
    st.free()
