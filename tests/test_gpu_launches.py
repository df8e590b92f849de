"""How sweeps of different kernels follow one another on the stream."""
import numpy as np
import pytest

from rustatevec_b200 import B200Backend, Circuit, DenseGate, Plan, PLAN_AS_GIVEN, PLAN_GREEDY
from rustatevec_b200 import ENGINE_CUDA_CORE, ENGINE_TENSOR_CORE
from rustatevec_b200 import _lib as L

pytestmark = pytest.mark.gpu


def unitary(k, rng):
    z = rng.normal(size=(1 << k, 1 << k)) + 1j * rng.normal(size=(1 << k, 1 << k))
    return np.linalg.qr(z)[0]


@pytest.mark.parametrize("precision,n,first,second", [("f32", 28, "dense_tc", "dense"), ("f64", 27, "diag", "dense")])
def test_two_sweeps_in_turn_cost_their_own_time(built, precision, n, first, second):
    """Kernels that need different splits of an SM's memory, in turn: k_tc_dense and k_dense_cols, k_diag and the
    four-qubit k_dense_mma. Launched programmatically the pairs took 17 % and 28 % longer than by themselves
    (blocks started early found SMs split for the other); ordinary launches add about 4 us each, 1 % at most. The
    bound lies between: 8 %."""
    import torch
    rng = np.random.default_rng(0)
    be = B200Backend(0, precision=precision)
    stream = torch.cuda.ExternalStream(be.stream())
    st = be.alloc(n)
    be.init_basis(st, 0)
    gates = {"dense": (DenseGate(4, unitary(4, rng)), list(range(10, 14)), PLAN_AS_GIVEN, ENGINE_CUDA_CORE),
             "dense_tc": (DenseGate(6, unitary(6, rng)), list(range(10, 16)), PLAN_GREEDY, ENGINE_TENSOR_CORE),
             "diag": (DenseGate(2, np.diag([1, 1, 1, -1])), [9, n - 1], PLAN_AS_GIVEN, ENGINE_CUDA_CORE)}
    plans = {}
    for name in (first, second):
        gate, qs, planner, engine = gates[name]
        c = Circuit(n)
        c.push(gate, qs)
        plans[name] = Plan(be, c, L.make_opts(planner, 6, engine, use_graph=False))
        assert plans[name].stats()["by_kind"] == {name: 1}

    def seconds(*names):
        best = float("inf")
        for _ in range(5):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record(stream)
            for _ in range(8):
                for name in names:
                    plans[name].run(st)
            e1.record(stream)
            e1.synchronize()
            best = min(best, e0.elapsed_time(e1))
        return best

    seconds(first, second)
    alone = seconds(first) + seconds(second)
    assert seconds(first, second) <= 1.08 * alone
    st.free()
    be.close()
