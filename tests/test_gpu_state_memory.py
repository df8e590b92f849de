"""Memory of freed states: what freeing leaves alone, and what the next state finds in it."""
import ctypes as C
import threading

import numpy as np
import pytest

from rustatevec_b200 import B200Backend, Circuit, DenseGate, Plan
from rustatevec_b200 import _lib as L
from rustatevec_b200.circuits import random_circuit

import oracle
from helpers import max_abs_diff, numpy_run

pytestmark = pytest.mark.gpu


def pointers(state):
    re, im = C.c_void_p(), C.c_void_p()
    L.check(L.lib().qsvb_state_info(state.handle, None, None, C.byref(re), C.byref(im)))
    return re.value, im.value


@pytest.mark.parametrize("exposed", [False, True])
def test_free_leaves_another_threads_capture_alone(be32, exposed):
    """One thread records a graph on its own stream (thread-local capture, which allows other threads any
    call) while another frees a state. A device-wide wait would invalidate the capture."""
    import torch
    state = be32.alloc(12)
    be32.init_basis(state, 0)
    if exposed:
        pointers(state)
    x = torch.zeros(1000, device="cuda")
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        graph.capture_begin(capture_error_mode="thread_local")
        x.add_(1)
        worker = threading.Thread(target=state.free)
        worker.start()
        worker.join()
        x.add_(1)
        graph.capture_end()
    assert state.handle is None
    graph.replay()
    torch.cuda.synchronize()
    assert bool((x == 2).all())


def test_reused_memory_shows_nothing_of_its_last_state(built):
    """One-shot circuits on states of changing sizes, whose memory held random amplitudes before."""
    for precision, tol in (("f64", 1e-12), ("f32", 1e-5)):
        be = B200Backend(0, precision=precision)
        for i, n in enumerate((13, 9, 13, 13, 14, 9)):
            for _ in range(2):
                junk = be.alloc(n)
                be.init_gaussian(junk, i)
                junk.free()
            c = random_circuit(n, 60, i)
            state = be.execute(c)
            re, im = oracle.run(c, oracle.REF, oracle.F64)
            assert max_abs_diff(re + 1j * im, be.download(state).as_complex()) <= tol
            state.free()
        be.close()


def test_two_states_never_share_memory(built):
    """Freed through another context, or with their pointers handed out, buffers are not handed on; live states
    of one size always differ."""
    a, b = B200Backend(0, precision="f32"), B200Backend(0, precision="f32")
    live = []
    for i in range(12):
        s = a.alloc(11)
        a.init_basis(s, i)
        if i % 3 == 0:
            b.norm_sqr(s)
        live.append(s)
        if i % 4 == 3:
            live.pop(0).free()
    spans = sorted(p for s in live for p in pointers(s))
    assert all(q - p >= 4 << 11 for p, q in zip(spans, spans[1:]))
    kept = [i for i in range(12) if i not in (0, 1, 2)]
    for i, s in zip(kept, live):
        psi = a.download(s).as_complex()
        assert psi[i] == 1 and np.count_nonzero(psi) == 1
        s.free()
    a.close()
    b.close()


def device_free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_kept_memory_counts_whole_states(built):
    """At most 64 MB of freed states are kept, both components of a state or neither, and the most recent sizes."""
    mb = 1 << 20
    be = B200Backend(0, precision="f32")
    before = device_free()
    be.alloc(24).free()  # two components of 64 MB
    assert device_free() == before
    held = [be.alloc(22) for _ in range(2)]  # 32 MB each
    for s in held:
        s.free()
    assert before - device_free() == 64 * mb
    be.alloc(21).free()  # 16 MB: the older of the two makes room
    assert before - device_free() == 48 * mb
    again = be.alloc(21)
    assert before - device_free() == 48 * mb  # found again
    again.free()
    be.alloc(23).free()  # 64 MB: everything else makes room
    assert before - device_free() == 64 * mb
    again = be.alloc(23)
    assert before - device_free() == 64 * mb
    again.free()
    be.close()


def test_kept_memory_is_given_back_before_an_allocation_fails(built):
    """With the device nearly full, a batch and a state that fit only without the kept states and the sampler's
    kept scratch. (The kernels run once before, so that loading them needs no memory then.)"""
    import torch
    mb = 1 << 20
    be = B200Backend(0, precision="f32")
    small = be.alloc(20)
    be.init_basis(small, 0)
    be.execute_batch([random_circuit(20, 40, 1)], probabilities=False)
    be.download(be.execute(random_circuit(24, 1, 1)))
    circuits = [random_circuit(20, 40, i) for i in range(15)]  # 16 MB each
    torch.cuda.synchronize()
    torch.cuda.empty_cache()

    def fill(leave):
        return torch.empty(device_free() - leave, dtype=torch.uint8, device="cuda")

    be.sample_device(small, 1000000, 1)
    be.alloc(23).free()
    full = fill(200 * mb)
    assert device_free() < 204 * mb
    z0, _, _ = be.execute_batch(circuits, probabilities=False)
    del full
    torch.cuda.empty_cache()
    assert max_abs_diff(z0, be.execute_batch(circuits, probabilities=False)[0]) == 0

    be.sample_device(small, 1000000, 1)  # keeps between 40 and 64 MB
    full = fill(100 * mb)
    state = be.alloc(24)  # 128 MB
    be.init_basis(state, 3)
    assert be.amplitude(state, 3) == 1
    state.free()
    del full
    torch.cuda.empty_cache()
    be.close()


def test_first_calls_of_a_context_find_their_memory_written(built):
    """Counters, flags and plan matrices are in place before the context's stream reads them, on memory that held
    other bits before."""
    import torch
    rng = np.random.default_rng(3)
    for i in range(20):
        junk = torch.full((64 << 20,), 255, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        del junk
        torch.cuda.empty_cache()
        be = B200Backend(0, precision="f64")
        s = be.alloc(9)
        be.init_basis(s, i)
        assert be.norm_sqr(s) == 1.0 and be.expectation_z(s, 1) == (-1.0 if i & 1 else 1.0)
        c = Circuit(9)
        for q in range(4):
            u = np.linalg.qr(rng.normal(size=(64, 64)) + 1j * rng.normal(size=(64, 64)))[0]
            c.push(DenseGate(6, u), list(range(q, q + 6)))
        psi = np.zeros(512, dtype=complex)
        psi[i] = 1
        Plan(be, c, L.make_opts(L.PLAN_AS_GIVEN, 6)).run(s)
        assert max_abs_diff(numpy_run(c, psi), be.download(s).as_complex()) <= 1e-12
        s.free()
        be.close()
