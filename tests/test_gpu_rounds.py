"""Register-phase programs (rounds) of tile sweeps on circuits that reach every kind of place in them."""
import numpy as np
import pytest

from rustatevec_b200 import _lib as L
from rustatevec_b200 import gate as G
from rustatevec_b200.circuit import Circuit

from helpers import max_abs_diff, numpy_run

pytestmark = pytest.mark.gpu


def haar1(rng):
    return np.linalg.qr(rng.normal(size=(2, 2)) + 1j * rng.normal(size=(2, 2)))[0]


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("kind", ["cphase", "rzz", "mixed"])
def test_tile_diagonals_in_every_place(be32, be64, precision, kind):
    """Rounds of 1-qubit gates with diagonals between them: register x register, register x group bits (one
    and two table windows) and register x tile bits, with the 0 side equal to 1 (controlled phases) and not,
    then CX gates up and down and a SWAP. Each gate is off by a few roundings of unit-norm vectors: 8 u a
    gate, u the unit roundoff, bounds the sum."""
    be = be32 if precision == "f32" else be64
    n = 16
    rng = np.random.default_rng(5)
    c = Circuit(n)
    for layer in range(3):
        for q in range(n):
            [c.h, lambda q: c.rx(q, 0.3 + q), lambda q: c.push(G.DenseGate(1, haar1(rng)), [q])][(q + layer) % 3](q)
            for k in (rng.permutation(n)[:4]).tolist():
                if k != q:
                    a = float(rng.uniform(0, 6))
                    if kind == "cphase" or (kind == "mixed" and k % 2):
                        c.cphase(q, k, a)
                    else:
                        c.rzz(q, k, a)
        for q in range(n - 1):
            c.cx(q, q + 1) if layer % 2 else c.cx(q + 1, q)
        c.swap(1, n - 2)
    psi = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    psi = (psi / np.linalg.norm(psi)).astype(np.complex64 if precision == "f32" else np.complex128)
    st = be.alloc(n)
    be.upload(st, psi.real, psi.imag)
    assert "tile" in be.run(st, c, L.make_opts(L.PLAN_TILE, 4))["by_kind"]
    err = max_abs_diff(numpy_run(c, psi), be.download(st).as_complex())
    assert err <= 8 * len(c) * (2.0 ** -24 if precision == "f32" else 2.0 ** -53), err
    st.free()
