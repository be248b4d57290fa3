"""Passes at the most shared memory their descriptors can take.

A pass holds up to 192 ops: two-qubit gates need about a stage for every two of
them and 16 matrix entries each, five-qubit diagonals 32 entries; with 64
gradients the FP64 reverse pass then nears what a block may have (227 KB).  One
pass of each kind also shares a launch of the serving loop, which takes the
larger of the two, not the sum of their largest parts.  Bounds: helpers.py, for
energies and gradients times 3 n >= the sum of |coefficients| of the operator
(random circuits leave both near zero, so their own size is no scale).
"""
import numpy as np
import pytest

import vqcb200 as V
from helpers import as_input, max_abs, rand_psi, tol
from oracle import oracle as O
from vqcb200 import workloads as W
from vqcb200.serve import Server

pytestmark = pytest.mark.gpu


def rand_unitary(rng, d):
    q, r = np.linalg.qr(rng.normal(size=(d, d)) + 1j * rng.normal(size=(d, d)))
    return q * (np.diag(r) / np.abs(np.diag(r)))


def crowded(rng, n, kind, count=200, params=64):
    """Gates of one pass: dense pairs, or diagonals on five qubits; then CRx with gradients."""
    gates = []
    for i in range(count):
        q = [int(x) + 1 for x in rng.choice(n, 2 if kind == "pairs" else 5, replace=False)]
        if kind == "pairs":
            gates.append(V.QuantumGate(tuple(q), rand_unitary(rng, 4)))
        else:
            gates.append(V.QuantumGate(tuple(q), np.diag(np.exp(1j * rng.uniform(0, 6, 32)))))
        if i % 3 == 0 and params:
            params -= 1
            gates.append(V.CRxGate(tuple(q[:2]), float(rng.uniform(0, 6)), isparas=True))
    return V.QCircuit(gates)


def reference(c):
    return [([p - 1 for p in g.positions], g.mat, g.derivatives()) for g in c]


@pytest.mark.parametrize("dtype,n", [(np.complex64, 12), (np.complex128, 11), (np.complex128, 20)])
@pytest.mark.parametrize("kind", ["pairs", "diagonals"])
def test_crowded_passes(dtype, n, kind):
    rng = np.random.default_rng(600 + n)
    c, H = crowded(rng, min(n, 11), kind), W.to_operator(W.xxz_spec(n, 0.5))
    psi = rand_psi(rng, n)
    s = V.StateVector(psi.astype(dtype), dtype=dtype)
    got = V.apply(c, V.StateVector(psi.astype(dtype), dtype=dtype))
    e, g = V.energy_and_gradient(H, c, s)
    assert max_abs(got.storage(), O.apply_circuit(as_input(psi, dtype), reference(c), nthreads=4)) < tol(dtype)
    e_ref, g_ref = O.energy_and_gradient(reference(c), O.terms_from_spec(W.xxz_spec(n, 0.5)), as_input(psi, dtype),
                                         nthreads=4)
    assert len(g_ref) == 64
    assert abs(e - e_ref) < tol(dtype) * 3 * n
    assert max_abs(g, g_ref) < tol(dtype) * 3 * n


@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
def test_crowded_passes_in_one_launch(dtype):
    n, rng = 11, np.random.default_rng(620)
    cs = [crowded(rng, n, k) for k in ("pairs", "diagonals") for _ in range(4)]
    h = W.xxz_spec(n, 0.5)
    with Server(dtype=dtype, memory_bytes=1 << 30, max_active=16) as srv:
        tickets = [srv.submit(n, c, W.to_operator(h), want_grad=True) for c in cs]
        results = [srv.wait(t) for t in tickets]
    for c, (e, g, _) in zip(cs, results):
        e_ref, g_ref = O.energy_and_gradient(reference(c), O.terms_from_spec(h), O.zero_state(n), nthreads=4)
        assert abs(e - e_ref) < tol(dtype) * 3 * n
        assert max_abs(g, g_ref) < tol(dtype) * 3 * n
