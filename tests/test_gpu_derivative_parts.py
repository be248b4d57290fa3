"""FP64 gradients of derivatives whose Hermitian part is small, not rounding.

U^dagger dU of a unitary family is anti-Hermitian and the reverse sweep then sums
half the values.  Here its Hermitian part is 3e-13 of it, far above FP64 rounding,
and (U, the state and the cotangent being real) it alone makes the gradient.
Bound: helpers.py.
"""
import numpy as np
import pytest

import vqcb200 as V
from helpers import rel, tol
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("jit", ["off", "on"])
def test_small_hermitian_parts_count(jit, monkeypatch):
    monkeypatch.setenv("VQC_JIT", jit)
    n, rng = 11, np.random.default_rng(990)
    X, Z = np.array([[0, 1], [1, 0]], complex), np.diag([1, -1]).astype(complex)
    gates = []
    for q in range(1, n + 1):
        t = float(rng.uniform(0, 6)) / 2
        U = np.array([[np.cos(t), -np.sin(t)], [np.sin(t), np.cos(t)]], complex)
        gates.append(V.Gate((q,), U, (t,), True, [U @ (1j * Z + 3e-13 * (X + np.eye(2)))]))
        gates.append(V.CNOTGate(q, q % n + 1))
    c = V.QCircuit(gates)
    ref = [([p - 1 for p in g.positions], g.mat, g.derivatives()) for g in c]
    psi0, target = [v / np.linalg.norm(v) for v in rng.standard_normal((2, 1 << n)).astype(complex)]
    g_ref, _ = O.circuit_gradient(ref, psi0.copy(), target.copy(), nthreads=4)
    y = c * V.StateVector(psi0)
    _, g, _ = V.back_propagate(V.StateVector(target), c, y)
    assert np.linalg.norm(g_ref) > 0 and rel(g, g_ref) < tol(np.complex128)
