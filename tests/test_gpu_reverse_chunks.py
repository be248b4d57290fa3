"""Gradients of circuits with many gates outside the tile passes.

Each such gate splits the reverse sweep into runs of passes, and every run is at
least one chunk of it: from 65 chunks on their doubling size once overflowed.
Bounds: helpers.py.
"""
import numpy as np
import pytest

import vqcb200 as V
from helpers import as_input, max_abs, rand_psi, rel, tol
from oracle import gates_ref as GR
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def circuit(rng, n, kind, count):
    gates = []
    for _ in range(count):
        q = [int(x) + 1 for x in rng.choice(n, 3, replace=False)]
        gates += [V.RxGate(k, float(rng.uniform(0, 6)), isparas=True) for k in q]
        if kind == "dense":
            gates.append(V.QuantumGate(tuple(q), GR.random_unitary(3, rng)))
        else:
            gates.append(V.CCPHASEGate(*q, float(rng.uniform(0, 6)), isparas=True))
    return V.QCircuit(gates)


@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
@pytest.mark.parametrize("kind,count", [("dense", 64), ("dense", 70), ("ccphase", 66), ("dense", 140)])
def test_many_gates_outside_the_passes(kind, count, dtype):
    n, rng = 10, np.random.default_rng(930 + count)
    c = circuit(rng, n, kind, count)
    ref = [([p - 1 for p in g.positions], g.mat, g.derivatives()) for g in c]
    psi0, target = as_input(rand_psi(rng, n), dtype), as_input(rand_psi(rng, n), dtype)
    g_ref, d_ref = O.circuit_gradient(ref, psi0, target, nthreads=4)
    y = c * V.StateVector(psi0.astype(dtype), dtype=dtype)
    delta, g, yin = V.back_propagate(V.StateVector(target.astype(dtype), dtype=dtype), c, y)
    assert rel(g, g_ref) < tol(dtype)
    assert max_abs(yin.storage(), psi0) < tol(dtype)
    assert max_abs(delta.storage(), d_ref) < tol(dtype)
