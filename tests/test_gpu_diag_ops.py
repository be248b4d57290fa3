"""Diagonal gates in the tile passes against the oracle.

A diagonal op costs what its table holds (one entry that is not 1, exactly -1,
or a full table) and where its qubits lie (the lane bit, another register bit,
a thread bit, outside the tile): the compiled passes write each combination
out.  The circuits put every class on every kind of place, next to dense gates
that move the register bits from stage to stage.  Bounds: helpers.py.
"""
import itertools

import numpy as np
import pytest

import vqcb200 as V
from helpers import as_input, max_abs, rand_psi, rel, tol
from oracle import oracle as O

pytestmark = pytest.mark.gpu

PLACES = [1, 2, 3, 7, 11, 13, 14]  # lane bit, low, middle, high, outside a tile of 12


def diag_gates(rng, k):
    """A flip, a phase at another entry than the last, and a full table on k-tuples of places."""
    out = []
    combos = list(itertools.permutations(PLACES, k))
    for i in rng.choice(len(combos), min(len(combos), 10), replace=False):
        q = combos[i]
        d = np.ones(1 << k, dtype=complex)
        d[-1] = -1
        out.append(V.QuantumGate(q, np.diag(d)))
        d = np.ones(1 << k, dtype=complex)
        d[rng.integers(0, 1 << k)] = np.exp(1j * rng.uniform(0, 6))
        out.append(V.QuantumGate(q, np.diag(d)))
        out.append(V.QuantumGate(q, np.diag(np.exp(1j * rng.uniform(0, 6, 1 << k)))))
    return out


def mixed(rng, n, diags):
    gates = []
    for g in diags:
        gates.append(V.U3Gate(int(rng.integers(1, n + 1)), *rng.uniform(0, 6, 3), isparas=True))
        gates.append(g)
    return V.QCircuit(gates)


def reference(c):
    return [([p - 1 for p in g.positions], g.mat, g.derivatives()) for g in c]


@pytest.mark.parametrize("jit", ["off", "on", "interp"])
@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
@pytest.mark.parametrize("k", [2, 3, 4, 5])
def test_diagonal_gates(dtype, k, jit, monkeypatch):
    monkeypatch.setenv("VQC_JIT", jit)
    n, rng = 14, np.random.default_rng(400 + k)
    c = mixed(rng, n, diag_gates(rng, k))
    psi = rand_psi(rng, n)
    s = V.apply(c, V.StateVector(psi.astype(dtype), dtype=dtype))
    assert max_abs(s.storage(), O.apply_circuit(as_input(psi, dtype), reference(c), nthreads=4)) < tol(dtype)


@pytest.mark.parametrize("jit", ["off", "on", "interp"])
@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
def test_diagonal_parameters(dtype, jit, monkeypatch):
    """CPHASE and CRZ partials: the diagonal bins of the reverse sweep."""
    monkeypatch.setenv("VQC_JIT", jit)
    n, rng = 14, np.random.default_rng(410)
    pairs = [p for p in itertools.permutations(PLACES, 2)]
    diags = [(V.CPHASEGate if i % 2 else V.CRzGate)(*pairs[j], float(rng.uniform(0, 6)), isparas=True)
             for i, j in enumerate(rng.choice(len(pairs), 24, replace=False))]
    c = mixed(rng, n, diags)
    psi0, target = as_input(rand_psi(rng, n), dtype), as_input(rand_psi(rng, n), dtype)
    g_ref, d_ref = O.circuit_gradient(reference(c), psi0, target, nthreads=4)
    y = c * V.StateVector(psi0.astype(dtype), dtype=dtype)
    delta, g, yin = V.back_propagate(V.StateVector(target.astype(dtype), dtype=dtype), c, y)
    assert rel(g, g_ref) < tol(dtype)
    assert max_abs(yin.storage(), psi0) < tol(dtype)
    assert max_abs(delta.storage(), d_ref) < tol(dtype)
