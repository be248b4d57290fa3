"""Gates whose phases the planner defers, against the oracle.

A merged one-qubit gate runs as [[1, x], [y, 1]] and leaves a phase pending on
its qubit until the next such gate there; controlled, two-qubit and diagonal
gates in between see rotated matrices, gates outside the tile passes must not
see any.  The cases are where that can go wrong: deep circuits (the factor of
the state), gates that are not unitary, pivots that are zero or tiny, two-qubit
gates and standalone gates between one-qubit ones, and every gradient's frame.
Bounds: helpers.py.
"""
import numpy as np
import pytest

import vqcb200 as V
from helpers import as_input, max_abs, rand_psi, rel, tol
from oracle import gates_ref as GR
from oracle import oracle as O
from vqcb200 import _lib
from vqcb200 import workloads as W

pytestmark = pytest.mark.gpu
DTYPES = [np.complex64, np.complex128]


def reference(c):
    return [([p - 1 for p in g.positions], g.mat, g.derivatives()) for g in c]


def check_forward(gates, n, dtype, rng, unitary=True):
    c = V.QCircuit(gates)
    psi = rand_psi(rng, n)
    got = V.apply(c, V.StateVector(psi.astype(dtype), dtype=dtype)).storage()
    want = O.apply_circuit(as_input(psi, dtype), reference(c), nthreads=4)
    assert (max_abs(got, want) if unitary else rel(got, want)) < tol(dtype)


def check_gradient(gates, n, dtype, rng):
    c = V.QCircuit(gates)
    psi0, target = as_input(rand_psi(rng, n), dtype), as_input(rand_psi(rng, n), dtype)
    g_ref, d_ref = O.circuit_gradient(reference(c), psi0, target, nthreads=4)
    y = c * V.StateVector(psi0.astype(dtype), dtype=dtype)
    delta, g, yin = V.back_propagate(V.StateVector(target.astype(dtype), dtype=dtype), c, y)
    assert rel(g, g_ref) < tol(dtype)
    assert max_abs(yin.storage(), psi0) < tol(dtype)
    assert max_abs(delta.storage(), d_ref) < tol(dtype)


def between(rng, n):
    """One gate of every kind a pending phase has to pass."""
    q = [int(x) + 1 for x in rng.choice(n, 3, replace=False)]
    t = float(rng.uniform(0, 6))
    return [V.CRxGate(q[0], q[1], t, isparas=True), V.CRyGate(q[1], q[2], t, isparas=True), V.CNOTGate(q[2], q[0]),
            V.CZGate(q[0], q[1]), V.CPHASEGate(q[1], q[2], t, isparas=True), V.iSWAPGate(q[0], q[2]),
            V.QuantumGate((q[2], q[1]), GR.random_unitary(2, rng)), V.TOFFOLIGate(*q), V.FREDKINGate(*q)]


@pytest.mark.parametrize("jit", ["off", "on", "interp"])
@pytest.mark.parametrize("dtype", DTYPES)
def test_every_gate_between(dtype, jit, monkeypatch):
    monkeypatch.setenv("VQC_JIT", jit)
    n, rng = 13, np.random.default_rng(600)
    gates = []
    for g in between(rng, n) + between(rng, n) + between(rng, n):
        for q in g.positions:
            gates.append(V.U3Gate(q, *rng.uniform(0, 6, 3), isparas=True))
        gates.append(g)
    check_forward(gates, n, dtype, rng)
    check_gradient(gates, n, dtype, rng)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("n", [9, 10, 13])
def test_deep_circuit(dtype, n):
    """Hundreds of deferred gates: their product of norms underflows unless it is applied pass by pass."""
    rng = np.random.default_rng(610 + n)
    gates = []
    for layer in range(40):
        gates += [V.U3Gate(q, *rng.uniform(0, 6, 3), isparas=layer % 8 == 0) for q in range(1, n + 1)]
        gates += [V.CZGate(q, q + 1) for q in range(1 + layer % 2, n, 2)]
    check_forward(gates, n, dtype, rng)
    check_gradient(gates[:12 * (n + n // 2)], n, dtype, rng)


@pytest.mark.parametrize("dtype", DTYPES)
def test_special_angles(dtype):
    """Pivots that are zero, tiny or one: X, RX(pi), RX(pi - 1e-7), RZ, H, Y."""
    n, rng = 10, np.random.default_rng(620)
    gates = []
    for _ in range(6):
        for q in range(1, n + 1):
            t = [0.0, np.pi, np.pi - 1e-7, np.pi / 2, 1e-9, 2 * np.pi][int(rng.integers(6))]
            gates.append([V.XGate(q), V.RxGate(q, t, isparas=True), V.RyGate(q, t, isparas=True),
                          V.RzGate(q, t, isparas=True), V.HGate(q), V.YGate(q)][int(rng.integers(6))])
        gates += [V.CNOTGate(q, q + 1) for q in range(1, n)]
    check_forward(gates, n, dtype, rng)
    check_gradient(gates, n, dtype, rng)


@pytest.mark.parametrize("dtype", DTYPES)
def test_gates_that_are_not_unitary(dtype):
    n, rng = 11, np.random.default_rng(630)
    gates = []
    for i in range(5):
        for q in range(1, n + 1):
            a = rng.standard_normal((2, 2)) + 1j * rng.standard_normal((2, 2))
            if q % 3 == 0:
                a = np.array([[1, 0.3j], [0.2, np.exp(1j * i)]])  # equal moduli on the diagonal
            if q % 5 == 0:
                a = np.diag([1.0, 0.0]) if i == 2 else a * 1e-3
            gates.append(V.QuantumGate((q,), a))
        gates += [V.CNOTGate(q, q + 1) for q in range(1, n)]
    check_forward(gates, n, dtype, rng, unitary=False)


@pytest.mark.parametrize("dtype", DTYPES)
def test_standalone_gates_between(dtype):
    """Three- and four-qubit dense gates run between the passes, on plain amplitudes."""
    n, rng = 12, np.random.default_rng(640)
    gates = []
    for k in (3, 4, 3):
        gates += [V.U3Gate(q, *rng.uniform(0, 6, 3), isparas=True) for q in range(1, n + 1)]
        gates += [V.CRxGate(q, q + 1, float(rng.uniform(0, 6)), isparas=True) for q in range(1, n)]
        gates.append(V.QuantumGate(tuple(int(x) + 1 for x in rng.choice(n, k, replace=False)), GR.random_unitary(k, rng)))
    gates += [V.U3Gate(q, *rng.uniform(0, 6, 3), isparas=True) for q in range(1, n + 1)]
    check_forward(gates, n, dtype, rng)
    check_gradient(gates, n, dtype, rng)


def test_new_angles_reuse_compiled_passes(monkeypatch):
    """Which form a gate takes depends on its place, not on its angle."""
    monkeypatch.setenv("VQC_JIT", "on")
    n, layers, rng = 18, 3, np.random.default_rng(650)
    H = W.to_operator(W.xxz_spec(n, 0.5))
    s = V.StateVector(n, dtype=np.complex64)
    for i in range(4):
        c = W.to_circuit(W.rxyz_crx_spec(n, layers, rng.uniform(0, 2 * np.pi, layers * (4 * n - 1))))
        _lib.profile_enable(True)
        V.energy_and_gradient(H, c, s)
        _lib.profile_enable(False)
        compiled = _lib.profile_read().get("jit_compiled_passes", (0,))[0]
        assert i == 0 or compiled == 0
