"""Deferred phases where they are planned: the range of the FP32 amplitudes in
flight, and the cases of test_gpu_deferred_phases.py on plans that defer.

The first part holds circuits whose deferred factors pile up unless the planner
counts them in the order the ops run: a gradient must be finite and within the
bounds.  The second runs deep circuits, special angles, gates that are not
unitary and standalone gates with run-time compiled passes (VQC_JIT=on) and the
packed interpreter (interp), and checks that phases were deferred at all.
Bounds: helpers.py.
"""
import os

import numpy as np
import pytest

import test_gpu_deferred_phases as D
import vqcb200 as V
from vqcb200 import _lib

pytestmark = pytest.mark.gpu
PLANS = [(np.complex64, "on"), (np.complex64, "interp"), (np.complex128, "on")]


def deferred(run):
    if _lib.load().vqc_debug_build() and os.environ.get("VQC_JIT") != "interp":
        pytest.skip("the debug library compiles no passes: nothing is deferred")
    _lib.profile_enable(True)
    try:
        run()
    finally:
        _lib.profile_enable(False)
    return _lib.profile_read().get("plan_forward_deferred", (0,))[0]


def blocks(rng, n, layers, block):
    """RZ RY RZ on every qubit and CZ inside blocks of qubits; RY carries a parameter in every tenth layer."""
    gates = []
    for layer in range(layers):
        for q in range(1, n + 1):
            t = rng.uniform(0, 2 * np.pi, 3)
            gates += [V.RzGate(q, t[0]), V.RyGate(q, t[1], isparas=layer % 10 == 5), V.RzGate(q, t[2])]
        gates += [V.CZGate(q, q + 1) for q in range(1, n) if (q - 1) // block == q // block]
    return gates


@pytest.mark.parametrize("block,layers", [(2, 20), (2, 40), (2, 80), (3, 40)])
def test_qubits_that_meet_in_blocks(block, layers, monkeypatch):
    """One stage runs all layers of its few qubits (interpreted: such passes take long to compile)."""
    monkeypatch.setenv("VQC_JIT", "interp")
    n, rng = 18, np.random.default_rng(900 + block + layers)
    D.check_gradient(blocks(rng, n, layers, block), n, np.complex64, rng)


@pytest.mark.parametrize("layers", [4, 8])
def test_rotations_next_to_pi(layers):
    """|m00| = 4e-8: two such gates leave the FP32 window."""
    n, rng = 18, np.random.default_rng(910 + layers)
    gates = []
    for layer in range(layers):
        gates += [V.RxGate(q, float(np.float32(np.pi)), isparas=layer % 4 == 1) for q in range(1, n + 1)]
        gates += [V.CZGate(q, q + 1) for q in range(1 + layer % 2, n, 2)]
    D.check_forward(gates, n, np.complex64, rng)
    gates += [V.RyGate(q, float(t), isparas=True) for q, t in enumerate(rng.uniform(0, 6, n), 1)]
    D.check_gradient(gates, n, np.complex64, rng)


@pytest.mark.parametrize("dtype,jit", PLANS)
@pytest.mark.parametrize("n", [9, 13])
def test_deep_circuit(dtype, jit, n, monkeypatch):
    monkeypatch.setenv("VQC_JIT", jit)
    assert deferred(lambda: D.test_deep_circuit(dtype, n)) > 0


@pytest.mark.parametrize("dtype,jit", PLANS)
@pytest.mark.parametrize("case", ["special_angles", "standalone_gates_between"])
def test_every_place(case, dtype, jit, monkeypatch):
    monkeypatch.setenv("VQC_JIT", jit)
    assert deferred(lambda: getattr(D, "test_" + case)(dtype)) > 0


@pytest.mark.parametrize("dtype,jit", PLANS)
def test_only_multiples_of_unitaries_are_deferred(dtype, jit, monkeypatch):
    monkeypatch.setenv("VQC_JIT", jit)
    assert deferred(lambda: D.test_gates_that_are_not_unitary(dtype)) == 0
    n, rng = 11, np.random.default_rng(920)
    gates = []
    for i in range(6):
        for q in range(1, n + 1):
            a = [1e-3, 1.0, 1e3][(q + i) % 3] * D.GR.random_unitary(1, rng)
            gates.append(V.QuantumGate((q,), a if (q + i) % 4 else a @ np.array([[1, 0.2], [0, 1]])))
        gates += [V.CNOTGate(q, q + 1) for q in range(1, n)]
    assert deferred(lambda: D.check_forward(gates, n, dtype, rng, unitary=False)) > 0


@pytest.mark.parametrize("dtype,n,defers", [(np.complex64, 17, False), (np.complex64, 18, True),
                                            (np.complex128, 20, False), (np.complex128, 22, False),
                                            (np.complex128, 23, True)])
def test_deferred_only_where_passes_are_compiled(dtype, n, defers, monkeypatch):
    """The interpreted passes run whole matrices."""
    monkeypatch.delenv("VQC_JIT", raising=False)
    c = V.QCircuit([V.U3Gate(q, 0.3 * q, 0.2, 0.1) for q in (1, 2)] + [V.CNOTGate(1, 2)] +
                   [V.U3Gate(q, 0.4, 0.2 * q, 0.1) for q in (1, 2)])
    psi = V.StateVector(n, dtype=dtype)
    assert (deferred(lambda: V.apply(c, psi)) > 0) == defers
    assert abs(psi.norm() - 1) < 1e-6
