"""Passes of one or two diagonal gates from 18 qubits, against the oracle.

Such a pass ends in a coalesced stage without ops, its matrices fill one 16-byte
word of shared memory, and nothing lies behind them: the interpreter must not
read ahead there (with the debug library the index checks see it).  Bounds:
helpers.py.
"""
import numpy as np
import pytest

import test_gpu_pass_memory as crowded
import vqcb200 as V
from helpers import as_input, max_abs, rand_psi, rel, tol
from oracle import oracle as O

pytestmark = pytest.mark.gpu

CIRCUITS = {"cz": [V.CZGate(2, 3)], "cphase": [V.CPHASEGate(1, 4, 0.7, isparas=True)],
            "two": [V.CZGate(2, 3), V.CPHASEGate(1, 2, 0.3, isparas=True)], "x": [V.XGate(2)]}


@pytest.mark.parametrize("dtype,n,jit", [(np.complex128, 18, ""), (np.complex128, 19, "off"), (np.complex64, 18, "off")])
@pytest.mark.parametrize("name", sorted(CIRCUITS))
def test_smallest_passes(name, dtype, n, jit, monkeypatch):
    if jit:
        monkeypatch.setenv("VQC_JIT", jit)
    c, rng = V.QCircuit(CIRCUITS[name]), np.random.default_rng(700)
    ref = [([p - 1 for p in g.positions], g.mat, g.derivatives()) for g in c]
    psi0, target = as_input(rand_psi(rng, n), dtype), as_input(rand_psi(rng, n), dtype)
    y = c * V.StateVector(psi0.astype(dtype), dtype=dtype)
    assert max_abs(y.storage(), O.apply_circuit(psi0.copy(), ref, nthreads=4)) < tol(dtype)
    g_ref, _ = O.circuit_gradient(ref, psi0, target, nthreads=4)
    _, g, yin = V.back_propagate(V.StateVector(target.astype(dtype), dtype=dtype), c, y)
    assert max_abs(yin.storage(), psi0) < tol(dtype)
    assert len(g) == len(g_ref) and (len(g) == 0 or rel(g, g_ref) < tol(dtype))


@pytest.mark.parametrize("kind", ["pairs", "diagonals"])
def test_crowded_packed_passes(kind, monkeypatch):
    """The other end, on the FP32 packed plan: up to 192 ops in a pass, 76 stages, 191 KB of shared memory."""
    monkeypatch.setenv("VQC_JIT", "interp")
    crowded.test_crowded_passes(np.complex64, 18, kind)
