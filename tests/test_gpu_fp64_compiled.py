"""FP64 passes compiled at run time against the interpreted ones.

Both run the same device functions in the same order, so a state, an energy
and a gradient have the same bits whichever kernel ran: a circuit's first call
(interpreted) and its later ones (compiled, from the second on) agree exactly.
The oracle bounds of both are asserted elsewhere (test_gpu_fused.py,
test_gpu_tile_forms.py, test_gpu_diag_ops.py with VQC_JIT on and off).
"""
import numpy as np
import pytest

import vqcb200 as V
from helpers import rand_psi
from test_gpu_fused import random_mixed_circuit
from vqcb200 import workloads as W

pytestmark = pytest.mark.gpu


def test_same_bits(monkeypatch):
    """Every kind of gate, forward and in the reverse sweep: the first call
    (interpreted) and the later ones (compiled)."""
    monkeypatch.delenv("VQC_JIT", raising=False)
    n = 23  # the smallest size that compiles by default
    rng = np.random.default_rng(500)
    c, _ = random_mixed_circuit(rng, n, 40, with_wide=False)
    psi0, target = rand_psi(rng, n), rand_psi(rng, n)
    first = None
    for _ in range(3):
        y = c * V.StateVector(psi0)
        out = y.storage()
        delta, g, yin = V.back_propagate(V.StateVector(target), c, y)
        got = (out, g, delta.storage(), yin.storage())
        first = first or got
        for a, b in zip(first, got):
            assert np.array_equal(a, b)


def test_calls_agree_across_the_compile(monkeypatch):
    """The default mode at a size that compiles: interpreted, then compiled."""
    monkeypatch.delenv("VQC_JIT", raising=False)
    n, layers = 23, 2
    rng = np.random.default_rng(510)
    c = W.to_circuit(W.rxyz_crx_spec(n, layers, rng.uniform(0, 2 * np.pi, layers * (4 * n - 1))))
    H, s = W.to_operator(W.xxz_spec(n, 0.5)), V.StateVector(n)
    first = V.energy_and_gradient(H, c, s)
    for _ in range(2):
        again = V.energy_and_gradient(H, c, s)
        assert again[0] == first[0]
        assert np.array_equal(again[1], first[1])
