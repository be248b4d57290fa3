"""FP64 passes compile when they should: on a structure's second call, once, and
in one thread where several meet it.  Results agree bit for bit throughout
(interpreted and compiled passes run the same device functions)."""
import threading

import numpy as np
import pytest

import vqcb200 as V
from helpers import rand_psi
from vqcb200 import _lib
from vqcb200 import workloads as W

pytestmark = pytest.mark.gpu


def compiled(run):
    if _lib.load().vqc_debug_build():
        pytest.skip("the debug library compiles no passes")
    _lib.profile_enable(True)
    try:
        run()
    finally:
        _lib.profile_enable(False)
    return _lib.profile_read().get("jit_compiled_passes", (0,))[0]


def test_threads_share_one_compile(monkeypatch):
    monkeypatch.setenv("VQC_JIT", "on")
    n, rng = 11, np.random.default_rng(980)  # one tile: one pass
    c = W.to_circuit(W.u3_cnot_spec(n, 1, 980))
    psi = rand_psi(rng, n)
    go, out = threading.Barrier(4), [None] * 4

    def work(i):
        s = V.StateVector(psi)
        go.wait()
        out[i] = V.apply(c, s).storage()

    def run():
        threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
        [t.start() for t in threads]
        [t.join() for t in threads]

    assert compiled(run) == 1
    assert all(np.array_equal(o, out[0]) for o in out)


def test_default_mode_compiles_on_the_second_call(monkeypatch):
    monkeypatch.delenv("VQC_JIT", raising=False)
    n, rng = 23, np.random.default_rng(981)
    c = W.to_circuit(W.rxyz_crx_spec(n, 1, rng.uniform(0, 6, 4 * n - 1)))
    psi, target, got, counts = rand_psi(rng, n), rand_psi(rng, n), [], []
    for _ in range(3):
        def forward():
            got.append([c * V.StateVector(psi)])

        def reverse():
            delta, g, yin = V.back_propagate(V.StateVector(target), c, got[-1][0])
            got[-1] = [yin.storage(), delta.storage(), g]
        counts.append((compiled(forward), compiled(reverse)))
    assert counts[0] == (0, 0) and min(counts[1]) > 0 and counts[2] == (0, 0)
    for later in got[1:]:
        for a, b in zip(got[0], later):
            assert np.array_equal(a, b)
