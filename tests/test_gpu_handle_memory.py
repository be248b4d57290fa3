"""Device memory kept between handles: reuse, and giving it back.

Handles that end leave their buffers (at most 1 GiB a device) to the next ones.
Whatever allocation of the library then fails must get that memory back first;
free memory is read from the driver.  Bounds of the results: helpers.py.
"""
import threading

import numpy as np
import pytest

import vqcb200 as V
from helpers import max_abs, max_rel, rand_psi
from oracle import oracle as O
from vqcb200 import _lib
from vqcb200 import workloads as W
from vqcb200.serve import Server

pytestmark = pytest.mark.gpu
MB = 1 << 20


def free_bytes():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def leave_buffers(count, n=25):
    """`count` buffers of 2^n FP32 amplitudes in the pool (256 MiB each at 25)."""
    states = [V.StateVector(n, dtype=np.complex64) for _ in range(count)]
    del states


def test_reuse_across_sizes_and_streams():
    """Handles in turn and in threads take over each other's buffers and stay right."""
    rng = np.random.default_rng(940)
    keep = V.StateVector(4)
    psi = {n: rand_psi(rng, n) for n in (9, 10, 12)}
    specs = {n: W.rxyz_crx_spec(n, 1, rng.uniform(0, 6, 4 * n - 1)) for n in psi}
    want = {n: O.apply_circuit(psi[n].copy(), O.from_spec(specs[n])) for n in psi}
    wrong = []

    def work(n):
        for _ in range(8):
            got = V.apply(W.to_circuit(specs[n]), V.StateVector(psi[n]))
            other = V.StateVector(n)  # a fresh handle is |0...0> whatever its buffer held
            if max_abs(got.storage(), want[n]) > 1e-12 or max_abs(other.storage(), O.zero_state(n)) > 0:
                wrong.append(n)

    for n in psi:
        work(n)
    threads = [threading.Thread(target=work, args=(n,)) for n in (9, 10, 12, 10)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not wrong and len(keep.storage()) == 16


def test_given_back_with_the_last_handle_and_on_a_failed_allocation():
    leave_buffers(1)  # (what the first handle of the process sets up stays out of the count)
    start = free_bytes()
    keep = V.StateVector(4)
    leave_buffers(3)
    assert start - free_bytes() > 700 * MB
    with pytest.raises(Exception):
        V.StateVector(36, dtype=np.complex64)  # 512 GiB
    assert start - free_bytes() < 100 * MB
    leave_buffers(3)
    assert start - free_bytes() > 700 * MB
    assert len(keep.storage()) == 16
    del keep
    assert start - free_bytes() < 100 * MB


def test_serving_takes_the_kept_memory():
    """A request's memory (516 MiB) fits only once the kept buffers (768 MiB) are given back."""
    import torch
    n, rng = 25, np.random.default_rng(950)
    c = W.to_circuit(W.hea_spec(n, 1, rng.uniform(0, 6, 2 * n)))
    H = W.to_operator(W.tfim_spec(n, 0.7))
    with Server(dtype=np.complex64, memory_bytes=1 << 30, max_active=2) as srv:
        e_ref, g_ref, _ = srv.wait(srv.submit(n, c, H, want_grad=True))
    keep = V.StateVector(4)
    leave_buffers(3)
    fill = [torch.empty(free_bytes() - 400 * MB, dtype=torch.uint8, device="cuda")]
    try:
        with Server(dtype=np.complex64, memory_bytes=1 << 30, max_active=2) as srv:
            e, g, _ = srv.wait(srv.submit(n, c, H, want_grad=True))
    finally:
        fill.clear()
        torch.cuda.empty_cache()
    assert abs(e - e_ref) <= 1e-5 * abs(e_ref) and np.linalg.norm(g - g_ref) <= 1e-5 * np.linalg.norm(g_ref)
    assert len(keep.storage()) == 16


@pytest.mark.parametrize("n,kept", [(9, True), (13, False)])
def test_a_large_partial_trace_leaves_nothing_on_its_handle(n, kept):
    """One qubit traced out of 13 is 256 MiB of result: it goes back with the call, and the handle's next
    allocation finds it (the second trace of the same size takes no more)."""
    rng = np.random.default_rng(960)
    psi = rand_psi(rng, n)
    rho = V.DensityMatrix(V.StateVector(psi.astype(np.complex64), dtype=np.complex64))
    m = psi.astype(np.complex64).astype(np.complex128).reshape(-1, 2)  # (the row's low bit is qubit 1)
    for _ in range(2):
        assert max_rel(V.partial_tr(rho, [1]), m @ m.conj().T) < 1e-5
    if kept:
        return
    with pytest.raises(Exception):
        V.StateVector(36, dtype=np.complex64)  # gives the kept memory back
    before = free_bytes()
    V.partial_tr(rho, [1])
    with pytest.raises(Exception):
        V.StateVector(36, dtype=np.complex64)
    assert before - free_bytes() < 64 * MB


def test_the_first_gradient_of_a_handle_sizes_its_buffers_once(monkeypatch):
    """Descriptors (forward, reverse), sums, rows: one growth each, not one for every chunk of the sweep."""
    monkeypatch.setenv("VQC_JIT", "interp")
    n, layers, rng = 18, 20, np.random.default_rng(970)
    c = W.to_circuit(W.rxyz_crx_spec(n, layers, rng.uniform(0, 6, layers * (4 * n - 1))))
    H, grown = W.to_operator(W.xxz_spec(n, 0.5)), []
    psi = V.StateVector(n, dtype=np.complex64)
    for _ in range(2):
        _lib.profile_enable(True)
        V.energy_and_gradient(H, c, psi)
        _lib.profile_enable(False)
        grown.append(_lib.profile_read().get("handle_buffer_grown", (0,))[0])
    assert 0 < grown[0] <= 4 and grown[1] == 0
