"""The workloads this engine is timed on: what a user of the package has it do.

Each case is a dict of plain values; `prepare` makes what the user's program
holds before the call (circuit, operator, state handles, inputs from the seed),
`run` is one pass through the public entry points, `exact` the same quantities
from plain torch in complex128.  FP32 states give results of FP32 precision
(their sums are FP64), so energies and gradients of such a case are returned as
float32.

Kinds:
  vqe       energy_and_gradient(H, circuit, psi0): the step of every
            variational optimisation
  circuit   reset + apply(circuit, psi): sampling and simulation of a circuit
  gates     apply(gate, psi) one gate at a time: interactive and adaptive use
  observe   expectation, transition element, H psi, norm and a measurement
            probability of a given state
  dm        a density matrix through a circuit, then partial trace and
            probabilities
  noisy     energy and gradient of a noisy circuit (gates and channels) on a
            density matrix
  serve     a burst of variational requests of uneven sizes through one Server
"""
import math
import os
import random
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vqc.jl_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import vqcb200 as V  # noqa: E402
from vqcb200.serve import Server  # noqa: E402

DEV = "cuda" if torch.cuda.is_available() else "cpu"


def listed():
    return [
        # the smallest gradient of the package's own configurations: a 12-qubit
        # hardware-efficient ansatz in ComplexF64, where latency and launches count
        {"name": "vqe_n12_c128", "kind": "vqe", "n": 12, "layers": 6, "ansatz": "hea", "dtype": "c128"},
        # a small odd size in ComplexF32, below the run-time compiled passes
        {"name": "vqe_n17_c64", "kind": "vqe", "n": 17, "layers": 5, "ansatz": "hea", "dtype": "c64"},
        # an ordinary gradient, one state in L2
        {"name": "vqe_n21_c64", "kind": "vqe", "n": 21, "layers": 6, "ansatz": "rxyz", "dtype": "c64"},
        # the reference's own precision at an ordinary size (the check every FP32 result is held to)
        {"name": "vqe_n23_c128", "kind": "vqe", "n": 23, "layers": 4, "ansatz": "rxyz", "dtype": "c128"},
        # the headline gradient: 26 qubits, 20 layers, XXZ
        {"name": "vqe_n26_c64", "kind": "vqe", "n": 26, "layers": 20, "ansatz": "rxyz", "dtype": "c64"},
        # the largest state of the configurations, a deep circuit of U3, CZ and Toffoli
        {"name": "circuit_n30_c64", "kind": "circuit", "n": 30, "layers": 10, "wires": 7, "dtype": "c64"},
        # the same family in the reference's precision
        {"name": "circuit_n27_c128", "kind": "circuit", "n": 27, "layers": 6, "wires": 3, "dtype": "c128"},
        # gates applied one by one, every class and low, middle and high targets
        {"name": "gates_n28_c64", "kind": "gates", "n": 28, "wires": 5, "dtype": "c64"},
        # a state's observables
        {"name": "observe_n25_c64", "kind": "observe", "n": 25, "dtype": "c64"},
        # the 13-qubit density matrix of the configurations (1 GiB)
        {"name": "dm_n13_c128", "kind": "dm", "n": 13, "layers": 8, "traced": 4, "dtype": "c128"},
        # training against a noise model
        {"name": "noisy_n9_c128", "kind": "noisy", "n": 9, "layers": 2, "dtype": "c128"},
        # a burst of requests, 10 to 17 qubits and 2 to 12 layers, half of them with
        # gradients (larger requests change kernels while a server warms up over
        # minutes, which a pass of milliseconds cannot show)
        {"name": "serve_40_c64", "kind": "serve", "count": 40, "nmin": 10, "nmax": 17, "wires": 1, "dtype": "c64"},
    ]


def draw(rng):
    kind = rng.choice(["vqe", "vqe", "vqe", "circuit", "circuit", "gates", "observe", "dm", "noisy", "serve"])
    dtype = rng.choice(["c64", "c128"])
    if kind == "vqe":
        n = rng.randint(10, 24 if dtype == "c64" else 22)
        return {"kind": kind, "n": n, "layers": rng.randint(2, 8), "ansatz": rng.choice(["hea", "rxyz"]),
                "dtype": dtype}
    if kind == "circuit":
        n = rng.randint(14, 27 if dtype == "c64" else 26)
        return {"kind": kind, "n": n, "layers": rng.randint(2, 10), "wires": rng.randint(0, 999), "dtype": dtype}
    if kind == "gates":
        return {"kind": kind, "n": rng.randint(14, 28 if dtype == "c64" else 26), "wires": rng.randint(0, 999),
                "dtype": dtype}
    if kind == "observe":
        return {"kind": kind, "n": rng.randint(12, 26 if dtype == "c64" else 25), "dtype": dtype}
    if kind == "dm":
        n = rng.randint(6, 12)
        return {"kind": kind, "n": n, "layers": rng.randint(2, 8), "traced": rng.randint(1, n - 1), "dtype": dtype}
    if kind == "noisy":
        return {"kind": kind, "n": rng.randint(4, 9), "layers": rng.randint(1, 3), "dtype": dtype}
    lo = rng.randint(9, 13)
    return {"kind": kind, "count": rng.randint(8, 40), "nmin": lo, "nmax": rng.randint(lo + 1, 17),
            "wires": rng.randint(0, 999), "dtype": dtype}


# ----------------------------------------------------------------------------- circuits as plain lists
# An item is (name, wires, angles) with 1-based wires, as the package counts them.
def _hea(n, layers, rng):
    items = []
    for _ in range(layers):
        for q in range(1, n + 1):
            items += [("ry", (q,), (_angle(rng),)), ("rz", (q,), (_angle(rng),))]
        items += [("cnot", (q, q + 1), ()) for q in range(1, n)]
    return items


def _rxyz(n, layers, rng):
    items = []
    for _ in range(layers):
        for q in range(1, n + 1):
            items += [(g, (q,), (_angle(rng),)) for g in ("rx", "ry", "rz")]
        items += [("crx", (q, q + 1), (_angle(rng),)) for q in range(1, n)]
    return items


def _u3_cz_toffoli(n, layers, wires, rng):
    pick, items = random.Random(wires), []
    for layer in range(layers):
        items += [("u3", (q,), (_angle(rng), _angle(rng), _angle(rng))) for q in range(1, n + 1)]
        items += [("cz", (q, q + 1), ()) for q in range(1 + layer % 2, n, 2)]
        items.append(("toffoli", tuple(pick.sample(range(1, n + 1), 3)), ()))
    return items


def _u3_cnot(n, layers, rng):
    items = []
    for _ in range(layers):
        items += [("u3", (q,), (_angle(rng), _angle(rng), _angle(rng))) for q in range(1, n + 1)]
        items += [("cnot", (q, q + 1), ()) for q in range(1, n)]
    return items


def _noisy(n, layers, rng):
    items = []
    for _ in range(layers):
        for q in range(1, n + 1):
            items += [("ry", (q,), (_angle(rng),)), ("rz", (q,), (_angle(rng),))]
        items += [("cnot", (q, q + 1), ()) for q in range(1, n)]
        items += [("depolarizing", (q,), (0.02,)) for q in range(1, n + 1)]
    items += [("damping", (q,), (0.05,)) for q in range(1, n + 1)]
    return items


def _gate_list(n, wires, rng):
    """Every class of gate on a low, a middle and a high qubit and on pairs that mix them."""
    pick = random.Random(wires)
    mid = pick.randint(max(6, n // 3), n - 5)
    a, b, c = pick.sample(range(1, n + 1), 3)
    five = tuple(pick.sample(range(1, n + 1), 5))
    t = lambda: _angle(rng)  # noqa: E731
    return [("u3", (1,), (t(), t(), t())), ("u3", (mid,), (t(), t(), t())), ("u3", (n,), (t(), t(), t())),
            ("h", (3,), ()), ("rz", (2,), (t(),)), ("rz", (n - 1,), (t(),)), ("x", (mid,), ()),
            ("cnot", (1, 2), ()), ("cnot", (n, 3), ()), ("cnot", (mid, n - 2), ()), ("cz", (4, mid + 1), ()),
            ("cz", (1, 2), ()), ("crx", (2, n), (t(),)), ("crx", (mid, mid + 1), (t(),)), ("swap", (2, n - 1), ()),
            ("toffoli", (a, b, c), ()), ("toffoli", (1, mid, n), ()), ("dense", (1, mid), (t(), t())),
            ("dense", (n, n - 3), (t(), t())), ("dense", (a, c, b), (t(), t())), ("dense", five, (t(), t()))]


def _angle(rng):
    return rng.uniform(0, 2 * math.pi)


# ----------------------------------------------------------------------------- matrices of the plain items
_X = np.array([[0, 1], [1, 0]], complex)
_Y = np.array([[0, -1j], [1j, 0]], complex)
_Z = np.diag([1.0 + 0j, -1])
_PAULI = {"X": _X, "Y": _Y, "Z": _Z}


def _rot(P, t):
    c, s = math.cos(t / 2), math.sin(t / 2)
    return c * np.eye(2) - 1j * s * P, -0.5 * s * np.eye(2) - 0.5j * c * P


def _control(U):
    """U controlled by the first wire (the low index bit)."""
    d = U.shape[0]
    M = np.eye(2 * d, dtype=complex)
    M[1::2, 1::2] = U
    return M


def _dense(k, angles):
    """A fixed unitary of k qubits from two angles: the Cayley transform of a Hermitian matrix."""
    d = 1 << k
    i, j = np.meshgrid(np.arange(d), np.arange(d), indexing="ij")
    A = np.cos(angles[0] * (1 + i + j)) + 1j * np.sin(angles[1] * (1 + i * 3 + j))
    H = (A + A.conj().T) / 4
    return np.linalg.solve(np.eye(d) + 1j * H, np.eye(d) - 1j * H)


def _matrix(name, angles, k):
    """(matrix, [derivative for each angle]) of an item."""
    if name in ("rx", "ry", "rz"):
        U, dU = _rot(_PAULI[name[1].upper()], angles[0])
        return U, [dU]
    if name == "crx":
        U, dU = _rot(_X, angles[0])
        D = np.zeros((4, 4), complex)
        D[1::2, 1::2] = dU
        return _control(U), [D]
    if name == "u3":
        t, p, m = angles
        c, s = math.cos(t / 2), math.sin(t / 2)
        return np.array([[c, -np.exp(1j * m) * s], [np.exp(1j * p) * s, np.exp(1j * (p + m)) * c]]), []
    if name == "h":
        return np.array([[1, 1], [1, -1]], complex) / math.sqrt(2), []
    if name == "x":
        return _X, []
    if name == "cnot":
        return _control(_X), []
    if name == "cz":
        return np.diag([1, 1, 1, -1]).astype(complex), []
    if name == "swap":
        return np.eye(4, dtype=complex)[[0, 2, 1, 3]], []
    if name == "toffoli":
        return _control(_control(_X)), []
    if name == "dense":
        return _dense(k, angles), []
    raise ValueError(name)


def _kraus(name, p):
    if name == "depolarizing":
        a, b = math.sqrt(1 - p), math.sqrt(p / 3)
        return [a * np.eye(2), b * _X, b * _Y, b * _Z]
    return [np.diag([1, math.sqrt(1 - p)]).astype(complex), np.array([[0, math.sqrt(p)], [0, 0]], complex)]


def _operator_terms(kind, n, rng):
    """[(coefficient, {wire: letter})]: open-chain Ising in a transverse field, or XXZ."""
    if kind == "tfim":
        g = rng.uniform(0.2, 1.5)
        return ([(1.0, {i: "Z", i + 1: "Z"}) for i in range(1, n)] + [(g, {i: "X"}) for i in range(1, n + 1)])
    terms = []
    for i in range(1, n):
        terms += [(1.0, {i: "X", i + 1: "X"}), (1.0, {i: "Y", i + 1: "Y"}), (0.5, {i: "Z", i + 1: "Z"})]
    return terms


# ----------------------------------------------------------------------------- the same through the package
_GATE = {
    "rx": lambda w, a: V.RxGate(w[0], a[0], isparas=True),
    "ry": lambda w, a: V.RyGate(w[0], a[0], isparas=True),
    "rz": lambda w, a: V.RzGate(w[0], a[0], isparas=True),
    "crx": lambda w, a: V.CRxGate(w[0], w[1], a[0], isparas=True),
    "u3": lambda w, a: V.U3Gate(w[0], *a),
    "h": lambda w, a: V.HGate(w[0]),
    "x": lambda w, a: V.XGate(w[0]),
    "cnot": lambda w, a: V.CNOTGate(*w),
    "cz": lambda w, a: V.CZGate(*w),
    "swap": lambda w, a: V.SWAPGate(*w),
    "toffoli": lambda w, a: V.TOFFOLIGate(*w),
    "dense": lambda w, a: V.QuantumGate(w, _dense(len(w), a)),
    "depolarizing": lambda w, a: V.Depolarizing(w[0], a[0]),
    "damping": lambda w, a: V.AmplitudeDamping(w[0], a[0]),
}


def _circuit(items):
    return V.QCircuit([_GATE[name](w, a) for name, w, a in items])


def _operator(terms):
    return V.QubitsOperator(*[V.QubitsTerm(ops, coeff=c) for c, ops in terms])


def _np_dtype(case):
    return np.complex64 if case["dtype"] == "c64" else np.complex128


def _torch_dtype(case):
    return torch.complex64 if case["dtype"] == "c64" else torch.complex128


class _Buffer:
    """A handle's amplitudes for torch (the handle lives as long as the tensor)."""

    def __init__(self, state):
        self.state = state
        self.__cuda_array_interface__ = {
            "shape": (len(state),), "typestr": "<c8" if state.dtype == np.complex64 else "<c16",
            "data": (V.load().vqc_state_device_ptr(state.handle), False), "version": 3, "strides": None}


def _tensor(state):
    return torch.as_tensor(_Buffer(state), device="cuda")


def _real(case, x):
    return np.asarray(x, np.float32 if case["dtype"] == "c64" else np.float64)


def _random_vector(n, seed, dtype):
    """A random normalised state vector on the device, from the seed alone."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    real = torch.float32 if dtype == torch.complex64 else torch.float64
    v = torch.randn((1 << n, 2), generator=g, device=DEV, dtype=real)
    v /= torch.linalg.vector_norm(v, dtype=torch.float64)
    return torch.view_as_complex(v)


def _random_state(case, seed):
    psi = V.StateVector(case["n"], dtype=_np_dtype(case))
    psi.sync()
    _tensor(psi).copy_(_random_vector(case["n"], seed, _torch_dtype(case)))
    torch.cuda.synchronize()
    return psi


def _vqe_items(case, rng):
    if case["ansatz"] == "hea":
        return _hea(case["n"], case["layers"], rng), _operator_terms("tfim", case["n"], rng)
    return _rxyz(case["n"], case["layers"], rng), _operator_terms("xxz", case["n"], rng)


def _serve_items(case, rng):
    """[(qubits, items, terms, gradient wanted)]: the sizes belong to the case, the angles to the seed."""
    pick, out = random.Random(case["wires"]), []
    for i in range(case["count"]):
        n, layers = pick.randint(case["nmin"], case["nmax"]), pick.randint(2, 12)
        out.append((n, _hea(n, layers, rng), _operator_terms("tfim", n, rng), i % 2 == 1))
    return out


def _observe_key(case):
    n = case["n"]
    return (1, n // 2, n)


def prepare(case, seed):
    rng, n, kind = random.Random(seed), case.get("n"), case["kind"]
    dt = _np_dtype(case)
    if kind == "vqe":
        items, terms = _vqe_items(case, rng)
        return {"case": case, "circuit": _circuit(items), "H": _operator(terms), "psi0": V.StateVector(n, dtype=dt)}
    if kind == "circuit":
        items = _u3_cz_toffoli(n, case["layers"], case["wires"], rng)
        return {"case": case, "circuit": _circuit(items), "psi": V.StateVector(n, dtype=dt)}
    if kind == "gates":
        return {"case": case, "gates": list(_circuit(_gate_list(n, case["wires"], rng))),
                "psi": _random_state(case, seed)}
    if kind == "observe":
        return {"case": case, "H": _operator(_operator_terms("xxz", n, rng)), "psi": _random_state(case, seed),
                "phi": _random_state(case, seed + 1), "key": V.QuantumGate(_observe_key(case), _dense(3, (0.3, 0.8)))}
    if kind == "dm":
        items = _u3_cnot(n, case["layers"], rng)
        return {"case": case, "circuit": _circuit(items), "rho": V.DensityMatrix(_random_state(case, seed))}
    if kind == "noisy":
        terms = _operator_terms("tfim", n, rng)
        delta = _dense_operator(terms, n).conj().T.astype(dt)
        return {"case": case, "circuit": _circuit(_noisy(n, case["layers"], rng)), "H": _operator(terms),
                "rho0": V.DensityMatrix(n, dtype=dt), "delta0": V.DensityMatrix(delta, dtype=dt)}
    reqs = [(m, _circuit(items), _operator(terms), g) for m, items, terms, g in _serve_items(case, rng)]
    return {"case": case, "server": Server(dtype=dt), "requests": reqs}


def run(s):
    case = s["case"]
    kind, n = case["kind"], case.get("n")
    if kind == "vqe":
        e, g = V.energy_and_gradient(s["H"], s["circuit"], s["psi0"])
        return {"energy": _real(case, e.real), "grads": _real(case, g)}
    if kind == "circuit":
        s["psi"].reset()
        V.apply(s["circuit"], s["psi"])
        return _tensor(s["psi"])
    if kind == "gates":
        for g in s["gates"]:
            V.apply(g, s["psi"])
        return _tensor(s["psi"])
    if kind == "observe":
        psi, phi, H = s["psi"], s["phi"], s["H"]
        t, k = V.expectation(phi, H, psi), V.expectation(s["key"], psi)
        return {"H": _real(case, V.expectation(H, psi).real), "transition": _real(case, [t.real, t.imag]),
                "key": _real(case, [k.real, k.imag]), "norm": _real(case, psi.norm()),
                "p0": _real(case, V.prob_zero(psi, n // 2)), "Hpsi": _tensor(V.apply_operator(H, psi))}
    if kind == "dm":
        rho = V.apply(s["circuit"], s["rho"])
        reduced = V.partial_tr(rho, list(range(n - case["traced"] + 1, n + 1)))
        return {"rho": _tensor(rho), "reduced": reduced.astype(_np_dtype(case)), "probs": _real(case, V.probabilities(rho))}
    if kind == "noisy":
        rho = V.apply(s["circuit"], s["rho0"].copy())
        e = V.expectation(s["H"], rho)
        delta, g, _ = V.back_propagate(s["delta0"].copy(), s["circuit"], rho)
        return {"energy": _real(case, e.real), "grads": _real(case, g), "delta": _tensor(delta)}
    tickets = [s["server"].submit(m, c, H, want_grad=g) for m, c, H, g in s["requests"]]
    energies, grads = [], []
    for t in tickets:
        e, g, _ = s["server"].wait(t)
        energies.append(e.real)
        if g is not None:
            grads.append(g)
    return {"energies": _real(case, energies), "grads": _real(case, np.concatenate(grads))}


# ----------------------------------------------------------------------------- work
def _apply_flops(items, n):
    """Real operations of one forward pass over 2^n amplitudes: runs of one-qubit
    gates on a wire as one 2x2 (14 per amplitude), a 2x2 behind c controls on
    2^-c of them, phases 6 per amplitude they touch, k-qubit matrices 8 * 2^k."""
    total, last = 0.0, {}
    for name, w, _ in items:
        if name in ("cnot", "x", "swap", "toffoli"):
            per = 0.0
        elif name == "cz":
            per = 0.25
        elif name == "crx":
            per = 14.0 / 2
        elif name == "dense":
            per = 8.0 * (1 << len(w))
        elif name in ("depolarizing", "damping"):
            per = 32.0
        else:
            per = 0.0 if last.get(w[0]) else 14.0
        for q in w:
            last[q] = len(w) == 1 and name not in ("depolarizing", "damping")
        total += per
    return total * 2.0 ** n


def work(case):
    kind, n, rng = case["kind"], case.get("n"), random.Random(0)
    amp = 8 if case["dtype"] == "c64" else 16
    if kind == "vqe":
        items, terms = _vqe_items(case, rng)
        fwd = _apply_flops(items, n)
        nparams = sum(len(a) for _, _, a in items)
        masks = len({tuple(sorted(q for q, p in ops.items() if p != "Z")) for _, ops in terms})
        return {"bytes": amp * 2.0 ** n + 8.0 * nparams, "flops": 3 * fwd + 8.0 * masks * 2.0 ** n}
    if kind == "circuit":
        return {"bytes": amp * 2.0 ** n, "flops": _apply_flops(_u3_cz_toffoli(n, case["layers"], case["wires"], rng), n)}
    if kind == "gates":  # every call reads and writes the amplitudes its gate changes
        share = {"rz": 1, "cnot": 0.5, "cz": 0.25, "crx": 0.5, "swap": 0.5, "toffoli": 0.25}
        items = _gate_list(n, case["wires"], rng)
        return {"bytes": sum(2 * amp * 2.0 ** n * share.get(name, 1) for name, _, _ in items),
                "flops": sum(_apply_flops([it], n) for it in items)}
    if kind == "observe":  # five calls, each reads its states once, H psi is written once
        return {"bytes": amp * 2.0 ** n * (1 + 2 + 1 + 1 + 2 + 2), "flops": 2.0 ** n * (3 * 16.0 * n + 64 + 8)}
    if kind == "dm":
        kept = n - case["traced"]
        return {"bytes": amp * 2 * 4.0 ** n + 16 * 4.0 ** kept + 8 * 2.0 ** n,
                "flops": 2 * _apply_flops(_u3_cnot(n, case["layers"], rng), 2 * n)}
    if kind == "noisy":
        return {"bytes": amp * 4 * 4.0 ** n, "flops": 6 * _apply_flops(_noisy(n, case["layers"], rng), 2 * n)}
    total = {"bytes": 0.0, "flops": 0.0}
    for m, items, terms, g in _serve_items(case, rng):
        fwd = _apply_flops(items, m)
        total["flops"] += (3 if g else 1) * fwd + 8.0 * (m + 1) * 2.0 ** m
        total["bytes"] += 8.0 * (1 + (sum(len(a) for _, _, a in items) if g else 0)) + amp
    return total


# ----------------------------------------------------------------------------- the same in 64 bits, plain torch
def _slices(v, n, wires):
    """Views of v, one for each value of the wires' bits (bit b of the value: wires[b])."""
    order = sorted(wires, reverse=True)
    shape, top = [], n
    for q in order:
        shape += [1 << (top - q), 2]
        top = q - 1
    t = v.view(shape + [1 << top])
    out = []
    for j in range(1 << len(wires)):
        at = [slice(None)] * t.dim()
        for b, q in enumerate(wires):
            at[2 * order.index(q) + 1] = (j >> b) & 1
        out.append(t[tuple(at)])
    return out


def _mix(xs, row):
    acc = None
    for x, u in zip(xs, row):
        if u != 0:
            acc = x * complex(u) if acc is None else acc.add_(x, alpha=complex(u))
    return torch.zeros_like(xs[0]) if acc is None else acc


def _mat(v, n, wires, U):
    """v <- U v on the wires, in place."""
    xs = _slices(v, n, wires)
    eye = np.eye(len(xs))
    rows = [r for r in range(len(xs)) if not np.array_equal(U[r], eye[r])]
    new = [_mix(xs, U[r]) for r in rows]
    for r, y in zip(rows, new):
        xs[r].copy_(y)


def _mat_add(out, v, n, wires, U):
    xs, os_ = _slices(v, n, wires), _slices(out, n, wires)
    for r, o in enumerate(os_):
        for c, x in enumerate(xs):
            if U[r, c] != 0:
                o.add_(x, alpha=complex(U[r, c]))


def _dot(a, b):
    return complex((a.conj() * b).sum())


def _reduced(lam, psi, n, wires):
    """A[a][b] = sum conj(lam_a) psi_b."""
    ls, ps = _slices(lam, n, wires), _slices(psi, n, wires)
    return np.array([[_dot(a, b) for b in ps] for a in ls])


def _keys(terms):
    """One matrix for each set of wires that terms share."""
    keys = {}
    for c, ops in terms:
        M = np.array([[complex(c)]])
        for q in sorted(ops):
            M = np.kron(_PAULI[ops[q]], M)
        w = tuple(sorted(ops))
        keys[w] = keys.get(w, 0) + M
    return keys


def _apply_keys(terms, v, n):
    out = torch.zeros_like(v)
    for w, M in _keys(terms).items():
        _mat_add(out, v, n, w, M)
    return out


def _dense_operator(terms, n):
    M = np.zeros((1 << n, 1 << n), complex)
    idx = np.arange(1 << n)
    for c, ops in terms:
        x, ph = 0, np.full(1 << n, complex(c))
        for q, p in ops.items():
            bit = (idx >> (q - 1)) & 1
            if p != "Z":
                x |= 1 << (q - 1)
            if p != "X":
                ph = ph * (1 - 2.0 * bit) * (1j if p == "Y" else 1)
        M[idx ^ x, idx] += ph
    return M


def _zero(n):
    v = torch.zeros(1 << n, dtype=torch.complex128, device=DEV)
    v[0] = 1
    return v


def _blocks(items):
    """Runs of one-qubit gates on a wire as one block: [(wires, matrix, [derivative of the block])]."""
    blocks, last = [], {}
    for name, w, a in items:
        U, dU = _matrix(name, a, len(w))
        if len(w) == 1 and last.get(w[0]) is not None:
            b = blocks[last[w[0]]]
            b[2] = [U @ d for d in b[2]] + [d @ b[1] for d in dU]
            b[1] = U @ b[1]
        else:
            blocks.append([w, U, list(dU)])
            for q in w:
                last[q] = len(blocks) - 1 if len(w) == 1 else None
    return blocks


def _order_of_parameters(items):
    """Block order -> the order of the items' parameters (a block holds its own in order)."""
    order, last, nblocks, where = [], {}, 0, []
    for name, w, a in items:
        k = len(a)
        if len(w) == 1 and last.get(w[0]) is not None:
            b = last[w[0]]
        else:
            b, nblocks = nblocks, nblocks + 1
            where.append(0)
            for q in w:
                last[q] = b if len(w) == 1 else None
        for _ in range(k):
            order.append((b, where[b]))
            where[b] += 1
    return order


def _exact_gradient(items, terms, n):
    blocks = _blocks(items)
    psi = _zero(n)
    for w, U, _ in blocks:
        _mat(psi, n, w, U)
    lam = _apply_keys(terms, psi, n)
    energy = _dot(psi, lam).real
    grads = [None] * len(blocks)
    for k in range(len(blocks) - 1, -1, -1):
        w, U, dU = blocks[k]
        Ud = U.conj().T
        _mat(psi, n, w, Ud)
        _mat(lam, n, w, Ud)
        if dU:
            A = _reduced(lam, psi, n, w)
            grads[k] = [2 * float(np.sum((Ud @ d) * A).real) for d in dU]
    return energy, np.array([grads[b][i] for b, i in _order_of_parameters(items)])


def _exact_vector(case, seed):
    return _random_vector(case["n"], seed, _torch_dtype(case)).to(torch.complex128)


def _channel(v, n, q, kraus, dagger=False):
    """A one-qubit channel (or its adjoint map) on the 2n-wire vector of a density matrix."""
    S = sum(np.kron(K.conj(), K) for K in kraus)
    _mat(v, 2 * n, (q, q + n), S.conj().T if dagger else S)


def _exact_noisy(case, seed):
    rng, n = random.Random(seed), case["n"]
    terms = _operator_terms("tfim", n, rng)
    items = _noisy(n, case["layers"], rng)

    def forward(v, name, w, a):
        if name in ("depolarizing", "damping"):
            _channel(v, n, w[0], _kraus(name, a[0]))
        else:
            U = _matrix(name, a, len(w))[0]
            _mat(v, 2 * n, w, U)
            _mat(v, 2 * n, tuple(q + n for q in w), U.conj())

    rho, before = _zero(2 * n), []
    for name, w, a in items:
        before.append(rho.clone())
        forward(rho, name, w, a)
    H = torch.from_numpy(_dense_operator(terms, n)).to(DEV)
    energy = complex((H * rho.view(1 << n, 1 << n)).sum())
    # the cotangent's column-major vector: delta[r + 2^n c] = conj(H[c, r])
    delta = H.conj().reshape(-1).clone()
    grads = []
    for (name, w, a), y in zip(reversed(items), reversed(before)):
        if name in ("depolarizing", "damping"):
            _channel(delta, n, w[0], _kraus(name, a[0]), dagger=True)
            continue
        U, dU = _matrix(name, a, len(w))
        wc = tuple(q + n for q in w)
        for d in reversed(dU):
            t = y.clone()
            _mat(t, 2 * n, w, d)
            _mat(t, 2 * n, wc, U.conj())
            grads.append(2 * _dot(delta, t).real)
        _mat(delta, 2 * n, w, U.conj().T)
        _mat(delta, 2 * n, wc, U.T)
    return {"energy": np.float64(energy.real), "grads": np.array(grads[::-1]), "delta": delta}


def exact(case, seed):
    kind, n, rng = case["kind"], case.get("n"), random.Random(seed)
    if kind == "vqe":
        items, terms = _vqe_items(case, rng)
        e, g = _exact_gradient(items, terms, n)
        return {"energy": np.asarray(e), "grads": g}
    if kind == "circuit":
        psi = _zero(n)
        for w, U, _ in _blocks(_u3_cz_toffoli(n, case["layers"], case["wires"], rng)):
            _mat(psi, n, w, U)
        return psi
    if kind == "gates":
        psi = _exact_vector(case, seed)
        for name, w, a in _gate_list(n, case["wires"], rng):
            _mat(psi, n, w, _matrix(name, a, len(w))[0])
        return psi
    if kind == "observe":
        psi, phi = _exact_vector(case, seed), _exact_vector(case, seed + 1)
        Hpsi = _apply_keys(_operator_terms("xxz", n, rng), psi, n)
        t, w = _dot(phi, Hpsi), _observe_key(case)
        mpsi = psi.clone()
        _mat(mpsi, n, w, _dense(3, (0.3, 0.8)))
        k = _dot(psi, mpsi)
        zero = _slices(psi, n, (n // 2,))[0]
        return {"H": np.asarray(_dot(psi, Hpsi).real), "transition": np.array([t.real, t.imag]),
                "key": np.array([k.real, k.imag]), "norm": np.asarray(math.sqrt(_dot(psi, psi).real)),
                "p0": np.asarray(_dot(zero, zero).real), "Hpsi": Hpsi}
    if kind == "dm":
        psi = _exact_vector(case, seed)
        for name, w, a in _u3_cnot(n, case["layers"], rng):
            _mat(psi, n, w, _matrix(name, a, len(w))[0])
        kept = n - case["traced"]
        m = psi.view(1 << case["traced"], 1 << kept)
        reduced = (m.T @ m.conj()).cpu().numpy()
        return {"rho": (psi.conj()[:, None] * psi[None, :]).reshape(-1), "reduced": reduced,
                "probs": (psi.abs() ** 2).cpu().numpy()}
    if kind == "noisy":
        return _exact_noisy(case, seed)
    energies, grads = [], []
    for m, items, terms, g in _serve_items(case, rng):
        e, gr = _exact_gradient(items, terms, m)
        energies.append(e)
        if g:
            grads.append(gr)
    return {"energies": np.array(energies), "grads": np.concatenate(grads)}
