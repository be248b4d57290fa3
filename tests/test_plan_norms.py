"""The factor that deferred phases leave on the amplitudes in flight, on the CPU.

The planner itself runs (plan_norms.cpp, linked against the engine's library):
over every op of a sweep, in the order the passes run them, the deferred norm
must stay inside the window the planner states for FP32, [1e-12, 1e12] in the
reverse sweep and [1e-18, 1e18] in the forward one.  The families are those that leave it when the gates are walked in any other order:
qubits that meet in small blocks only, so that one stage runs all their layers,
and rotations next to pi, whose diagonal is tiny.
"""
import os
import shutil
import subprocess

import pytest

from vqcb200 import _build, _lib

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def plan_norms(tmp_path_factory):
    if shutil.which(_build.NVCC) is None:
        pytest.skip("no nvcc")
    _lib.load()
    exe = str(tmp_path_factory.mktemp("plan") / "plan_norms")
    lib = os.path.dirname(_build.LIB)
    cmd = [_build.NVCC] + _build.ARCH + ["-O1", "-std=c++17", "--expt-relaxed-constexpr", "-x", "cu",
                                         "-I", _build.INCLUDE, "-I", _build.CSRC, os.path.join(HERE, "plan_norms.cpp"),
                                         "-o", exe, "-L", lib, "-lvqcb200", "-Xlinker", "-rpath=" + lib]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return exe


@pytest.mark.parametrize("family,n,layers", [("blocks2", 18, 20), ("blocks2", 18, 80), ("blocks3", 19, 40),
                                             ("pi", 18, 8), ("pi", 24, 8), ("u3", 21, 30)])
def test_norm_stays_in_the_window(plan_norms, family, n, layers):
    for seed in range(8):
        r = subprocess.run([plan_norms, family, str(n), str(layers), str(seed)], capture_output=True, text=True)
        if r.returncode == 3:
            pytest.skip("no run-time compiler: nothing is deferred")
        assert r.returncode == 0, r.stderr
        fwd_lo, fwd_hi, lo, hi, rows, _ = r.stdout.split()
        assert 1e-18 <= float(fwd_lo) < 1 and float(fwd_hi) <= 1e18
        assert 1e-12 <= float(lo) < 1 and float(hi) <= 1e12
        assert family == "u3" or int(rows) > 0


@pytest.mark.parametrize("family,n,layers,seeds", [("u3", 18, 8, 40), ("u3", 20, 4, 20), ("blocks2", 18, 6, 20)])
def test_angles_do_not_change_the_structure(plan_norms, family, n, layers, seeds):
    """Compiled passes are reused for new angles, those with a tiny diagonal included."""
    found = set()
    for seed in range(seeds):
        r = subprocess.run([plan_norms, family, str(n), str(layers), str(seed)], capture_output=True, text=True)
        if r.returncode == 3:
            pytest.skip("no run-time compiler: nothing is deferred")
        found.add(r.stdout.split()[5])
    assert len(found) == 1
