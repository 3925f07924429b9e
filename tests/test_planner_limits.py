"""Planner calls that have no plan end with an error, and soon; planning time
(CPU)."""
import os
import shutil
import subprocess
import sys

import numpy as np
import pytest

from subquokka_dev_b200 import Circuit, Plan, make_gate

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("dtype", ["c128", "c64"])
@pytest.mark.parametrize("gates", [
    'make_gate("RY", [0], 0.3), make_gate("SWAP", [0, 2])',                                # factored programs
    'make_gate("RY", [0], 0.3), make_gate("U2", [0, 2], 0.0, np.linalg.qr(m)[0])',         # general programs
])
def test_two_tile_qubits_in_a_one_qubit_tile_is_an_error(dtype, gates):
    # in a child with a limit: a planner that makes no progress does not return
    code = f"""
import resource
resource.setrlimit(resource.RLIMIT_AS, (8 << 30, 8 << 30))
import numpy as np
from subquokka_dev_b200 import Circuit, Plan, make_gate
m = np.random.default_rng(1).standard_normal((4, 4))
try:
    Plan(Circuit([{gates}]), 3, "{dtype}", tile_bits=1, reg_bits=1)
except Exception as e:
    print(type(e).__name__, e)
"""
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and "QK_ERR_ARG" in r.stdout and "needs 2 tile qubits" in r.stdout, r.stdout + r.stderr


def test_one_qubit_tiles_take_what_needs_one():
    cnot = np.eye(4)[[0, 1, 3, 2]]
    c = Circuit([make_gate("RY", [0], 0.3), make_gate("CP", [0, 1], 0.4), make_gate("U2", [0, 2], 0.0, cnot)])
    for dtype in ("c128", "c64"):
        assert Plan(c, 3, dtype, tile_bits=1, reg_bits=1).stats()[0] >= 1


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ absent")
@pytest.mark.parametrize("check,opt", [("alloc_check", "-O1"), ("plan_time_check", "-O2")])
def test_planner_check(check, opt, tmp_path):
    csrc = os.path.join(ROOT, "subquokka_dev_b200", "csrc")
    exe = tmp_path / check
    cmd = ["g++", opt, "-std=c++17", "-I", os.path.join(ROOT, "include"), "-I", csrc, "-I", os.path.join(ROOT, "tests"),
           os.path.join(ROOT, "tests", check + ".cpp")]
    cmd += [os.path.join(csrc, f) for f in ("qk_factor.cpp", "qk_plan.cpp", "qk_rewrite.cpp", "qk_parse.cpp", "qk_dense_host.cpp")]
    build = subprocess.run(cmd + ["-o", str(exe), "-lpthread"], capture_output=True, text=True)
    assert build.returncode == 0, build.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
