"""Factored fused passes: gates that only move amplitudes are exact, and the
amplitudes may be as large as their type allows, but for the growth the plans
keep below 2^16 (complex64) and 2^48 (complex128).

CPU: tests/factored_steps_check.cpp runs the programs as the engine plans them
in the arithmetic of the state's type.  GPU: plans, subcircuit files and
gradients at the sizes where a tile, a warp or a thread's registers are not
full, one tile and many."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import oracle
from subquokka_dev_b200 import Circuit, Plan, StateVector, adjoint_grad, circuits, make_gate

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "subquokka_dev_b200", "csrc")
SIZES = [1, 2, 3, 5, 9, 10, 11, 12, 13, 15]


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ absent")
def test_steps_compute_the_circuit(tmp_path):
    exe = tmp_path / "factored_steps_check"
    cmd = ["g++", "-O1", "-g", "-std=c++17", "-ffp-contract=off", "-fsanitize=address,undefined",
           "-I", os.path.join(ROOT, "include"), "-I", CSRC, "-I", os.path.join(ROOT, "tests"),
           os.path.join(ROOT, "tests", "factored_steps_check.cpp")]
    cmd += [os.path.join(CSRC, f) for f in ("qk_factor.cpp", "qk_plan.cpp", "qk_rewrite.cpp", "qk_parse.cpp",
                                            "qk_dense_host.cpp")]
    build = subprocess.run(cmd + ["-o", str(exe), "-lpthread"], capture_output=True, text=True)
    assert build.returncode == 0, build.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr


def moving_circuit(n, ngates, seed):
    """X, Y, CX, SWAP (and VSWAP) gates."""
    rng = np.random.default_rng(seed)
    kinds = ["X", "Y"] + (["CX", "SWAP"] if n > 1 else []) + (["VSWAP"] if n > 3 else [])
    gates = []
    for _ in range(ngates):
        k = kinds[rng.integers(len(kinds))]
        q = [int(x) for x in rng.choice(n, min(n, 4), replace=False)]
        if k == "CX":
            gates.append(make_gate("U2", sorted(q[:2]), coeff=circuits.CNOT_BIG_ENDIAN))
        else:
            gates.append(make_gate(k, q if k == "VSWAP" else sorted(q[:2]) if k == "SWAP" else q[:1]))
    return Circuit(gates)


def mixed_circuit(n, ngates, seed):
    """Unitaries, rotations by pi, H, X and Y among phases and CX."""
    rng = np.random.default_rng(seed)
    kinds = ["X", "Y", "H", "U1", "RXPI", "RYPI", "RY"] + (["CP", "CZ", "CX", "RZZ"] if n > 1 else [])
    gates = []
    for _ in range(ngates):
        k = kinds[rng.integers(len(kinds))]
        q = sorted(int(x) for x in rng.choice(n, min(n, 2), replace=False))
        ang = float(rng.uniform(-3, 3))
        if k == "U1":
            gates.append(make_gate(k, q[:1], coeff=circuits.u3_matrix(*rng.uniform(-3, 3, 3))))
        elif k == "CX":
            gates.append(make_gate("U2", q, coeff=circuits.CNOT_BIG_ENDIAN))
        elif k == "CZ":
            gates.append(make_gate("CP", q, np.pi))
        elif k.endswith("PI"):
            gates.append(make_gate(k[:2], q[:1], np.pi))
        else:
            gates.append(make_gate(k, q if k in ("CP", "RZZ") else q[:1], ang))
    return Circuit(gates)


def both_ways(circ, n, dtype, init):
    with StateVector(n, dtype) as sv:
        for run in (lambda: Plan(circ, n, dtype).apply(sv), lambda: sv.apply_groups(circ)):
            sv.upload(init)
            run()
            yield sv.download()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["c128", "c64"])
@pytest.mark.parametrize("n", SIZES)
def test_gates_that_move_amplitudes_are_exact(n, dtype):
    circ = moving_circuit(n, 40, n)
    random = circuits.random_state(n, 5).astype(np.complex64).astype(np.complex128)
    basis = np.zeros(1 << n, dtype=np.complex128)
    basis[(1 << n) // 3] = 1
    for init in (random, basis):
        ref = oracle.apply_circuit(init, n, circ)
        for got in both_ways(circ, n, dtype, init):
            assert np.array_equal(got, ref)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,scale", [("c128", 1.0), ("c128", 1e290), ("c64", 1.0), ("c64", 1e20), ("c64", 1e30)])
@pytest.mark.parametrize("n", SIZES)
def test_large_amplitudes(n, dtype, scale):
    # 120 gates of at most four roundings (2^-53 / 2^-24) of the state's norm
    circ = mixed_circuit(n, 120, 50 + n)
    init = circuits.random_state(n, 6)
    ref = oracle.apply_circuit(init, n, circ)
    tol = 120 * 4 * (2.0 ** -53 if dtype == "c128" else 2.0 ** -24)
    for got in both_ways(circ, n, dtype, init * scale):
        assert np.linalg.norm(got / scale - ref) <= tol


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["c128", "c64"])
@pytest.mark.parametrize("n", [1, 2, 3, 5, 8, 9, 10, 13])
def test_gradients_of_circuits_with_h_and_x(n, dtype):
    # the H constant of the circuit format is 1.1e-11 off a unitary's: its
    # gates scale what is computed on either side of them by 1 + 2.2e-11
    circ = mixed_circuit(n, 60, 70 + n)
    names = {6: "RX", 7: "RY", 8: "RZ"}
    idx, k = [], 0
    for g in circ.gate_list():
        idx.append(k if g.kind in names else -1)
        k += g.kind in names
    rng = np.random.default_rng(n)
    terms = [(float(rng.standard_normal()), 1 << q, 0) for q in range(n)]
    terms += [(float(rng.standard_normal()), 0, (1 << q) | (1 << ((q + 1) % n))) for q in range(n)]
    init = circuits.random_state(n, 3)
    ref = oracle.adjoint_grad(init, n, circ, idx, k, terms)
    # complex64: 60 gates x 4 roundings of 2^-24 on each of the two states
    tol = 2 * n * (60 * 2.2e-11 + (1e-12 if dtype == "c128" else 2 * 60 * 4 * 2.0 ** -24))
    with StateVector(n, dtype) as sv:
        sv.upload(init)
        ev, grad, _ = adjoint_grad(sv, circ, idx, k, terms, 2, True)
        assert abs(ev - ref[0]) <= tol and np.abs(grad - ref[1]).max() <= tol


@pytest.mark.parametrize("n,passes", [(25, 3), (27, 3), (28, 4)])
def test_plans_of_little_work_take_wide_tiles(n, passes):
    # 2048-amplitude tiles with the three lowest qubits: eight more a pass
    circ = Circuit([make_gate("H", [q]) for q in range(n)])
    assert Plan(circ, n, "c128").stats()[0] == passes


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["c128", "c64"])
@pytest.mark.parametrize("n", [17, 18, 19, 20])
def test_tile_shapes_by_size(n, dtype):
    # about the sizes where the shape changes; 200 gates of at most four
    # roundings of the state's norm
    init = circuits.random_state(n, 6)
    tol = 200 * 4 * (2.0 ** -53 if dtype == "c128" else 2.0 ** -24)
    for circ in (Circuit([make_gate(g, [q]) for g in "HX" for q in range(n)]), mixed_circuit(n, 200, n)):
        ref = oracle.apply_circuit(init, n, circ)
        for got in both_ways(circ, n, dtype, init):
            assert np.linalg.norm(got - ref) <= tol
