"""Factored fused passes (qk_factor.cpp, qk_fpass.cu).

CPU: tests/factored_check.cpp runs factored programs by an emulator of their
steps.  GPU: plans, subcircuit files and adjoint sweeps of random circuits in
the factored gate set against the FP64 oracle, at the sizes where a tile, a
warp or a thread's registers are not full, one tile and many, and at every
tile and register shape a plan can be asked for."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import oracle
from subquokka_dev_b200 import Circuit, Plan, StateVector, adjoint_grad, circuits, make_gate

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "subquokka_dev_b200", "csrc")
CNOT = circuits.CNOT_BIG_ENDIAN


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ absent")
def test_factored_programs_compute_the_circuit(tmp_path):
    exe = tmp_path / "factored_check"
    cmd = ["g++", "-O1", "-g", "-std=c++17", "-fsanitize=address,undefined", "-fno-omit-frame-pointer",
           "-I", os.path.join(ROOT, "include"), "-I", CSRC, "-I", os.path.join(ROOT, "tests"),
           os.path.join(ROOT, "tests", "factored_check.cpp")]
    cmd += [os.path.join(CSRC, f) for f in ("qk_factor.cpp", "qk_plan.cpp", "qk_rewrite.cpp", "qk_parse.cpp",
                                            "qk_dense_host.cpp")]
    build = subprocess.run(cmd + ["-o", str(exe)], capture_output=True, text=True)
    assert build.returncode == 0, build.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr


def random_circuit(n, ngates, seed, adjoint=False):
    """Gates of every factored kind; with adjoint no H (its constant is no
    unitary) and no VSWAP."""
    rng = np.random.default_rng(seed)
    one = ["X", "Y", "Z", "P", "RX", "RY", "RZ", "U1"] + ([] if adjoint else ["H"])
    two = ["CP", "CZ", "RZZ", "SWAP", "CX"] + ([] if adjoint or n < 4 else ["VSWAP"])
    gates = []
    for _ in range(ngates):
        kind = one[rng.integers(len(one))] if n < 2 or rng.integers(2) else two[rng.integers(len(two))]
        ang = float(rng.uniform(-np.pi, np.pi))
        q = sorted(int(x) for x in rng.choice(n, 2, replace=False)) if n > 1 else [0]
        if kind == "U1":
            gates.append(make_gate("U1", q[:1], coeff=circuits.u3_matrix(*rng.uniform(-np.pi, np.pi, 3))))
        elif kind == "CZ":
            gates.append(make_gate("CP", q, np.pi))
        elif kind == "CX":
            gates.append(make_gate("U2", q, coeff=CNOT))
        elif kind == "VSWAP":
            gates.append(make_gate("VSWAP", [int(x) for x in rng.choice(n, 4, replace=False)]))
        else:
            gates.append(make_gate(kind, q if kind in two else [int(rng.integers(n))], ang))
    return Circuit(gates)


# complex128: 60 gates of a few roundings of 2^-53; complex64: 60 gates of at
# most three roundings of 2^-24 each relative to the state's norm
TOL = {"c128": 1e-12, "c64": 1.1e-5}


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["c128", "c64"])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 7, 9, 10, 11, 12, 13, 15])
def test_plan_and_groups_match_oracle(n, dtype):
    for seed in (n, 100 + n):
        circ = random_circuit(n, 60, seed)
        init = circuits.random_state(n, seed)
        ref = oracle.apply_circuit(init, n, circ)
        with StateVector(n, dtype) as sv:
            for run in (lambda: Plan(circ, n, dtype).apply(sv), lambda: sv.apply_groups(circ)):
                sv.upload(init)
                run()
                assert np.abs(sv.download() - ref).max() <= TOL[dtype]


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,tile,reg", [(d, t, r) for d in ("c128", "c64") for t in (2, 3, 4, 6, 9, 12, 13, 14)
                                            for r in (0, 2, 3, 4) if max(r, 2) <= t])
def test_tile_shapes_match_oracle(dtype, tile, reg):
    n = 14
    if tile - (reg or 4) > (8 if dtype == "c128" and (reg or 4) == 4 else 9) or (dtype == "c128" and tile > 13):
        pytest.skip("refused shape")
    if tile < (reg or 4):
        pytest.skip("fewer tile bits than register bits")
    circ = random_circuit(n, 60, 7)
    init = circuits.random_state(n, 8)
    ref = oracle.apply_circuit(init, n, circ)
    with StateVector(n, dtype) as sv:
        sv.upload(init)
        Plan(circ, n, dtype, tile_bits=tile, reg_bits=reg).apply(sv)
        assert np.abs(sv.download() - ref).max() <= TOL[dtype]


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 3, 5, 8, 9, 10, 13])
def test_adjoint_matches_oracle(n):
    # random rotations (every one trainable) among fixed gates; the gradient
    # sums products of 2^n amplitudes of norm 1: 1e-12 a term of H
    circ = random_circuit(n, 50, 20 + n, adjoint=True)
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
    with StateVector(n, "c128") as sv:
        sv.upload(init)
        ev, grad, _ = adjoint_grad(sv, circ, idx, k, terms, 2, True)
        assert abs(ev - ref[0]) <= 1e-12 * 2 * n and np.abs(grad - ref[1]).max() <= 1e-12 * 2 * n
        assert np.abs(sv.download() - init).max() <= 1e-12
