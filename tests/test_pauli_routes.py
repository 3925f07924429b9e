"""Pauli sums where their route changes: one group of strings on states about
the sizes where it has a sweep of its own or a tile, and groups that share a
tile."""
import numpy as np
import pytest

import oracle
from subquokka_dev_b200 import Circuit, StateVector, adjoint_grad, circuits, expval, last_sweep, make_gate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nterms", [1, 2, 8, 9, 64, 65])
@pytest.mark.parametrize("n", [1, 5, 16, 17, 18, 20, 21, 22])
def test_one_group(n, nterms):
    rng = np.random.default_rng(100 * n + nterms)
    state = circuits.random_state(n, 5)
    for x in (0, 1 << (n - 1), (1 << min(n, 10)) - 1):
        terms = [(float(rng.standard_normal()), x, int(rng.integers(1 << n))) for _ in range(nterms)]
        scale = sum(abs(c) for c, _, _ in terms)
        ref = oracle.pauli_expval(state, n, terms)
        # sums of 2^n products of a state of norm 1; complex64: a rounded state, 2 x 2^-24 a product
        for dtype, tol in (("c128", 1e-13), ("c64", 2.0 ** -22)):
            with StateVector(n, dtype) as sv:
                sv.upload(state)
                assert abs(expval(sv, terms) - ref) <= tol * scale, dtype


@pytest.mark.parametrize("dtype", ["c128", "c64"])
def test_sweep_bytes_count_every_reduction(dtype):
    # H = sum Z Z + sum X on 14 qubits: tiles of 1024 amplitudes with the
    # lowest qubits; <H> comes with them in complex128 unless a mask is too
    # wide for a tile, in complex64 it is a sweep of its own
    n = 14
    circ, _, J, h = circuits.hea(n, 2, 3)
    idx = [-1] * circ.ngates
    S = float((16 if dtype == "c128" else 8) << n)
    chain = [(float(c), 1 << q, 0) for q, c in enumerate(h)] + [(float(c), 0, 3 << q) for q, c in enumerate(J)]
    tiles = 2   # 7 and 6 of the 14 X masks beside the low three (four) qubits' ones
    for terms, sums, dot in ((chain, tiles, dtype == "c64"), (chain + [(0.5, (1 << n) - 1, 0)], tiles + 1, True),
                             ([], 0, False)):
        with StateVector(n, dtype) as sv:
            adjoint_grad(sv, circ, idx, 0, terms, 2, True)
            st = last_sweep(sv)
        rest = st["alg_bytes"] - 2 * S * st["forward_passes"] - 4 * S * st["backward_passes"] - 2 * 6 * S
        assert rest == (2 * S + 3 * S * (sums - 1) + (2 * S if dot else 0) if sums else S)


def kinds(n, kind, seed):
    rng = np.random.default_rng(seed)
    full = (1 << n) - 1
    if kind == "chain":
        t = [(1 << i, 0) for i in range(n)] + [(0, (1 << i) | (1 << ((i + 1) % n))) for i in range(n)]
    elif kind == "wide":   # masks that fit no tile among others
        t = [(int(rng.integers(1 << n)), int(rng.integers(1 << n))) for _ in range(20)] + [(full, 0), (full, full), (0, 0)]
    else:                  # several launches, groups of many terms
        t = [(1, int(rng.integers(1 << n))) for _ in range(100)] + [(int(x) & full, 0) for x in range(40)]
    return [(float(rng.standard_normal()), x, z) for x, z in t]


@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("kind", ["chain", "wide", "many"])
@pytest.mark.parametrize("n", [3, 10, 13])
def test_complex64_gradient_matches_oracle(n, kind, fused):
    # both states take 3 n gates of at most four roundings of 2^-24, and H psi
    # one for each X mask
    terms = kinds(n, kind, 60 + n)
    scale = sum(abs(c) for c, _, _ in terms)
    masks = len({x for _, x, _ in terms})
    rng = np.random.default_rng(n)
    circ = Circuit([make_gate(g, [q], float(rng.uniform(-3, 3))) for q in range(n) for g in ("RY", "RZ", "RX")])
    idx = list(range(circ.ngates))
    init = circuits.random_state(n, 6)
    ev, grad = oracle.adjoint_grad(init, n, circ, idx, len(idx), terms)
    tol = scale * 2.0 ** -24 * (2 * 4 * 3 * n + masks)
    with StateVector(n, "c64") as sv:
        sv.upload(init)
        e, g, _ = adjoint_grad(sv, circ, idx, len(idx), terms, 0, fused)
        assert abs(e - ev) <= tol and np.abs(g - grad).max() <= tol


@pytest.mark.parametrize("n,layers", [(14, 4), (20, 3)])
def test_complex64_gradient_of_an_ansatz(n, layers):
    # many tiles a thread block; against the complex128 sweep
    circ, _, J, h = circuits.hea(n, layers, 5)
    rotations = [g.kind in (7, 8) for g in circ.gate_list()]
    idx = list(np.cumsum(rotations) - 1)
    idx = [int(k) if r else -1 for k, r in zip(idx, rotations)]
    terms = [(float(c), 1 << q, 0) for q, c in enumerate(h)] + [(float(c), 0, 3 << q) for q, c in enumerate(J)]
    got = {}
    for dtype in ("c128", "c64"):
        with StateVector(n, dtype) as sv:
            got[dtype] = adjoint_grad(sv, circ, idx, sum(rotations), terms, 2, True)
    tol = sum(abs(c) for c, _, _ in terms) * 2.0 ** -24 * (2 * 4 * circ.ngates + n + 1)
    assert abs(got["c64"][0] - got["c128"][0]) <= tol
    assert np.abs(got["c64"][1] - got["c128"][1]).max() <= tol
