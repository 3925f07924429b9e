"""Sums of Pauli strings by tiles (k_pauli_tile): strings of X, Y and Z whose
X masks fit a tile, do not fit one, share one, or are more than one launch
takes, on states smaller than a warp, a thread block and a tile, and larger."""
import numpy as np
import pytest

import oracle
from subquokka_dev_b200 import Circuit, StateVector, adjoint_grad, circuits, expval, make_gate

pytestmark = pytest.mark.gpu


def random_terms(n, kind, seed):
    rng = np.random.default_rng(seed)
    full = (1 << n) - 1
    if kind == "chain":      # Z Z and X, as the variational Hamiltonians
        t = [(1 << i, 0) for i in range(n)] + [(0, (1 << i) | (1 << ((i + 1) % n))) for i in range(n)]
    elif kind == "dense":    # any string: X masks too wide for a tile among them
        t = [(int(rng.integers(1 << n)), int(rng.integers(1 << n))) for _ in range(30)] + [(full, 0), (full, full), (0, 0)]
    else:                    # one X mask with many Z masks, and many X masks
        t = [(1, int(rng.integers(1 << n))) for _ in range(150)] + [(int(x) & full, 0) for x in range(60)]
    return [(float(rng.standard_normal()), x, z) for x, z in t]


@pytest.mark.parametrize("kind", ["chain", "dense", "many"])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 6, 8, 10, 11, 12, 14, 16])
def test_expval_matches_oracle(n, kind):
    terms = random_terms(n, kind, n)
    state = circuits.random_state(n, 5)
    scale = sum(abs(c) for c, _, _ in terms)
    ref = oracle.pauli_expval(state, n, terms)
    for dtype, tol in (("c128", 1e-13), ("c64", 2.0 ** -22)):   # a rounded state: 2 x 2^-24 a product
        with StateVector(n, dtype) as sv:
            sv.upload(state)
            assert abs(expval(sv, terms) - ref) <= tol * scale, dtype


@pytest.mark.parametrize("kind", ["chain", "dense", "many"])
@pytest.mark.parametrize("n", [3, 10, 13])
def test_adjoint_matches_oracle(n, kind):
    terms = random_terms(n, kind, 40 + n)
    scale = sum(abs(c) for c, _, _ in terms)
    rng = np.random.default_rng(n)
    circ = Circuit([make_gate(g, [q], float(rng.uniform(-3, 3))) for q in range(n) for g in ("RY", "RZ", "RX")])
    idx = list(range(circ.ngates))
    init = circuits.random_state(n, 6)
    ev, grad = oracle.adjoint_grad(init, n, circ, idx, len(idx), terms)
    for fused in (False, True):
        with StateVector(n, "c128") as sv:
            sv.upload(init)
            e, g, _ = adjoint_grad(sv, circ, idx, len(idx), terms, 0, fused)
            assert abs(e - ev) <= 1e-13 * scale and np.abs(g - grad).max() <= 1e-13 * scale
