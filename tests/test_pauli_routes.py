"""Pauli sums where their route changes: one group of strings on states about
the sizes where it has a sweep of its own or a tile, and groups that share a
tile."""
import numpy as np
import pytest

import oracle
from subquokka_dev_b200 import StateVector, circuits, expval

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
