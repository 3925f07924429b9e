"""A run of diagonal gates leaves bit for bit what the gates leave one by one."""
import numpy as np
import pytest

from subquokka_dev_b200 import Circuit, StateVector, circuits, make_gate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["c128", "c64"])
@pytest.mark.parametrize("common", [False, True])
@pytest.mark.parametrize("n", [1, 2, 5, 9, 11, 14])
def test_runs_equal_single_gates(n, common, dtype):
    rng = np.random.default_rng(n)
    init = circuits.random_state(n, 4)
    for ngates in (2, 32, 33, 70):
        gates = []
        for _ in range(ngates):
            kind = ["Z", "P", "RZ", "CP", "RZZ", "U2"][rng.integers(6 if n > 1 else 3)]
            if common:
                kind = "CP" if n > 1 and rng.integers(4) else "P"
            q = [n // 2] if common else [int(rng.integers(n))]
            if kind in ("CP", "RZZ", "U2"):
                q = sorted(q + [int((q[0] + 1 + rng.integers(n - 1)) % n)])
            diagonal = np.diag(np.exp(1j * rng.uniform(-3, 3, 4)))
            gates.append(make_gate(kind, q, float(rng.uniform(-3, 3)), diagonal if kind == "U2" else None))
        with StateVector(n, dtype) as a, StateVector(n, dtype) as b:
            a.upload(init)
            b.upload(init)
            a.apply(Circuit(gates))
            for g in gates:
                b.apply(Circuit([g]))
            assert np.array_equal(a.download().view(np.uint64), b.download().view(np.uint64))
