"""Runs of diagonal gates on the per-gate path (k_diag_run): one sweep for up
to 32 consecutive Z, P, RZ, CP and RZZ gates, with and without a qubit common
to all, across the bounds of runs and windows, on states smaller than a block
and larger, against the oracle and against the gates applied one by one."""
import numpy as np
import pytest

import oracle
from subquokka_dev_b200 import Circuit, QkError, StateVector, circuits, make_gate

pytestmark = pytest.mark.gpu


def diagonal_circuit(n, ngates, seed, common):
    rng = np.random.default_rng(seed)
    gates = []
    for _ in range(ngates):
        kind = ["Z", "P", "RZ", "CP", "RZZ"][rng.integers(5 if n > 1 else 3)]
        q = sorted(int(x) for x in rng.choice(n, 2, replace=False)) if n > 1 else [0]
        if common:   # phases that all act where qubit n // 2 is 1
            kind = "CP" if n > 1 and rng.integers(4) else "P"
            c = n // 2
            q = sorted([c, int((c + 1 + rng.integers(n - 1)) % n)]) if kind == "CP" else [c]
        gates.append(make_gate(kind, q if kind in ("CP", "RZZ") else q[:1], float(rng.uniform(-3, 3))))
    return gates


@pytest.mark.parametrize("dtype", ["c128", "c64"])
@pytest.mark.parametrize("common", [False, True])
@pytest.mark.parametrize("n", [1, 2, 3, 5, 6, 9, 11, 13])
def test_runs_match_oracle_and_single_gates(n, common, dtype):
    tol = {"c128": 1e-13, "c64": 70 * 2.0 ** -23}[dtype]   # one rounded product a gate
    init = circuits.random_state(n, 4)
    for ngates in (2, 31, 32, 33, 70):
        gates = diagonal_circuit(n, ngates, 7 * n + ngates, common)
        gates.insert(ngates // 2, make_gate("H", [n - 1]))   # two runs
        circ = Circuit(gates)
        with StateVector(n, dtype) as a, StateVector(n, dtype) as b, StateVector(n, dtype) as c:
            for sv in (a, b, c):
                sv.upload(init)
            a.apply(circ)
            for g in gates:
                b.apply(Circuit([g]))
            with c.capture(circ) as graph:
                graph.launch()
            got = a.download()
            assert np.abs(got - oracle.apply_circuit(init, n, circ)).max() <= tol
            assert np.abs(got - b.download()).max() <= tol
            assert np.array_equal(got, c.download())


def test_gates_before_one_in_error_are_applied():
    n = 6
    init = circuits.random_state(n, 9)
    good = diagonal_circuit(n, 5, 1, False)
    bad = make_gate("Z", [n])
    with StateVector(n) as sv:
        sv.upload(init)
        with pytest.raises(QkError):
            sv.apply(Circuit(good + [bad] + good))
        assert np.abs(sv.download() - oracle.apply_circuit(init, n, Circuit(good))).max() <= 1e-13
