"""The work this engine is used for, as a set of measured cases.

Each case is one call (or one training step) through the package's public
entry points: the per-gate path on a flat circuit, fused plans in both
precisions, tensor-core blocks, a subcircuit file, observables, adjoint
gradients, a batch of variational circuits.  The circuits are the ones the
package's benchmark and tests use: the QFT, bricks of U3 and CZ, and the
hardware-efficient ansatz with H = sum J_i Z_i Z_{i+1} + sum h_i X_i.
"""
import math

import numpy as np
import torch

import subquokka_dev_b200 as sq
from subquokka_dev_b200.torch_shim import ParamCircuit, expectation

H_CONST = 0.70710678118  # the H gate's constant in the circuit format
CNOT = [[1, 0, 0, 0], [0, 1, 0, 0], [0, 0, 0, 1], [0, 0, 1, 0]]


def listed():
    return [
        # a 20-qubit QFT on a random state, gate by gate: a state that lives in
        # L2, where a launch costs about as much as a sweep
        {"name": "qft20_gates_c128", "kind": "gates", "circuit": "qft", "n": 20, "layers": 1, "dtype": "c128"},
        # a brick circuit from |0...0>, gate by gate, on a state far larger than L2
        {"name": "brick28_gates_c128", "kind": "gates", "circuit": "brick", "n": 28, "layers": 20, "dtype": "c128"},
        # the same family as a fused plan that is kept and applied again
        {"name": "brick28_plan_c128", "kind": "plan", "circuit": "brick", "n": 28, "layers": 20, "dtype": "c128", "width": 0},
        # a single-precision fused plan
        {"name": "brick29_plan_c64", "kind": "plan", "circuit": "brick", "n": 29, "layers": 20, "dtype": "c64", "width": 0},
        # six-qubit unitaries on the tensor cores, single precision
        {"name": "brick28_blocks6_c64", "kind": "plan", "circuit": "brick", "n": 28, "layers": 24, "dtype": "c64", "width": 6},
        # five-qubit unitaries on the tensor cores, double precision
        {"name": "brick25_blocks5_c128", "kind": "plan", "circuit": "brick", "n": 25, "layers": 12, "dtype": "c128", "width": 5},
        # a subcircuit file (12-qubit chunks) of the QFT, run as the file's runner does: planned on each call
        {"name": "qft27_groups_c128", "kind": "groups", "circuit": "qft", "n": 27, "layers": 1, "dtype": "c128", "chunk": 12},
        # <H> and its gradient, one training step: a large ansatz ...
        {"name": "hea26_grad_c128", "kind": "grad", "n": 26, "layers": 12, "dtype": "c128"},
        # ... a mid-sized one in single precision ...
        {"name": "hea23_grad_c64", "kind": "grad", "n": 23, "layers": 10, "dtype": "c64"},
        # ... and a small one, where the step's host work and launches count
        {"name": "hea13_grad_c128", "kind": "grad", "n": 13, "layers": 5, "dtype": "c128"},
        # many small variational circuits of uneven size, one training step of all
        {"name": "batch40_c64", "kind": "batch", "circuits": 40, "nmin": 14, "nmax": 20, "lmin": 4, "lmax": 12, "dtype": "c64"},
        # an energy on a state that is already there
        {"name": "energy27_c128", "kind": "energy", "n": 27, "dtype": "c128"},
    ]


def draw(rng):
    kind = rng.choice(["gates", "plan", "plan", "blocks", "groups", "grad", "grad", "batch", "energy"])
    dtype = rng.choice(["c128", "c64"])
    circuit = rng.choice(["qft", "brick"])
    if kind == "gates":
        return {"kind": "gates", "circuit": circuit, "n": rng.randint(10, 27), "dtype": dtype,
                "layers": 1 if circuit == "qft" else rng.randint(2, 20)}
    if kind == "plan":
        return {"kind": "plan", "circuit": circuit, "n": rng.randint(10, 28), "dtype": dtype, "width": 0,
                "layers": 1 if circuit == "qft" else rng.randint(2, 20)}
    if kind == "blocks":
        return {"kind": "plan", "circuit": "brick", "n": rng.randint(13, 27), "dtype": dtype,
                "width": rng.choice([5, 6]), "layers": rng.randint(2, 20)}
    if kind == "groups":
        return {"kind": "groups", "circuit": circuit, "n": rng.randint(14, 27), "dtype": dtype,
                "layers": 1 if circuit == "qft" else rng.randint(2, 12), "chunk": rng.choice([8, 10, 12])}
    if kind == "grad":
        return {"kind": "grad", "n": rng.randint(8, 25), "layers": rng.randint(2, 12), "dtype": dtype}
    if kind == "batch":
        lo, la = rng.randint(10, 14), rng.randint(2, 5)
        return {"kind": "batch", "circuits": rng.randint(8, 40), "nmin": lo, "nmax": lo + rng.randint(0, 5),
                "lmin": la, "lmax": la + rng.randint(0, 7), "dtype": dtype}
    return {"kind": "energy", "n": rng.randint(16, 27), "dtype": dtype}


# ---- circuits ---------------------------------------------------------------

def u3(theta, phi, lam):
    c, s = math.cos(theta / 2), math.sin(theta / 2)
    return np.array([[c, -np.exp(1j * lam) * s], [np.exp(1j * phi) * s, np.exp(1j * (phi + lam)) * c]])


def gate_list(case, seed):
    """[(name, qubits, angle or matrix)] of a case's circuit."""
    n, out = case["n"], []
    if case["circuit"] == "qft":
        for i in range(n):
            out.append(("H", [i], 0.0))
            out += [("CP", [i, j], math.pi / 2 ** (j - i)) for j in range(i + 1, n)]
        return out + [("SWAP", [i, n - 1 - i], 0.0) for i in range(n // 2)]
    ang = np.random.default_rng(seed).uniform(0.0, 2 * math.pi, size=(case["layers"], n, 3))
    for layer in range(case["layers"]):
        out += [("U1", [q], u3(*ang[layer, q])) for q in range(n)]
        out += [("CP", [a, a + 1], math.pi) for a in range(layer % 2, n - 1, 2)]
    return out


def circuit_of(gates):
    return sq.Circuit([sq.make_gate(g, q, 0.0, v) if g == "U1" else sq.make_gate(g, q, v) for g, q, v in gates])


def ansatz(n, layers):
    pc = ParamCircuit(n)
    for _ in range(layers):
        for q in range(n):
            pc.rot("RY", q, pc.param())
            pc.rot("RZ", q, pc.param())
        for q in range(n - 1):
            pc.fixed("U2", [q, q + 1], coeff=np.array(CNOT, dtype=np.complex128))
    return pc


def variational(n, layers, rng):
    """(angles, J, h) of one ansatz and its Hamiltonian."""
    return rng.uniform(-math.pi, math.pi, 2 * n * layers), rng.standard_normal(n - 1), rng.standard_normal(n)


def batch_sizes(case, rng):
    return [(int(rng.integers(case["nmin"], case["nmax"] + 1)), int(rng.integers(case["lmin"], case["lmax"] + 1)))
            for _ in range(case["circuits"])]


# ---- states -----------------------------------------------------------------

def random_amplitudes(n, seed):
    """A normalised complex128 state, re and im i.i.d. N(0, 1) before it."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    a = torch.view_as_complex(torch.randn(1 << n, 2, dtype=torch.float64, device="cuda", generator=g))
    return a.div_(torch.linalg.vector_norm(a))


def product_qubits(n, seed):
    """One (cos, sin e^{i phi}) pair a qubit: a state whose energy is far from 0."""
    rng = np.random.default_rng(seed)
    th, ph = rng.uniform(0.2, 1.3, n), rng.uniform(-0.6, 0.6, n)
    return np.stack([np.cos(th), np.sin(th) * np.exp(1j * ph)], 1)


def product_amplitudes(qubits):
    a = torch.ones(1, dtype=torch.complex128, device="cuda")
    for v in qubits:
        a = torch.kron(torch.as_tensor(v, device="cuda"), a)
    return a


def prepare(case, seed):
    kind = case["kind"]
    if kind == "grad":
        rng = np.random.default_rng(seed)
        p, J, h = variational(case["n"], case["layers"], rng)
        theta = torch.tensor(p, dtype=torch.float64, requires_grad=True)
        return {"kind": kind, "pc": ansatz(case["n"], case["layers"]), "theta": theta, "dtype": case["dtype"],
                "terms": sq.zz_x_hamiltonian(case["n"], J, h)}
    if kind == "batch":
        rng = np.random.default_rng(seed)
        items = []
        for n, layers in batch_sizes(case, np.random.default_rng(case["circuits"])):
            p, J, h = variational(n, layers, rng)
            items.append((ansatz(n, layers), p, sq.zz_x_hamiltonian(n, J, h)))
        return {"kind": kind, "batch": sq.Batch(items, case["dtype"]), "params": [p for _, p, _ in items]}
    n = case["n"]
    sv = sq.StateVector(n, case["dtype"])
    if kind == "energy":
        sv.as_torch().copy_(product_amplitudes(product_qubits(n, seed)))
        _, J, h = variational(n, 0, np.random.default_rng(seed + 1))
        return {"kind": kind, "sv": sv, "terms": sq.zz_x_hamiltonian(n, J, h)}
    if case["circuit"] == "qft":
        sv.as_torch().copy_(random_amplitudes(n, seed))
    circuit = circuit_of(gate_list(case, seed))
    state = {"kind": kind, "sv": sv, "circuit": circuit, "out": sv.as_torch()}
    if kind == "plan":
        state["plan"] = sq.Plan(circuit, n, case["dtype"], fuse_width=case["width"])
    if kind == "groups":
        state["circuit"] = sq.chunk_groups(circuit, n, case["chunk"])
    return state


def run(state):
    kind = state["kind"]
    if kind == "grad":
        theta = state["theta"]
        theta.grad = None
        loss = expectation(theta, state["pc"], state["terms"], dtype=state["dtype"])
        loss.backward()
        return {"loss": loss.detach(), "grad": theta.grad}
    if kind == "batch":
        state["batch"].set_params(state["params"])
        ev, grads, _ = state["batch"].run()
        return {"energies": ev, "grads": np.concatenate(grads)}
    if kind == "energy":
        return np.float64(sq.expval(state["sv"], state["terms"]))
    if kind == "gates":
        state["sv"].apply(state["circuit"])
    elif kind == "groups":
        state["sv"].apply_groups(state["circuit"])
    else:
        state["plan"].apply(state["sv"])
    return state["out"]


def work(case):
    """The state read and written once (twice each way for a gradient), and
    the circuit's arithmetic: 14 operations an amplitude for a dense
    one-qubit gate, 4 for a Hadamard, 1.5 for a controlled phase, 0.5 for CZ."""
    kind = case["kind"]
    size = 16 if case["dtype"] == "c128" else 8
    if kind == "batch":
        shapes = batch_sizes(case, np.random.default_rng(case["circuits"]))
    elif kind == "grad":
        shapes = [(case["n"], case["layers"])]
    elif kind == "energy":
        return {"bytes": size << case["n"], "flops": (6 * case["n"]) << case["n"]}
    else:
        n = case["n"]
        if case["circuit"] == "qft":
            ops = 4 * n + 1.5 * n * (n - 1) / 2
        else:
            ops = case["layers"] * (14 * n + 0.5 * (n - 1) / 2)
        return {"bytes": 2 * size << n, "flops": ops * 2.0 ** n}
    # forward once, backward on two states, a dot product a parameter pair
    return {"bytes": sum(4 * size << n for n, _ in shapes),
            "flops": sum((3 * 14 + 12) * n * layers * 2.0 ** n for n, layers in shapes)}


# ---- the same in plain torch, 64 bits ---------------------------------------

def apply1(a, q, m):
    v = a.view(-1, 2, 1 << q)
    x, y = v[:, 0].clone(), v[:, 1].clone()
    v[:, 0] = complex(m[0][0]) * x + complex(m[0][1]) * y
    v[:, 1] = complex(m[1][0]) * x + complex(m[1][1]) * y


def quarters(a, p, q):
    """View [rest, bit max, rest, bit min, rest] of a state."""
    lo, hi = min(p, q), max(p, q)
    return a.view(-1, 2, 1 << (hi - lo - 1), 2, 1 << lo)


def cnot(a, c, t):
    v = quarters(a, c, t)
    i, j = (v[:, 1, :, 0], v[:, 1, :, 1]) if c > t else (v[:, 0, :, 1], v[:, 1, :, 1])
    x = i.clone()
    i.copy_(j)
    j.copy_(x)


def run_gates(a, gates):
    for name, q, v in gates:
        if name == "H":
            apply1(a, q[0], [[H_CONST, H_CONST], [H_CONST, -H_CONST]])
        elif name == "U1":
            apply1(a, q[0], v)
        elif name == "CP":
            quarters(a, *q)[:, 1, :, 1] *= complex(math.cos(v), math.sin(v))
        else:  # SWAP
            w = quarters(a, *q)
            x = w[:, 0, :, 1].clone()
            w[:, 0, :, 1] = w[:, 1, :, 0]
            w[:, 1, :, 0] = x


def ry(t):
    return [[math.cos(t / 2), -math.sin(t / 2)], [math.sin(t / 2), math.cos(t / 2)]]


def rz(t):
    return [[complex(math.cos(t / 2), -math.sin(t / 2)), 0], [0, complex(math.cos(t / 2), math.sin(t / 2))]]


def signs(n, q):
    s = torch.ones(1 << n, dtype=torch.float64, device="cuda")
    s.view(-1, 2, 1 << q)[:, 1] = -1
    return s


def hamiltonian(a, n, J, h):
    out = torch.zeros_like(a)
    d = torch.zeros(1 << n, dtype=torch.float64, device="cuda")
    for i in range(n - 1):
        d += J[i] * signs(n, i) * signs(n, i + 1)
    out += d * a
    for i in range(n):
        out += h[i] * a.view(-1, 2, 1 << i).flip(1).reshape(-1)
    return out


def gradient(n, layers, p, J, h):
    """<H> and its gradient, the forward state undone gate by gate."""
    psi = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
    psi[0] = 1
    p = p.reshape(layers, n, 2)
    for layer in range(layers):
        for q in range(n):
            apply1(psi, q, np.array(rz(p[layer, q, 1])) @ np.array(ry(p[layer, q, 0])))
        for q in range(n - 1):
            cnot(psi, q, q + 1)
    lam = hamiltonian(psi, n, J, h)
    energy = torch.vdot(psi, lam).real
    grad = torch.zeros(layers, n, 2, dtype=torch.float64, device="cuda")
    for layer in reversed(range(layers)):
        for q in reversed(range(n - 1)):
            cnot(psi, q, q + 1)
            cnot(lam, q, q + 1)
        for q in range(n):
            x, y = psi.view(-1, 2, 1 << q), lam.view(-1, 2, 1 << q)
            grad[layer, q, 1] = (y[:, 0].conj() * x[:, 0] - y[:, 1].conj() * x[:, 1]).sum().imag
            for s in (psi, lam):
                apply1(s, q, rz(-p[layer, q, 1]))
            grad[layer, q, 0] = (y[:, 1].conj() * x[:, 0] - y[:, 0].conj() * x[:, 1]).sum().real
            for s in (psi, lam):
                apply1(s, q, ry(-p[layer, q, 0]))
    return float(energy), grad.cpu().numpy().ravel()


def exact(case, seed):
    kind, rng = case["kind"], np.random.default_rng(seed)
    if kind == "grad":
        e, g = gradient(case["n"], case["layers"], *variational(case["n"], case["layers"], rng))
        return {"loss": torch.tensor(e, dtype=torch.float64), "grad": torch.from_numpy(g)}
    if kind == "batch":
        got = [gradient(n, layers, *variational(n, layers, rng))
               for n, layers in batch_sizes(case, np.random.default_rng(case["circuits"]))]
        return {"energies": np.array([e for e, _ in got]), "grads": np.concatenate([g for _, g in got])}
    n = case["n"]
    if kind == "energy":
        v = product_qubits(n, seed)
        _, J, h = variational(n, 0, np.random.default_rng(seed + 1))
        z = np.abs(v[:, 0]) ** 2 - np.abs(v[:, 1]) ** 2
        x = 2 * (v[:, 0].conj() * v[:, 1]).real
        return np.float64(np.sum(J * z[:-1] * z[1:]) + np.sum(h * x))
    if case["circuit"] == "qft":
        a = random_amplitudes(n, seed)
    else:
        a = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
        a[0] = 1
    run_gates(a, gate_list(case, seed))
    return a
