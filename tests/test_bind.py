"""ParamCircuit.bind: what it takes as parameters, and the records it fills
(CPU)."""
import ctypes

import numpy as np
import pytest
import torch

from subquokka_dev_b200 import make_gate
from subquokka_dev_b200.torch_shim import ParamCircuit

U = np.array([[0.6, -0.8], [0.8, 0.6]])
VALUES = [0.25, -1.5, 3.0]


def circuit():
    pc = ParamCircuit(4)
    p = [pc.param() for _ in range(3)]
    pc.rot("RX", 0, p[1])
    pc.fixed("U1", [2], coeff=U)
    pc.fixed("CP", [0, 3], 0.5)
    pc.rot("RZ", 3, p[0])
    pc.fixed("VSWAP", [0, 1, 2, 3])
    pc.rot("RY", 1, p[1])
    return pc


@pytest.mark.parametrize("params", [
    np.array(VALUES), np.array(VALUES, dtype=np.float32), np.array(VALUES).reshape(3, 1)[:, 0], VALUES, tuple(VALUES),
    dict(enumerate(VALUES)), torch.tensor(VALUES, dtype=torch.float64),
    torch.tensor(VALUES, dtype=torch.float64, requires_grad=True),
], ids=["float64", "float32", "strided", "list", "tuple", "dict", "tensor", "tensor with gradient"])
def test_parameters_of_every_kind(params):
    circ, idx = circuit().bind(params)
    want = [make_gate("RX", [0], VALUES[1]), make_gate("U1", [2], coeff=U), make_gate("CP", [0, 3], 0.5),
            make_gate("RZ", [3], VALUES[0]), make_gate("VSWAP", [0, 1, 2, 3]), make_gate("RY", [1], VALUES[1])]
    assert idx.dtype == np.int32 and idx.tolist() == [1, -1, -1, 0, -1, 1]
    assert [ctypes.string_at(ctypes.byref(g), ctypes.sizeof(g)) for g in circ.gate_list()] == \
        [ctypes.string_at(ctypes.byref(g), ctypes.sizeof(g)) for g in want]


def test_missing_parameter_is_an_index_error():
    for params in (np.zeros(1), [0.0]):
        with pytest.raises(IndexError):
            circuit().bind(params)
