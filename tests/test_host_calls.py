"""The native module that calls the kernels' C entry points: arguments arrive as ctypes would pass them, and what is refused is refused (no GPU)."""
from __future__ import annotations

import ctypes

import pytest
import torch

from thintensor_b200.kernels import build


class Refused(RuntimeError):
    pass


@pytest.fixture(scope="module")
def host():
    module = build.host_calls()
    if module is None:
        pytest.skip("no C++ compiler, or no Python headers")
    module.set_error(Refused)
    yield module
    from thintensor_b200.kernels import api

    module.set_error(api.KernelError)


TYPES = {"p": ctypes.c_void_p, "i": ctypes.c_int, "l": ctypes.c_longlong, "u": ctypes.c_ulonglong, "f": ctypes.c_float}


def callee(signature: str):
    """A C function of these arguments that notes what it was given."""
    seen = []

    def note(*arguments):
        seen.append(arguments)
        return len(seen) - 3

    function = ctypes.CFUNCTYPE(ctypes.c_int, *(TYPES[letter] for letter in signature))(note)
    return function, ctypes.cast(function, ctypes.c_void_p).value, seen


@pytest.mark.parametrize("signature", ["", "p", "f", "pilufp", "ffffffff", "i" * 40, "ifpl" * 8, "pilipilippppppiiiiiiipp" + "f" * 8, "l" * 6 + "f" * 8 + "i" * 34])
def test_arguments_arrive(host, signature):
    function, address, seen = callee(signature)
    values = {"p": lambda k: 0x7000_0000_0000 + 16 * k, "i": lambda k: (-1) ** k * (1000 + k), "l": lambda k: -(1 << 40) - k, "u": lambda k: (1 << 63) + k,
              "f": lambda k: 0.5 * k - 3.25}
    given = [values[letter](k) for k, letter in enumerate(signature)]
    call = host.Function(address, signature, "note")
    assert call(*given) == -2 and call(*given) == -1 and call(*given) == 0
    assert all(list(arguments) == given for arguments in seen) and len(seen) == 3


def test_arguments_are_taken_and_refused_as_ctypes_takes_and_refuses_them(host):
    function, address, seen = callee("pilf")
    call = host.Function(address, "pilf", "note")
    call(None, True, -1, 2)                                    # no pointer, a truth value, a whole number for a float
    assert seen[-1] == (None, 1, -1, 2.0)
    call(5, (1 << 32) + 7, 3, 1e300 * 0)                       # an int keeps its low 32 bits
    assert seen[-1] == (5, 7, 3, 0.0)
    for wrong in ((1, 2, 3), (1, 2, 3, 4.0, 5), (1, 2.0, 3, 4.0), (1, 2, "3", 4.0), (1, None, 3, 4.0), (1, 2, 3, "4"), (1.0, 2, 3, 4.0)):
        with pytest.raises(TypeError):
            call(*wrong)
    with pytest.raises(TypeError):
        call(1, 2, 3, x=4.0)
    assert len(seen) == 2
    for signature in ("x", "i" * 47, "f" * 9):
        with pytest.raises(ValueError):
            host.Function(address, signature, "note")
    with pytest.raises(ValueError):
        host.Function(0, "i", "note")


def test_tensors_are_checked(host):
    x = torch.zeros(4, 6)
    assert host.pointer(None) == 0
    for check in (lambda: host.pointer(x), lambda: host.need(x, torch.bfloat16, "x"), lambda: host.need(x.T, torch.float32, "x"),
                  lambda: host.need_columns(x.T, torch.float32, "x"), lambda: host.need_columns(x, torch.int32, "x"), lambda: host.need_columns(torch.tensor(1.0), torch.float32, "x")):
        with pytest.raises(Refused):
            check()
    for check in (lambda: host.pointer(3), lambda: host.need([1.0], torch.float32, "x"), lambda: host.need(x, "float32", "x"), lambda: host.need(x, torch.float32)):
        with pytest.raises(TypeError):
            check()
    assert host.need(x, torch.float32, "x") is None and host.need_columns(x[:, 2:], torch.float32, "x") is None
    with pytest.raises(Refused, match="x must be torch.bfloat16, got torch.float32"):
        host.need(x, torch.bfloat16, "x")


def test_operands_of_tiled_products_are_those_of_the_rule_in_python(host, monkeypatch):
    from thintensor_b200.kernels import api

    monkeypatch.setattr(api, "_host", False)
    wide = torch.zeros(24, 64, dtype=torch.bfloat16)
    forms = [wide, wide[:, :40], wide[:, 8:48], wide[:, 4:44], wide[:, :36], wide[1:], wide[:, ::2], wide.T, wide.float(), torch.zeros(24, 40, dtype=torch.bfloat16),
             torch.zeros(24, 36, dtype=torch.bfloat16), wide[:0], wide[:, :0]]
    for a in forms:
        for b in forms:
            assert host.tiled_operands(a, b) == api.gemm_tcgen05_usable(a, b), (a.shape, a.stride(), b.shape, b.stride())
