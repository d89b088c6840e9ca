"""The kernels called through the native module and through ctypes: the same bits, the same refusals."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def randn(*shape, seed, dtype=torch.float32):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(dtype).to(DEV)


def i32(values):
    return torch.tensor(values, dtype=torch.int32, device=DEV)


def some_calls(api):
    """Calls with pointers, absent pointers, ints, strides and floats, of few and of many arguments."""
    results = []
    x, w, status = randn(70, 128, seed=1), randn(96, 128, seed=2), torch.zeros(1, dtype=torch.int32, device=DEV)
    out = torch.empty(2, 70, 96, device=DEV)
    api.gemm_simt(x, w, None, out)
    results.append(out.clone())
    api.gemm_simt(x, w, randn(96, seed=3), out)
    results.append(out)
    narrow = torch.empty(1, 70, 96, device=DEV)
    api.gemm_tcgen05(x.bfloat16(), w.bfloat16(), randn(96, seed=3), narrow, status)
    results.append(narrow)
    residual, normed = randn(70, 128, seed=4), torch.empty(70, 128, dtype=torch.bfloat16, device=DEV)
    api.add_rmsnorm(residual, x[None], randn(128, seed=5), 1e-5, normed, None, 0.25)
    results += [residual, normed]
    proj, weight, state, conv = randn(1, 70, 64, seed=6), randn(64, 4, seed=7), randn(1, 3, 64, seed=8), torch.empty(70, 64, device=DEV)
    api.causal_conv(proj, 0, 64, weight, None, True, state, conv, i32([0, 70]), i32([0]), 1, 70, False)
    results += [conv, state]
    cols = (3 + 2 + 2) * 32
    pools = [torch.zeros(4, 2, 64, 32, dtype=torch.bfloat16, device=DEV), torch.zeros(4, 2, 32, 64, dtype=torch.bfloat16, device=DEV)]
    q = torch.empty(70, 96, dtype=torch.bfloat16, device=DEV)
    api.qk_norm_rope_append(randn(1, 70, cols, seed=9), randn(32, seed=10), None, 1e-6, torch.linspace(1.0, 0.1, 16, device=DEV), 32, True, 1.5, q, *pools, i32([[2, 0]]), i32([0, 70]),
                            i32([5]), 1, 70, 3, 2, 32, 32, status, q_gain=(0.3, 20))
    results += [q, *pools]
    logits, request, step, token = randn(4, 300, seed=11), i32([1, 2, 3, 4]), i32([0, 5, 6, 7]), i32([0] * 4)
    api.sample_rows(logits, 0.7, 20, 0.9, (1 << 63) + 5, request, step, token)
    results.append(token)
    assert int(status) == 0
    return [r.clone() for r in results]


def test_native_calls_and_ctypes_calls(monkeypatch):
    from thintensor_b200.kernels import api, build

    native = some_calls(api)
    assert api._host, "the native module was not built"
    plain = {name: getattr(api, name) for name in ("_ptr", "_need", "_need_columns")}
    monkeypatch.setattr(build, "host_calls", lambda: None)
    monkeypatch.setattr(api, "_host", None)
    monkeypatch.setattr(api, "_functions", {})
    for name in plain:                                  # what stands there until the module is bound
        monkeypatch.setattr(api, name, getattr(api, name + "_in_python"))
    through_ctypes = some_calls(api)
    assert api._host is False
    for a, b in zip(native, through_ctypes):
        assert torch.equal(a, b)


@pytest.mark.parametrize("native", [True, False])
def test_refusals(monkeypatch, native):
    from thintensor_b200.kernels import api, build

    x, w, out = randn(20, 64, seed=1), randn(32, 64, seed=2), torch.empty(1, 20, 32, device=DEV)
    api.gemm_simt(x, w, None, out)
    if not native:
        monkeypatch.setattr(build, "host_calls", lambda: None)
        monkeypatch.setattr(api, "_host", None)
        monkeypatch.setattr(api, "_functions", {})
        for name in ("_ptr", "_need", "_need_columns"):
            monkeypatch.setattr(api, name, getattr(api, name + "_in_python"))
    launched = api.launch_count()
    for operands in ((x.cpu(), w, None, out), (x, w.cpu(), None, out), (x, w, None, out.cpu()), (x, w, torch.zeros(32), out), (x, w, torch.zeros(32, device=DEV).half(), out),
                     (x, w, None, out.transpose(1, 2)), (x.half(), w, None, out), (x, w[:, :32], None, out)):
        with pytest.raises(api.KernelError):
            api.gemm_simt(*operands)
    assert api.launch_count() == launched
