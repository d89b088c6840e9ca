"""Kernels at the sizes where their tiles, slices and vector accesses change: against the same arithmetic in float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def randn(*shape, seed, scale=1.0, dtype=torch.float32):
    generator = torch.Generator().manual_seed(seed)
    return (torch.randn(*shape, generator=generator) * scale).to(dtype).to(DEV)


# ------------------------------------------------------------------------- exact product: 64 x 128 tiles, 16 k a stage, rows kernel
@pytest.mark.parametrize("m,n,k,pad,splits", [
    (1, 1, 1, 0, 1), (3, 5, 130, 2, 1), (9, 127, 128, 0, 1), (16, 130, 132, 4, 1),                  # few rows: one and two passes of eight
    (17, 127, 15, 0, 1), (64, 128, 16, 4, 1), (65, 129, 17, 1, 1), (96, 256, 100, 4, 3), (97, 300, 1000, 2, 8), (130, 64, 40, 0, 4),
])
@pytest.mark.parametrize("x_dtype,w_dtype", [(torch.float32, torch.float32), (torch.float32, torch.bfloat16), (torch.bfloat16, torch.float32)])
def test_exact_product_at_tile_edges(m, n, k, pad, splits, x_dtype, w_dtype):
    """``pad``: operands are ranges of wider matrices, which moves rows off 16-byte boundaries; the result is a range of
    columns.  An empty last slice (130 x 64 x 40 in four) holds zeros."""
    from thintensor_b200.kernels import api

    x = randn(m, k + pad, seed=1, dtype=x_dtype)[:, pad:]
    w = randn(n, k + pad, seed=2, dtype=w_dtype)[:, pad:]
    bias = randn(n, seed=3)
    wide = torch.full((splits, m, n + pad), 7.0, device=DEV)
    api.gemm_simt(x, w, bias, wide[:, :, :n])
    want = x.double() @ w.double().T + bias.double()
    # k products of unit variance, each sum of at most k terms rounded at 2^-24 of its size
    torch.testing.assert_close(wide[:, :, :n].double().sum(0), want, rtol=0, atol=2.0 ** -24 * (k + splits) * 4 * k ** 0.5 + 1e-6)
    assert bool((wide[:, :, n:] == 7.0).all())


def test_exact_product_slices_follow_the_sizes():
    from thintensor_b200.kernels import api

    assert api.gemm_simt_splits(16, 2048, 8192, 148) == 1               # the kernel for few rows takes no slices
    assert api.gemm_simt_splits(193, 2048, 255, 148) == 1               # slices hold at least 256
    for tokens, features, k in ((17, 64, 512), (193, 2048, 8192), (193, 16384, 2048), (4096, 4096, 4096)):
        splits = api.gemm_simt_splits(tokens, features, k, 148)
        assert 1 <= splits <= 8 and k >= 256 * splits


# ----------------------------------------------------------- recurrences with a decay per head, a chunk of 64 tokens at a time
def i32(values):
    return torch.tensor(values, dtype=torch.int32, device=DEV)


def recurrence(x, b, c, decay, dt, skip, state):
    """Token by token: x [T, H, P], b and c [T, H, N], decay and dt [T, H], state [H, P, N]."""
    out = torch.empty_like(x)
    for t in range(x.shape[0]):
        state = decay[t][:, None, None] * state + (dt[t][:, None] * x[t])[:, :, None] * b[t][:, None, :]
        out[t] = (state @ c[t][:, :, None])[..., 0] + skip[:, None] * x[t]
    return out, state


@pytest.mark.parametrize("heads,groups,P,N,pad", [
    (2, 1, 32, 128, 0), (4, 2, 16, 64, 0), (3, 3, 33, 65, 1), (40, 1, 64, 128, 0), (80, 80, 40, 24, 0), (2, 2, 7, 3, 2),        # both widths of a CTA's columns, both sizes of state
])
@pytest.mark.parametrize("fixed", [False, True])
def test_recurrence_in_chunks(heads, groups, P, N, pad, fixed):
    """Sequences around a chunk's edges and one without tokens, states that are not zero in slots out of order; decays from
    nearly one to nearly nothing, and among the constant ones zero, one and a negative one."""
    from thintensor_b200.kernels import api

    news, slot_ids = [63, 64, 0, 1, 130, 65], [4, 0, 6, 2, 1, 5]
    tokens, inner, sequences = sum(news), heads * P, len(news)
    width = inner + 2 * groups * N + pad
    rows = randn(tokens, width, seed=5)
    x, b, c = rows[:, :inner], rows[:, inner:inner + groups * N], rows[:, inner + groups * N:inner + 2 * groups * N]
    state = randn(8, heads, P, N, seed=6)
    before = state.clone()
    cu = [sum(news[:i]) for i in range(sequences + 1)]
    y = torch.full((tokens, inner), 7.0, device=DEV)
    a_log, dt_bias, skip = randn(heads, seed=7, scale=2.0), randn(heads, seed=8), randn(heads, seed=9)
    raw = randn(2, tokens, heads + 3, seed=10)
    scores, factors = (torch.full(shape, float("nan"), device=DEV) for shape in api.scan_chunks_scratch(tokens, sequences, heads, groups))
    if fixed:
        constant = torch.tensor([0.97, 0.0, 1.0, -0.8], device=DEV).repeat(heads)[:heads].contiguous()
        api.scan_chunks(x, b, c, state, y, i32(cu), i32(slot_ids), sequences, heads, P, N, groups, scores, factors, fixed_decay=constant)
        dt = torch.ones(tokens, heads, device=DEV, dtype=torch.float64)
        decay, skip = constant.double().expand(tokens, heads), torch.zeros(heads, device=DEV)
    else:
        api.scan_chunks(x, b, c, state, y, i32(cu), i32(slot_ids), sequences, heads, P, N, groups, scores, factors, steps=(raw, 2, dt_bias, a_log, skip))
        dt = torch.nn.functional.softplus(raw.double().sum(0)[:, 2:2 + heads] + dt_bias.double())
        decay = torch.exp(-torch.exp(a_log.double()) * dt)
    each = heads // groups
    for s, slot in enumerate(slot_ids):
        span = slice(cu[s], cu[s + 1])
        wide = lambda z: z[span].double().reshape(-1, groups, N).repeat_interleave(each, 1)
        want, last = recurrence(x[span].double().reshape(-1, heads, P), wide(b), wide(c), decay[span], dt[span], skip.double(), before[slot].double())
        # float32 sums over up to 64 tokens and 128 rows; as for the kernels that go token by token
        if news[s]:
            assert float((y[span].double().reshape(-1, heads, P) - want).abs().max()) <= 2e-5 * max(1.0, float(want.abs().max()))
        assert float((state[slot].double() - last).abs().max()) <= 2e-5 * max(1.0, float(last.abs().max()))
    assert torch.equal(state[[3, 7]], before[[3, 7]])
