"""Kernels at the sizes where their tiles, slices and vector accesses change: against the same arithmetic in float64."""
import ctypes

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


@pytest.mark.parametrize("m,n,k,pad,splits", [
    (1, 1, 1, 0, 1), (17, 255, 63, 1, 1), (32, 256, 64, 4, 1), (33, 257, 65, 2, 2), (100, 40, 1000, 0, 4), (193, 600, 520, 4, 3),
    (224, 512, 128, 0, 9), (256, 300, 192, 3, 1), (257, 130, 320, 0, 2), (600, 270, 72, 4, 1),
])
def test_product_in_parts_at_tile_edges(m, n, k, pad, splits):
    """As above, the operands in three bfloat16 parts; more slices than blocks of 64 k leave slices of zeros."""
    from thintensor_b200.kernels import api

    x, w, bias = randn(m, k + pad, seed=1)[:, pad:], randn(n, k + pad, seed=2)[:, pad:], randn(n, seed=3)
    wide = torch.full((splits, m, n + pad), 7.0, device=DEV)
    parts = torch.empty(api.gemm_split_parts(m, k), dtype=torch.bfloat16, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    api.gemm_split(x, w, bias, wide[:, :, :n], parts, status)
    want = x.double() @ w.double().T + bias.double()
    # the products of parts that are left out are at most 2^-23 of a product; the sum of 64 k takes 24 additions that lose up to 2^-23 each, then come the blocks and slices
    size = x.double().abs() @ w.double().abs().T + bias.double().abs()
    error = (wide[:, :, :n].double().sum(0) - want).abs()
    assert bool((error <= (2.0 ** -23 + 24 * 2.0 ** -23 + (k // 64 + splits + 2) * 2.0 ** -24) * size).all())
    # and no further from 64 bits than the multiply-adds, which round k times
    plain = torch.empty(1, m, n, device=DEV)
    api.gemm_simt(x, w, bias, plain)
    if m * n * k >= 1 << 20:
        assert float(error.square().mean()) <= float((plain[0].double() - want).square().mean())
    assert bool((wide[:, :, n:] == 7.0).all()) and int(status) == 0


@pytest.mark.parametrize("m,n,k", [(17, 4096, 64), (100, 1000, 100), (150, 3, 100), (193, 2048, 512), (40, 1024, 2048)])
@pytest.mark.parametrize("kind", ["one sign", "cancelling", "few large", "one alone"])
def test_product_in_parts_of_other_sums(m, n, k, kind):
    """Sums of one sign (the tensor cores truncate), sums that cancel to a thousandth, sums that one product in a few dozen dominates: no further from 64 bits than the
    multiply-adds.  A product that stands alone is right to a unit or two in the last place."""
    from thintensor_b200.kernels import api

    x, w = randn(m, k, seed=190), randn(n, k, seed=191)
    if kind == "one sign":
        x, w = x.abs(), w.abs()
    elif kind == "cancelling":
        half = k // 2
        x[:, half:2 * half] = x[:, :half]
        w[:, half:2 * half] = 1e-3 * randn(n, half, seed=192) - w[:, :half]
    elif kind == "few large":
        x[:, ::40] *= 1e5
    else:
        x[:, 1:] = 0.0
    out, plain = torch.empty(1, m, n, device=DEV), torch.empty(1, m, n, device=DEV)
    parts, status = torch.empty(api.gemm_split_parts(m, k), dtype=torch.bfloat16, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    api.gemm_split(x, w, None, out, parts, status)
    api.gemm_simt(x, w, None, plain)
    want = x.double() @ w.double().T
    assert int(status) == 0
    if kind == "one alone":
        # two products of parts left out, 2^-24 of it at most each, and a truncation to the 24 bits of the largest term (two units of a sum just below a power of two)
        assert bool(((out[0].double() - want).abs() <= (2.0 ** -23 + 2.0 ** -22) * want.abs()).all())
    else:
        in_parts, multiplied = (float((got[0].double() - want).norm() / want.norm()) for got in (out, plain))
        assert in_parts <= multiplied, (in_parts, multiplied)


def test_product_in_parts_of_what_is_not_finite():
    """Infinities, NaN and numbers whose first part would round up to infinity: what the multiply-adds make of them, and nothing
    else is touched."""
    from thintensor_b200.kernels import api

    m, n, k = 70, 300, 200
    x, w = randn(m, k, seed=4), randn(n, k, seed=5)
    clean = torch.empty(1, m, n, device=DEV)
    parts = torch.empty(api.gemm_split_parts(m, k), dtype=torch.bfloat16, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    api.gemm_split(x, w, None, clean, parts, status)
    x[3, 7], x[40, 199], x[69, 0] = float("inf"), float("nan"), 3.4028e38
    w[299, 100], w[0, 0] = float("-inf"), 1e-30
    w[5, 0] = 0.0
    got, want = torch.empty(1, m, n, device=DEV), torch.empty(1, m, n, device=DEV)
    api.gemm_split(x, w, None, got, parts, status)
    api.gemm_simt(x, w, None, want)
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf()) and int(status) == 0
    torch.testing.assert_close(got, want, rtol=2.0 ** -24 * k, atol=2.0 ** -24 * k * k ** 0.5, equal_nan=True)
    rows = torch.ones(m, dtype=torch.bool)
    rows[[3, 40, 69]] = False
    assert torch.equal(got[0][rows][:, 6:299], clean[0][rows][:, 6:299])


@pytest.mark.parametrize("small_x,small_w", [(2.0 ** -100, 1.0), (2.0 ** -110, 1.0), (2.0 ** -120, 1.0), (2.0 ** -70, 2.0 ** -50), (1.0, 2.0 ** -118)])
def test_product_in_parts_of_tiny_numbers(small_x, small_w):
    """Numbers whose third part is below what bfloat16 holds keep the bits of float32; rows of zeros beside them stay zeros."""
    from thintensor_b200.kernels import api

    m, n, k = 40, 130, 192
    x, w = randn(m, k, seed=6) * small_x, randn(n, k, seed=7) * small_w
    x[5], w[9] = 0.0, 0.0
    out, plain = torch.empty(2, m, n, device=DEV), torch.empty(1, m, n, device=DEV)
    parts, status = torch.empty(api.gemm_split_parts(m, k), dtype=torch.bfloat16, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    api.gemm_split(x, w, None, out, parts, status)
    api.gemm_simt(x, w, None, plain)
    want = x.double() @ w.double().T
    in_parts, multiplied = (float((got.double().sum(0) - want).norm() / want.norm()) for got in (out, plain))
    assert in_parts <= multiplied, (in_parts, multiplied)
    assert bool((out[:, 5] == 0.0).all()) and bool((out[:, :, 9] == 0.0).all()) and int(status) == 0


def test_slices_of_products_in_parts_follow_the_sizes():
    from thintensor_b200.kernels import api

    assert api.gemm_split_splits(193, 2048, 255, 148) == 1              # slices hold at least 128
    assert api.gemm_split_splits(193, 16384, 2048, 148) == 1            # enough tiles
    assert api.gemm_split_splits(193, 2048, 8192, 148) == 9             # 8 pairs of 74
    assert not api.gemm_split_pays(16, 2048, 8192) and api.gemm_split_pays(17, 2048, 2048) and not api.gemm_split_pays(300, 64, 64)


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
    x, b, c = rows[:, pad:pad + inner], rows[:, pad + inner:pad + inner + groups * N], rows[:, pad + inner + groups * N:pad + inner + 2 * groups * N]
    places = (pad, pad + inner, pad + inner + groups * N)
    state = randn(8, heads, P, N, seed=6)
    before = state.clone()
    cu = [sum(news[:i]) for i in range(sequences + 1)]
    y = torch.full((tokens, inner), 7.0, device=DEV)
    a_log, dt_bias, skip = randn(heads, seed=7, scale=2.0), randn(heads, seed=8), randn(heads, seed=9)
    raw = randn(2, tokens, heads + 3, seed=10)
    scratch = torch.full(api.scan_chunks_scratch(tokens, sequences, heads, groups), float("nan"), device=DEV)
    if fixed:
        constant = torch.tensor([0.97, 0.0, 1.0, -0.8], device=DEV).repeat(heads)[:heads].contiguous()
        api.scan_chunks(rows, *places, state, y, i32(cu), i32(slot_ids), sequences, heads, P, N, groups, scratch, fixed_decay=constant)
        dt = torch.ones(tokens, heads, device=DEV, dtype=torch.float64)
        decay, skip = constant.double().expand(tokens, heads), torch.zeros(heads, device=DEV)
    else:
        api.scan_chunks(rows, *places, state, y, i32(cu), i32(slot_ids), sequences, heads, P, N, groups, scratch, steps=(raw, 2, dt_bias, a_log, skip))
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


@pytest.mark.parametrize("heads,qk_heads,D,V", [(2, 1, 128, 128), (3, 3, 65, 33), (4, 2, 64, 30), (64, 32, 24, 64), (40, 40, 128, 72), (2, 2, 3, 7)])
def test_delta_rule_in_chunks(heads, qk_heads, D, V):
    """As above for the gated delta rule; the last token of the longest sequence repeats the keys before it (a system whose
    off-diagonal numbers are as large as they get)."""
    from thintensor_b200.kernels import api

    news, slot_ids = [63, 64, 0, 1, 130, 65], [4, 0, 6, 2, 1, 5]
    tokens, sequences, qk = sum(news), len(news), qk_heads * D
    qkv = randn(tokens, 2 * qk + heads * V, seed=15)
    cu = [sum(news[:i]) for i in range(sequences + 1)]
    qkv[cu[5] - 20:cu[5], qk:2 * qk] = qkv[cu[5] - 1, qk:2 * qk]
    state = randn(8, heads, V, D, seed=16)
    before = state.clone()
    out = torch.full((tokens, heads * V), 7.0, device=DEV)
    a_log, dt_bias = randn(heads, seed=17, scale=2.0), randn(heads, seed=18)
    raw = randn(2, tokens, 2 * heads + 3, seed=19)
    scratch = torch.full(api.delta_chunks_scratch(tokens, sequences, heads, D, V), float("nan"), device=DEV)
    api.delta_chunks(qkv, raw, 1, heads + 2, dt_bias, a_log, state, out, i32(cu), i32(slot_ids), sequences, heads, qk_heads, D, V, scratch)
    z = raw.double().sum(0)
    beta = torch.sigmoid(z[:, 1:1 + heads])
    decay = torch.exp(-torch.exp(a_log.double()) * torch.nn.functional.softplus(z[:, heads + 2:2 * heads + 2] + dt_bias.double()))
    unit = lambda y: y / (y.square().sum(-1, keepdim=True) + 1e-6).sqrt()
    share = heads // qk_heads
    q = (unit(qkv[:, :qk].double().reshape(-1, qk_heads, D)) * D ** -0.5).repeat_interleave(share, 1)
    k = unit(qkv[:, qk:2 * qk].double().reshape(-1, qk_heads, D)).repeat_interleave(share, 1)
    v = qkv[:, 2 * qk:].double().reshape(-1, heads, V)
    for s, slot in enumerate(slot_ids):
        S = before[slot].double()
        want = torch.empty(news[s], heads, V, dtype=torch.float64, device=DEV)
        for i in range(news[s]):
            t = cu[s] + i
            S = decay[t][:, None, None] * S
            u = beta[t][:, None] * (v[t] - (S @ k[t][:, :, None])[..., 0])
            S = S + u[:, :, None] * k[t][:, None, :]
            want[i] = (S @ q[t][:, :, None])[..., 0]
        if news[s]:
            got = out[cu[s]:cu[s + 1]].double().reshape(-1, heads, V)
            assert float((got - want).abs().max()) <= 2e-5 * max(1.0, float(want.abs().max()))
        assert float((state[slot].double() - S).abs().max()) <= 2e-5 * max(1.0, float(S.abs().max()))
    assert torch.equal(state[[3, 7]], before[[3, 7]])


@pytest.mark.parametrize("heads,N", [(2, 128), (2, 24), (100, 128), (100, 64)])                     # 16 and 32 columns a CTA, both sizes of state
@pytest.mark.parametrize("what", ["x", "b", "c", "dt"])
@pytest.mark.parametrize("token,value", [(0, float("inf")), (30, float("inf")), (30, float("nan")), (63, float("-inf")), (81, float("nan"))])
def test_recurrence_in_chunks_keeps_later_tokens_out(heads, N, what, token, value):
    """A number that is not finite reaches what it reaches token by token: the earlier tokens' outputs, the other columns and the
    other sequence keep their bits."""
    from thintensor_b200.kernels import api

    P, news = 20, [130, 70]
    tokens, inner = sum(news), heads * P
    cu, slots = i32([0, news[0], tokens]), i32([1, 0])
    a_log, dt_bias, skip = randn(heads, seed=7, scale=2.0), randn(heads, seed=8), randn(heads, seed=9)
    outs = []
    for poisoned in (False, True):
        rows, raw = randn(tokens, inner + 2 * N, seed=90), randn(1, tokens, heads, seed=91)
        if poisoned:
            place = {"x": 3, "b": inner + 2, "c": inner + N + 2, "dt": 1}[what]
            (raw[0] if what == "dt" else rows)[token, place] = value
        forms = []
        for chunks in (True, False):
            state, y = randn(2, heads, P, N, seed=92), torch.full((tokens, inner), 7.0, device=DEV)
            if chunks:
                scratch = torch.full(api.scan_chunks_scratch(tokens, 2, heads, 1), float("nan"), device=DEV)
                api.scan_chunks(rows, 0, inner, inner + N, state, y, cu, slots, 2, heads, P, N, 1, scratch, steps=(raw, 0, dt_bias, a_log, skip))
            else:
                api.mamba2_scan(rows, raw, 0, dt_bias, a_log, skip, state, y, cu, slots, 2, heads, P, N, 1)
            forms.append((y, state))
        outs.append(forms)
    (clean, clean_state), (y, state) = outs[0][0], outs[1][0]
    by_token, by_token_state = outs[1][1]
    assert torch.equal(y[:token], clean[:token]) and torch.equal(y[news[0]:], clean[news[0]:]) and torch.equal(state[0], clean_state[0])
    assert torch.equal(y.isfinite(), by_token.isfinite()) and torch.equal(state.isfinite(), by_token_state.isfinite())


@pytest.mark.parametrize("heads,D", [(2, 128), (2, 24), (100, 128), (100, 64)])
@pytest.mark.parametrize("what", ["q", "k", "v", "beta", "decay"])
@pytest.mark.parametrize("token,value", [(0, float("inf")), (30, float("inf")), (30, float("nan")), (63, float("-inf")), (81, float("nan"))])
def test_delta_rule_in_chunks_keeps_later_tokens_out(heads, D, what, token, value):
    from thintensor_b200.kernels import api

    V, news = 20, [130, 70]
    tokens, qk = sum(news), heads * D
    cu, slots = i32([0, news[0], tokens]), i32([1, 0])
    a_log, dt_bias = randn(heads, seed=17, scale=2.0), randn(heads, seed=18)
    outs = []
    for poisoned in (False, True):
        qkv, raw = randn(tokens, 2 * qk + heads * V, seed=93), randn(1, tokens, 2 * heads, seed=94)
        if poisoned:
            place = {"q": 2, "k": qk + 2, "v": 2 * qk + 3, "beta": 1, "decay": heads + 1}[what]
            (raw[0] if what in ("beta", "decay") else qkv)[token, place] = value
        forms = []
        for chunks in (True, False):
            state, out = randn(2, heads, V, D, seed=95), torch.full((tokens, heads * V), 7.0, device=DEV)
            if chunks:
                scratch = torch.full(api.delta_chunks_scratch(tokens, 2, heads, D, V), float("nan"), device=DEV)
                api.delta_chunks(qkv, raw, 0, heads, dt_bias, a_log, state, out, cu, slots, 2, heads, heads, D, V, scratch)
            else:
                api.delta_scan(qkv, raw, 0, heads, dt_bias, a_log, state, out, cu, slots, 2, heads, heads, D, V)
            forms.append((out, state))
        outs.append(forms)
    (clean, clean_state), (out, state) = outs[0][0], outs[1][0]
    by_token, by_token_state = outs[1][1]
    assert torch.equal(out[:token], clean[:token]) and torch.equal(out[news[0]:], clean[news[0]:]) and torch.equal(state[0], clean_state[0])
    assert torch.equal(out.isfinite(), by_token.isfinite()) and torch.equal(state.isfinite(), by_token_state.isfinite())


# --------------------------------------------------------------------------------- the passes around the recurrences
@pytest.mark.parametrize("group,groups,tokens", [(4, 3, 2), (128, 5, 9), (132, 2, 3), (256, 4, 33), (260, 1, 40), (1024, 2, 600), (1028, 1, 7), (4096, 1, 1030), (8192, 1, 3), (30, 4, 5)])
@pytest.mark.parametrize("splits,gate_first,gate,dtype", [(1, True, "silu", torch.bfloat16), (5, False, "sigmoid", torch.float32)])
def test_gated_group_norm_by_pieces(group, groups, tokens, splits, gate_first, gate, dtype):
    """A warp a group, a block a group with one and with four pieces a thread, and sizes without whole pieces."""
    from thintensor_b200.kernels import api

    width, col = group * groups, 8
    y, proj, weight = randn(tokens, width, seed=20), randn(splits, tokens, width + 12, seed=21), 1.0 + randn(group, seed=22, scale=0.1)
    out = torch.empty(tokens, width, dtype=dtype, device=DEV)
    api.gated_group_norm(y, group, proj, col, weight, 1e-6, gate_first, out, gate)
    z = proj.double().sum(0)[:, col:col + width].reshape(tokens, groups, group)
    z = torch.sigmoid(z) * (1.0 if gate == "sigmoid" else z)
    v = y.double().reshape(tokens, groups, group)
    norm = lambda a: a / (a.square().mean(-1, keepdim=True) + 1e-6).sqrt() * weight.double()
    want = (norm(v * z) if gate_first else norm(v) * z).reshape(tokens, width)
    limit = dict(rtol=2.0 ** -8, atol=1e-6) if dtype == torch.bfloat16 else dict(rtol=1e-5, atol=1e-5)
    torch.testing.assert_close(out.double(), want, **limit)


@pytest.mark.parametrize("splits", [1, 2])
@pytest.mark.parametrize("taps", [1, 4, 8])
def test_convolution_tiles_inside_and_across_sequences(taps, splits):
    """Sequences that start and end inside, at and beyond the tiles (of 8 tokens in one slice, of 16 in two)."""
    from thintensor_b200.kernels import api

    news, slot_ids, channels, col = [16, 40, 1, 23, 33], [3, 0, 5, 1, 2], 130, 3
    tokens = sum(news)
    cu = [sum(news[:i]) for i in range(len(news) + 1)]
    proj, weight, bias = randn(splits, tokens, channels + 7, seed=23), randn(channels, taps, seed=24), randn(channels, seed=25)
    state = randn(6, max(taps - 1, 1), channels, seed=26)[:, :taps - 1].contiguous()
    before = state.clone()
    out = torch.empty(tokens, channels, device=DEV)
    api.causal_conv(proj, col, channels, weight, bias, True, state, out, i32(cu), i32(slot_ids), len(news), tokens, False)
    x = proj.double().sum(0)[:, col:col + channels]
    for s, slot in enumerate(slot_ids):
        rows = torch.cat((before[slot].double(), x[cu[s]:cu[s + 1]]))
        want = sum(rows[j:j + news[s]] * weight[:, j].double() for j in range(taps)) + bias.double()
        torch.testing.assert_close(out[cu[s]:cu[s + 1]].double(), want * torch.sigmoid(want), rtol=1e-5, atol=1e-5)
        torch.testing.assert_close(state[slot].double(), rows[rows.shape[0] - (taps - 1):], rtol=1e-6, atol=1e-6)


@pytest.mark.parametrize("channels,col,extra", [(4, 0, 0), (132, 4, 8), (516, 0, 4), (1032, 8, 0)])
@pytest.mark.parametrize("news", [[1, 2, 3, 7, 8, 9, 17], [5, 0, 0, 64, 1], [700]])
def test_convolution_four_channels_a_thread(channels, col, extra, news):
    """Four taps in 16-byte pieces: sequences shorter than the filter, tiles whole and in part, sequences without tokens; states moved on in the same launch."""
    from thintensor_b200.kernels import api

    tokens, taps, slot_ids = sum(news), 4, [(3 * i + 1) % 8 for i in range(len(news))]
    cu = [sum(news[:i]) for i in range(len(news) + 1)]
    proj, weight, bias = randn(1, tokens, col + channels + extra, seed=33), randn(channels, taps, seed=34), randn(channels, seed=35)
    state = randn(8, taps - 1, channels, seed=36)
    before = state.clone()
    out = torch.full((tokens, channels), 7.0, device=DEV)
    api.causal_conv(proj, col, channels, weight, bias, False, state, out, i32(cu), i32(slot_ids), len(news), tokens, False)
    x = proj[0].double()[:, col:col + channels]
    for s, slot in enumerate(slot_ids):
        rows = torch.cat((before[slot].double(), x[cu[s]:cu[s + 1]]))
        want = sum(rows[j:j + news[s]] * weight[:, j].double() for j in range(taps)) + bias.double()
        torch.testing.assert_close(out[cu[s]:cu[s + 1]].double(), want, rtol=1e-5, atol=1e-5)        # four products in float32
        assert torch.equal(state[slot].double(), rows[rows.shape[0] - (taps - 1):])
    assert all(torch.equal(state[i], before[i]) for i in range(8) if i not in slot_ids)


@pytest.mark.parametrize("heads,D,V,rotary,tokens", [(3, 128, 256, 128, 5), (2, 64, 20, 24, 1030), (2, 12, 8, 0, 3), (2, 10, 8, 4, 3), (1, 256, 4, 256, 2)])
@pytest.mark.parametrize("activation", [False, True])
def test_linear_attention_inputs_by_pieces(heads, D, V, rotary, tokens, activation):
    from thintensor_b200.kernels import api

    qk, hv, past = heads * D, heads * V, 77
    proj = randn(2, tokens, 2 * qk + hv + 4, seed=27)
    inv_freq = (100.0 ** (-torch.arange(0, max(rotary, 2), 2, dtype=torch.float64) / max(rotary, 2))).float().to(DEV)
    vkq = torch.empty(tokens, hv + 2 * qk, device=DEV)
    api.linear_attention_prepare(proj, heads, D, V, activation, inv_freq, rotary, 0.5, vkq, i32([0, tokens]), i32([past]), 1, tokens, 2.0)
    x = proj.double().sum(0)
    x = x * torch.sigmoid(x) if activation else x
    q, k, v = (part.reshape(tokens, heads, -1) for part in x[:, :2 * qk + hv].split((qk, qk, hv), 1))
    angle = ((past + torch.arange(tokens, device=DEV)).float()[:, None, None] * inv_freq[:rotary // 2]).double()

    def turn(z):
        a, b, h = z[..., :rotary // 2], z[..., rotary // 2:rotary], z[..., rotary:]
        return torch.cat((a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin(), h), -1) if rotary else z

    want = torch.cat((v.reshape(tokens, -1), 0.5 * turn(k).reshape(tokens, -1), 2.0 * turn(q).reshape(tokens, -1)), 1)
    torch.testing.assert_close(vkq.double(), want, rtol=1e-5, atol=2e-5)


# ------------------------------------------------------------------------------------ exact attention in tiles of 32 queries
@pytest.mark.parametrize("heads,kv_heads,D,V", [(4, 2, 64, 64), (3, 1, 128, 128), (2, 2, 48, 80), (2, 1, 16, 112), (2, 1, 30, 17)])
@pytest.mark.parametrize("window,sink,cap", [(0, False, 0.0), (40, True, 5.0), (-48, False, 0.0)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_exact_attention_tiles(heads, kv_heads, D, V, window, sink, cap, dtype):
    """Sequences that end inside, at and behind tiles and cache blocks, with and without a past; whatever lies in the cache beside what
    is seen is no number, and one late value is not either: only its own query and the later ones may meet it."""
    from thintensor_b200.kernels import api

    news, past = [31, 64, 1, 33, 65], [0, 40, 63, 64, 5]
    tokens, sequences = sum(news), len(news)
    cu = [sum(news[:i]) for i in range(sequences + 1)]
    width = 4
    blocks = sequences * width
    order = torch.randperm(blocks, generator=torch.Generator().manual_seed(1)).tolist()
    k_pool = torch.full((blocks, kv_heads, 64, D), float("nan"), dtype=dtype, device=DEV)
    v_pool = torch.full((blocks, kv_heads, V, 64), float("nan"), dtype=dtype, device=DEV)
    table = [[order[s * width + i] if i * 64 < past[s] + news[s] else -1 for i in range(width)] for s in range(sequences)]
    q = randn(tokens, heads * D, seed=30, dtype=dtype)
    sinks = randn(heads, seed=31) if sink else None
    slopes = randn(heads, seed=32).abs() * 0.01 if cap else None
    gate = randn(2, tokens, heads * V, seed=33) if window > 0 else None
    values, keys = [], []
    for s in range(sequences):
        n = past[s] + news[s]
        k, v = randn(n, kv_heads, D, seed=40 + s, dtype=dtype), randn(n, kv_heads, V, seed=50 + s, dtype=dtype)
        keys.append(k)
        values.append(v)
        for i in range(-(-n // 64)):
            part = slice(64 * i, min(n, 64 * i + 64))
            k_pool[table[s][i], :, :part.stop - part.start] = k[part].transpose(0, 1)
            v_pool[table[s][i], :, :, :part.stop - part.start] = v[part].permute(1, 2, 0)
    poisoned = past[1] + 20                                     # a place of the second sequence
    v_pool[table[1][poisoned // 64], :, :, poisoned % 64] = float("nan")
    out = torch.full((tokens, heads * V), 7.0, dtype=dtype, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    api.attention(q, k_pool, v_pool, i32(table), i32(cu), i32(past), sequences, tokens, heads, kv_heads, D, D ** -0.5, window, 1, out, None, None, status,
                  value_dim=V, sinks=sinks, softcap=cap, slopes=slopes, gate=gate)
    assert int(status) == 0
    for s in range(sequences):
        n = past[s] + news[s]
        for h in range(heads):
            place = past[s] + torch.arange(news[s], device=DEV)
            key = torch.arange(n, device=DEV)
            score = q[cu[s]:cu[s + 1]].double().reshape(-1, heads, D)[:, h] @ keys[s][:, h // (heads // kv_heads)].double().T * D ** -0.5
            if cap:
                score = cap * torch.tanh(score / cap) - slopes[h].double() * (place[:, None] - key[None])
            seen = key[None] <= place[:, None]
            if window > 0:
                seen &= key[None] > place[:, None] - window
            if window < 0:
                seen &= key[None] >= (place - place % -window)[:, None]
            score = score.masked_fill(~seen, -float("inf"))
            if sink:
                score = torch.cat((score, sinks[h].double().expand(news[s], 1)), 1)
            want = torch.softmax(score, -1)[:, :n] @ values[s][:, h // (heads // kv_heads)].double()
            if gate is not None:
                want = want * torch.sigmoid(gate.double().sum(0)[cu[s]:cu[s + 1], h * V:(h + 1) * V])
            got = out[cu[s]:cu[s + 1]].double().reshape(-1, heads, V)[:, h]
            clean = ~seen[:, poisoned] if s == 1 else torch.ones(news[s], dtype=torch.bool, device=DEV)
            limit = dict(rtol=2e-5, atol=2e-5) if dtype == torch.float32 else dict(rtol=2.0 ** -8, atol=1e-4)
            torch.testing.assert_close(got[clean], want[clean], **limit)
            assert bool(got[~clean].isnan().all())


# ------------------------------------------------------------------------- latent attention: several tokens of a head together
@pytest.mark.parametrize("heads,dim,rot,V,rank,dtype,tensor_cores", [
    (16, 64, 64, 128, 512, torch.bfloat16, True), (5, 24, 16, 20, 48, torch.bfloat16, True), (20, 9, 32, 33, 144, torch.bfloat16, True),
    (3, 20, 10, 17, 40, torch.float32, False), (2, 16, 8, 12, 20, torch.float32, False),
])
@pytest.mark.parametrize("tokens", [1, 7, 8, 13])
@pytest.mark.parametrize("gate", [None, "head", "each"])
def test_latent_decode_groups(heads, dim, rot, V, rank, dtype, tensor_cores, tokens, gate):
    """One token for each of as many sequences: fewer than a group, a whole one, and one and a part; slices that lie in one cache block and in
    two, empty ones, and heads that do not fill sixteen rows."""
    from thintensor_b200.kernels import api

    window, scale, row = 100, (dim + rot) ** -0.5, rank + rot
    past = [(37 * i + 63) % 190 for i in range(tokens)]
    width = 3
    pool = randn(tokens * width, 1, 64, row, seed=60, dtype=dtype)
    order = torch.randperm(tokens * width, generator=torch.Generator().manual_seed(2)).tolist()
    table = [order[i * width:(i + 1) * width] for i in range(tokens)]
    q = randn(2, tokens, heads * (dim + rot), seed=61)
    w_key, w_value = (randn(heads * n, rank, seed=62 + i, scale=rank ** -0.5, dtype=dtype) for i, n in enumerate((dim, V)))
    gates = None if gate is None else randn(3, tokens, heads if gate == "head" else heads * V, seed=64)
    inv_freq = torch.tensor([1.0, 0.1, 0.01, 0.001], device=DEV)
    out = torch.full((tokens, heads * V), 7.0, dtype=dtype, device=DEV)
    splits = 2 if tensor_cores else 3
    scratch = lambda n: torch.full((n,), float("nan"), device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    api.latent_attention(q, w_key, w_value, pool, i32(table), i32(list(range(tokens + 1))), i32(past), tokens, tokens, heads, dim, rot, V, rank, inv_freq, 8, scale,
                         window, splits, out, scratch(tokens * heads * row), scratch(tokens * heads * splits * rank), scratch(tokens * heads * splits * 2), status,
                         tensor_cores, gate=gates)
    assert int(status) == 0
    z = q.double().sum(0).reshape(tokens, heads, dim + rot)
    for t in range(tokens):
        angle = (past[t] * inv_freq).double()
        a, b = z[t, :, dim:dim + 4], z[t, :, dim + 4:dim + 8]
        turned = torch.cat((a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin(), z[t, :, dim + 8:]), 1)
        folded = torch.cat((torch.einsum("hd,hdr->hr", z[t, :, :dim], w_key.double().reshape(heads, dim, rank)), turned), 1) * scale
        rows = pool[torch.tensor(table[t], device=DEV)].double().reshape(-1, row)[max(0, past[t] + 1 - window):past[t] + 1]
        mixed = torch.softmax(folded @ rows.T, -1) @ rows[:, :rank]
        want = torch.einsum("hr,hvr->hv", mixed, w_value.double().reshape(heads, V, rank)).reshape(-1)
        if gate is not None:
            g = torch.sigmoid(gates.double().sum(0)[t])
            want = want * (g.repeat_interleave(V) if gate == "head" else g)
        # bfloat16: folded queries, probabilities and the result are narrowed, each to eight bits
        error = float((out[t].double() - want).norm() / want.norm())
        assert error <= (2e-5 if dtype == torch.float32 else 3 * 2.0 ** -8), (t, error)


@pytest.mark.parametrize("dtype,tensor_cores", [(torch.bfloat16, True), (torch.float32, False)])
@pytest.mark.parametrize("off", [1, 4])
def test_latent_slice_sums_off_their_boundary(dtype, tensor_cores, off):
    """The slices' sums 4 and 16 bytes off: fragments are stored through shared memory, and at 4 bytes the kernel that combines slices
    four numbers at a time leaves the call to the one that takes them singly."""
    from thintensor_b200.kernels import api

    tokens, heads, dim, rot, V, rank, splits, past = 9, 16, 16, 16, 24, 48, 2, 100
    row = rank + rot
    pool, table = randn(tokens * 2, 1, 64, row, seed=80, dtype=dtype), torch.arange(tokens * 2, dtype=torch.int32, device=DEV).reshape(tokens, 2)
    q = randn(1, tokens, heads * (dim + rot), seed=81)
    w_key, w_value = (randn(heads * n, rank, seed=82, scale=rank ** -0.5, dtype=dtype) for n in (dim, V))
    outs = []
    for shift in (0, off):
        out, status = torch.full((tokens, heads * V), 7.0, dtype=dtype, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
        part = torch.full((tokens * heads * splits * rank + 8,), float("nan"), device=DEV)
        api.latent_attention(q, w_key, w_value, pool, table, i32(list(range(tokens + 1))), i32([past] * tokens), tokens, tokens, heads, dim, rot, V, rank,
                             torch.ones(rot // 2, device=DEV), rot, row ** -0.5, 0, splits, out, torch.empty(tokens * heads * row, device=DEV),
                             part[shift:-8 + shift], torch.empty(tokens * heads * splits * 2, device=DEV), status, tensor_cores)
        assert int(status) == 0
        outs.append(out.double())
    # the same numbers with the expansion's float32 sums in another order, then (bfloat16) narrowed once
    assert float((outs[1] - outs[0]).norm() / outs[0].norm()) <= (1e-6 if dtype == torch.float32 else 2.0 ** -8)


# --------------------------------------------------------------------------------------------- routing, a warp a token
@pytest.mark.parametrize("hidden,experts,extra", [(8, 5, 0), (2048, 16, 1), (2056, 33, 0), (4096, 40, 2), (4104, 8, 0), (100, 8, 0)])
@pytest.mark.parametrize("tokens", [1024, 1025, 1031])
def test_routing_of_prompts(hidden, experts, extra, tokens):
    """Rows of one piece a lane and of the most there are, rows that are no whole pieces, and too long ones (both forms)."""
    from thintensor_b200.kernels import api

    x = randn(tokens, hidden, seed=70, dtype=torch.bfloat16)
    w = randn(experts + extra, hidden, seed=71, scale=hidden ** -0.5, dtype=torch.bfloat16)
    top = 3
    gates, chosen, weights = torch.empty(tokens, experts + extra, device=DEV), torch.empty(tokens, top, dtype=torch.int32, device=DEV), torch.empty(tokens, top, device=DEV)
    api.route_rows(x, w, top, 1, 1, gates, chosen, weights, extra=extra)
    logits = x.double() @ w.double().T
    score = torch.softmax(logits[:, :experts], -1)
    value, index = score.topk(top + 1, -1)
    clear = (value[:, :-1] - value[:, 1:]).amin(1) > 1e-5           # float32 sums of up to 4,104 products decide closer calls as they fall
    assert float(clear.double().mean()) > 0.95
    assert torch.equal(chosen[clear].long(), index[clear, :top])
    torch.testing.assert_close(weights[clear].double(), (value / value[:, :top].sum(1, keepdim=True))[clear, :top], rtol=1e-4, atol=1e-6)
    torch.testing.assert_close(gates[:, experts:].double(), torch.sigmoid(logits[:, experts:]), rtol=1e-4, atol=1e-6)
    dense = torch.zeros(tokens, experts, device=DEV).scatter_(1, chosen.long(), weights)
    assert torch.equal(gates[:, :experts], dense)


@pytest.mark.parametrize("hidden,experts,extra,tokens", [(512, 6, 1, 1185), (504, 8, 0, 1185), (768, 16, 0, 1200), (1024, 40, 0, 1300), (1536, 5, 0, 1037), (1792, 7, 0, 1025),
                                                         (2560, 16, 0, 1025), (2568, 9, 1, 1030), (3584, 20, 0, 1025), (3592, 8, 0, 1025)])
def test_routing_at_row_lengths(hidden, experts, extra, tokens):
    """Both forms on both sides of the shortest rows that a warp takes, and every instance at the ends of its row lengths."""
    test_routing_of_prompts(hidden, experts, extra, tokens)


@pytest.mark.parametrize("width,shared", [(8, 0), (16, 24), (5, 0), (12, 3)])                       # whole 16-byte pieces, and single numbers
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("tokens", [1, 37, 700])
def test_weights_of_experts(width, shared, dtype, tokens):
    """What an expert made of a token that did not choose it is left out, be it a number or not; every other product is one
    rounding of the exact one."""
    from thintensor_b200.kernels import api

    experts = 6
    act = randn(tokens, experts * width + shared, seed=96, dtype=dtype)
    gates = randn(tokens, experts + (1 if shared else 0), seed=97).abs() + 0.1
    gates[:, :experts] *= torch.arange(experts, device=DEV) % 3 == torch.arange(tokens, device=DEV)[:, None] % 3
    each = gates[:, :experts].repeat_interleave(width, 1)
    each = torch.cat((each, gates[:, experts:].expand(tokens, shared)), 1) if shared else each
    act[each == 0] = float("inf")
    act[:, 1] = torch.where(each[:, 1] == 0, float("nan"), act[:, 1].float()).to(dtype)
    want = torch.where(each == 0, torch.zeros((), device=DEV), act.float() * each).to(dtype)
    api.scale_expert_columns(act, width, gates, experts, shared)
    assert torch.equal(act, want)


@pytest.mark.parametrize("group,groups,tokens", [(4, 700, 6), (32, 4, 1023), (32, 4, 1025), (60, 1, 4100), (64, 1, 5)])
@pytest.mark.parametrize("splits,gate_first", [(1, True), (9, False)])
def test_gated_group_norm_of_small_groups(group, groups, tokens, splits, gate_first):
    """On both sides of the number of groups from which small ones go in pieces, with slices that do not fill a round of loads."""
    test_gated_group_norm_by_pieces(group, groups, tokens, splits, gate_first, "silu", torch.float32)


@pytest.mark.parametrize("heads,D,V,rotary,tokens", [(16, 128, 128, 128, 32), (16, 128, 128, 128, 33), (2, 256, 4, 256, 200), (2, 12, 8, 0, 3200), (3, 64, 20, 24, 1400)])
def test_linear_attention_inputs_of_prompts(heads, D, V, rotary, tokens):
    """On both sides of the size from which they are made in pieces."""
    test_linear_attention_inputs_by_pieces(heads, D, V, rotary, tokens, True)


@pytest.mark.parametrize("m,n,k,pad,splits", [(17, 300, 500, 0, 1), (65, 63, 40, 0, 1), (100, 64, 64, 4, 1), (130, 129, 257, 1, 2), (9, 300, 130, 0, 1), (16, 64, 64, 0, 1),
                                              (193, 2048, 512, 0, 1), (193, 3072, 512, 4, 2), (97, 300, 1000, 2, 8)])
@pytest.mark.parametrize("x_dtype,w_dtype", [(torch.float32, torch.float32), (torch.float32, torch.bfloat16), (torch.bfloat16, torch.float32), (torch.bfloat16, torch.bfloat16)])
def test_exact_product_is_exact_to_float32(m, n, k, pad, splits, x_dtype, w_dtype):
    """Tiles of both widths, few rows in several passes.  A chain of k multiply-adds whose partial sums grow like sqrt(i) is off by about
    2^-24 sqrt(k) / 2.4 of the result (2-norm); operands rounded to eleven or eight bits would be off by 2^-12 or more."""
    from thintensor_b200.kernels import api

    x, w = randn(m, k + pad, seed=1, dtype=x_dtype)[:, pad:], randn(n, k + pad, seed=2, dtype=w_dtype)[:, pad:]
    wide = torch.full((splits, m, n + pad), 7.0, device=DEV)
    api.gemm_simt(x, w, None, wide[:, :, :n])
    want = x.double() @ w.double().T
    assert float((wide[:, :, :n].double().sum(0) - want).norm() / want.norm()) <= 2.0 ** -24 * (2 * k ** 0.5 + 4)
    assert bool((wide[:, :, n:] == 7.0).all())


@pytest.mark.parametrize("heads,kv_heads,D,V", [(4, 2, 64, 64), (32, 8, 48, 80), (3, 1, 128, 128)])
@pytest.mark.parametrize("sequences,new,past", [(1, 8, 0), (1, 17, 40), (3, 31, 0), (3, 32, 32), (2, 47, 9), (2, 48, 0), (1, 64, 0)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_exact_attention_of_one_block(heads, kv_heads, D, V, sequences, new, past, dtype):
    """Tables one block wide, on both sides of the line from which queries go in tiles; the block's places behind the last key hold no
    numbers."""
    from thintensor_b200.kernels import api

    tokens, n = sequences * new, past + new
    k_pool = torch.full((sequences, kv_heads, 64, D), float("nan"), dtype=dtype, device=DEV)
    v_pool = torch.full((sequences, kv_heads, V, 64), float("nan"), dtype=dtype, device=DEV)
    k_pool[:, :, :n] = randn(sequences, kv_heads, n, D, seed=110, dtype=dtype)
    v_pool[:, :, :, :n] = randn(sequences, kv_heads, V, n, seed=111, dtype=dtype)
    table = torch.arange(sequences, dtype=torch.int32, device=DEV).flip(0)[:, None].contiguous()
    q, out = randn(tokens, heads * D, seed=112, dtype=dtype), torch.full((tokens, heads * V), 7.0, dtype=dtype, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    api.attention(q, k_pool, v_pool, table, i32([new * i for i in range(sequences + 1)]), i32([past] * sequences), sequences, tokens, heads, kv_heads, D, D ** -0.5,
                  0, 1, out, None, None, status, value_dim=V)
    assert int(status) == 0
    each = heads // kv_heads
    for s in range(sequences):
        K, W = (pool[sequences - 1 - s].double() for pool in (k_pool, v_pool))
        score = torch.einsum("thd,hnd->htn", q[s * new:(s + 1) * new].double().reshape(new, heads, D), K[:, :n].repeat_interleave(each, 0)) * D ** -0.5
        score = score.masked_fill(torch.arange(n, device=DEV)[None] > past + torch.arange(new, device=DEV)[:, None], -float("inf"))
        want = torch.einsum("htn,hvn->thv", torch.softmax(score, -1), W[:, :, :n].repeat_interleave(each, 0)).reshape(new, -1)
        limit = dict(rtol=2e-5, atol=2e-5) if dtype == torch.float32 else dict(rtol=2.0 ** -8, atol=1e-4)
        torch.testing.assert_close(out[s * new:(s + 1) * new].double(), want, **limit)


# ------------------------------------------------------------------------------------------ long prompts through the tiles and chunks
@pytest.mark.parametrize("taps", [1, 4, 8])
def test_convolution_of_long_prompts(taps):
    """One k-slice and at least 1,024 tokens: tiles of 16 tokens whose inputs are asked for at once.  Sequences that end inside, at and
    across tiles, one of a single token, and a last tile that is not full."""
    from thintensor_b200.kernels import api

    news, slot_ids, channels, col = [16, 40, 1, 23, 911, 33, 15], [3, 0, 5, 1, 2, 6, 4], 130, 3
    tokens = sum(news)
    assert tokens >= 1024 and tokens % 16
    cu = [sum(news[:i]) for i in range(len(news) + 1)]
    proj, weight, bias = randn(1, tokens, channels + 7, seed=23), randn(channels, taps, seed=24), randn(channels, seed=25)
    state = randn(8, max(taps - 1, 1), channels, seed=26)[:, :taps - 1].contiguous()
    before = state.clone()
    out = torch.full((tokens, channels), 7.0, device=DEV)
    api.causal_conv(proj, col, channels, weight, bias, True, state, out, i32(cu), i32(slot_ids), len(news), tokens, False)
    x = proj[0].double()[:, col:col + channels]
    for s, slot in enumerate(slot_ids):
        rows = torch.cat((before[slot].double(), x[cu[s]:cu[s + 1]]))
        want = sum(rows[j:j + news[s]] * weight[:, j].double() for j in range(taps)) + bias.double()
        torch.testing.assert_close(out[cu[s]:cu[s + 1]].double(), want * torch.sigmoid(want), rtol=1e-5, atol=1e-5)
        assert torch.equal(state[slot].double(), rows[rows.shape[0] - (taps - 1):])
    assert torch.equal(state[7], before[7])


@pytest.mark.parametrize("heads,qk_heads,D,V", [(2, 1, 64, 130), (2, 2, 128, 257), (3, 3, 24, 70), (40, 20, 64, 130)])
def test_delta_rule_in_chunks_in_several_value_tiles(heads, qk_heads, D, V):
    """Value columns beyond a tile of 64 or 128: the first kernel's halves take further tiles in the keys' and queries' place."""
    test_delta_rule_in_chunks(heads, qk_heads, D, V)


@pytest.mark.parametrize("heads,P,N", [(2, 32, 128), (70, 64, 64)])
def test_recurrence_in_many_chunks(heads, P, N):
    """Seventeen chunks, so that both stages of shared memory are filled many times; among the constant decays some beyond one."""
    from thintensor_b200.kernels import api

    news = [1027, 200]
    tokens, inner = sum(news), heads * P
    cu, slots = i32([0, news[0], tokens]), i32([1, 0])
    rows, state = randn(tokens, inner + 2 * heads * N, seed=100, scale=0.5), randn(2, heads, P, N, seed=101)
    before, y = state.clone(), torch.full((tokens, inner), 7.0, device=DEV)
    decays = torch.tensor([0.99, 1.003, -1.002, 0.5], device=DEV).repeat(heads)[:heads].contiguous()
    scratch = torch.full(api.scan_chunks_scratch(tokens, 2, heads, heads), float("nan"), device=DEV)
    api.scan_chunks(rows, 0, inner, inner + heads * N, state, y, cu, slots, 2, heads, P, N, heads, scratch, fixed_decay=decays)
    x, b, c = (z.double().reshape(tokens, heads, -1) for z in rows.split((inner, heads * N, heads * N), 1))
    for s, slot in enumerate((1, 0)):
        span = slice(int(cu[s]), int(cu[s + 1]))
        ones = torch.ones(news[s], heads, dtype=torch.float64, device=DEV)
        want, last = recurrence(x[span], b[span], c[span], decays.double() * ones, ones, torch.zeros(heads, dtype=torch.float64, device=DEV), before[slot].double())
        # heads grow by up to 1.003^1,027 = 22: each against its own size, as in the shorter test
        for h in range(heads):
            assert float((y[span].double().reshape(-1, heads, P)[:, h] - want[:, h]).abs().max()) <= 2e-5 * max(1.0, float(want[:, h].abs().max()))
            assert float((state[slot, h].double() - last[h]).abs().max()) <= 2e-5 * max(1.0, float(last[h].abs().max()))


@pytest.mark.parametrize("heads,groups,P,N", [(4, 1, 32, 128), (4, 2, 24, 64)])
def test_recurrence_in_chunks_is_as_close_as_token_by_token(heads, groups, P, N):
    """Outputs against 64 bits, 2-norm: no further off than token by token but for a twentieth (the scores' sums of 32 in one chain, which a
    chunk's outputs are made of, were a quarter to a third further off)."""
    from thintensor_b200.kernels import api

    tokens, inner = 900, heads * P
    rows, raw = randn(tokens, inner + 2 * groups * N, seed=120), randn(1, tokens, heads, seed=121)
    a_log, dt_bias, skip = randn(heads, seed=122), randn(heads, seed=123), randn(heads, seed=124)
    cu, slots = i32([0, tokens]), i32([0])
    outs = []
    for chunks in (True, False):
        state, y = torch.zeros(1, heads, P, N, device=DEV), torch.empty(tokens, inner, device=DEV)
        if chunks:
            scratch = torch.empty(api.scan_chunks_scratch(tokens, 1, heads, groups), device=DEV)
            api.scan_chunks(rows, 0, inner, inner + groups * N, state, y, cu, slots, 1, heads, P, N, groups, scratch, steps=(raw, 0, dt_bias, a_log, skip))
        else:
            api.mamba2_scan(rows, raw, 0, dt_bias, a_log, skip, state, y, cu, slots, 1, heads, P, N, groups)
        outs.append((y.double().reshape(tokens, heads, P), state[0].double()))
    x, b, c = rows.double().split((inner, groups * N, groups * N), 1)
    wide = lambda z: z.reshape(tokens, groups, N).repeat_interleave(heads // groups, 1)
    dt = torch.nn.functional.softplus(raw[0].double() + dt_bias.double())
    want, last = recurrence(x.reshape(tokens, heads, P), wide(b), wide(c), torch.exp(-torch.exp(a_log.double()) * dt), dt, skip.double(),
                            torch.zeros(heads, P, N, dtype=torch.float64, device=DEV))
    for i, exact in enumerate((want, last)):
        chunked, by_token = (float((o[i] - exact).norm() / exact.norm()) for o in outs)
        assert chunked <= 1.05 * by_token, (i, chunked, by_token)


def scan_columns(heads, sequences, P, N):
    """Columns of a CTA of the walk over the chunks, as the launcher chooses them."""
    from thintensor_b200.kernels import api, build

    return build.load("recurrent_chunks").tt_scan_chunks_columns(heads, sequences, P, N, api.sm_count())


def delta_columns(heads, sequences, D, V):
    from thintensor_b200.kernels import api, build

    return build.load("recurrent_chunks").tt_delta_chunks_columns(heads, sequences, D, V, api.sm_count())


CHUNKED = 6         # sequences of test_recurrence_in_chunks


@pytest.mark.parametrize("heads,groups,P,N,columns", [(24, 24, 128, 128, 128), (22, 22, 100, 128, 128), (24, 24, 130, 128, 32), (24, 24, 256, 128, 128), (24, 24, 120, 64, 128), (24, 4, 110, 50, 128),
                                                      (24, 4, 64, 128, 64), (24, 24, 50, 128, 64), (40, 40, 130, 128, 64), (24, 24, 50, 40, 64), (40, 8, 70, 128, 32), (3, 3, 50, 128, 16),
                                                      (5, 1, 90, 128, 32), (5, 1, 90, 64, 32)])
@pytest.mark.parametrize("fixed", [False, True])
def test_recurrence_in_chunks_in_wide_tiles(heads, groups, P, N, columns, fixed):
    """Grids whose CTAs hold 16 to 128 columns, whole and in part, with one tile and several."""
    assert scan_columns(heads, CHUNKED, P, N) == columns
    test_recurrence_in_chunks(heads, groups, P, N, 0, fixed)


@pytest.mark.parametrize("n_tokens,sequences,heads,groups,N", [(1, 1, 1, 1, 1), (200, 3, 8, 4, 64), (4097, 1, 64, 1, 65), (700, 16, 3, 3, 128)])
def test_chunks_scratch_is_what_the_kernels_lay_out(n_tokens, sequences, heads, groups, N):
    from thintensor_b200.kernels import api, build

    lib, slots = build.load("recurrent_chunks"), api.chunk_slots(n_tokens, sequences)
    lib.tt_scan_chunks_scratch_bytes.restype = lib.tt_delta_chunks_scratch_bytes.restype = ctypes.c_longlong
    assert 4 * api.scan_chunks_scratch(n_tokens, sequences, heads, groups, N)[0] == lib.tt_scan_chunks_scratch_bytes(slots, heads, groups, N)
    for V in (1, 20, 128):
        assert 4 * api.delta_chunks_scratch(n_tokens, sequences, heads, N, V, groups)[0] == lib.tt_delta_chunks_scratch_bytes(slots, heads, groups, N, V)


@pytest.mark.parametrize("heads,P,N,columns", [(70, 128, 128, 128), (70, 100, 64, 128), (70, 64, 128, 64), (70, 130, 64, 64), (100, 130, 64, 32), (100, 130, 128, 32), (1, 20, 128, 16)])
@pytest.mark.parametrize("what", ["x", "c", "state"])
@pytest.mark.parametrize("decay,token", [(0.9, 100), (0.5, 100), (0.5, 125)])
def test_recurrence_in_chunks_keeps_other_columns(heads, P, N, columns, what, decay, token):
    """A number that is not finite, in the widths of a CTA's columns, ahead of a chunk's tail and in it: what it does not reach keeps its bits, what it reaches is what it
    is token by token."""
    from thintensor_b200.kernels import api

    assert scan_columns(heads, 2, P, N) == columns
    news, inner = [150, 70], heads * P
    tokens = sum(news)
    cu, slots, decays = i32([0, news[0], tokens]), i32([1, 0]), torch.full((heads,), decay, device=DEV)
    outs = []
    for poisoned, chunks in ((False, True), (True, True), (True, False)):
        rows, state = randn(tokens, inner + 2 * heads * N, seed=130), randn(2, heads, P, N, seed=131)
        if poisoned and what == "state":
            state[1, 0, 5, 1] = float("inf")
        elif poisoned:
            rows[token, 5 if what == "x" else inner + heads * N + 2] = float("nan")
        y = torch.full((tokens, inner), 7.0, device=DEV)
        if chunks:
            scratch = torch.full(api.scan_chunks_scratch(tokens, 2, heads, heads, N), float("nan"), device=DEV)
            api.scan_chunks(rows, 0, inner, inner + heads * N, state, y, cu, slots, 2, heads, P, N, heads, scratch, fixed_decay=decays)
        else:
            api.decay_scan(rows, decays, state, y, cu, slots, 2, heads, N, P)
        outs.append((y, state))
    (clean, clean_state), (y, state), (by_token, by_token_state) = outs
    assert torch.equal(y.isfinite(), by_token.isfinite()) and torch.equal(state.isfinite(), by_token_state.isfinite())
    reached = torch.zeros(tokens, inner, dtype=torch.bool, device=DEV)
    if what == "c":
        reached[token:news[0], :P] = True         # the token's outputs; the tokens behind it in the chunk are taken one by one
    else:
        reached[token if what == "x" else 0:news[0], 5] = True
    assert torch.equal(y[~reached], clean[~reached])
    keeps = torch.ones_like(state, dtype=torch.bool)
    keeps[1, 0, :P if what == "c" else 6] = False
    assert torch.equal(state[keeps], clean_state[keeps])


@pytest.mark.parametrize("heads,D,V,columns", [(70, 128, 64, 64), (70, 128, 60, 64), (70, 128, 32, 32), (70, 64, 64, 64), (70, 64, 32, 32), (2, 128, 20, 16)])
@pytest.mark.parametrize("what,token", [("v", 100), ("v", 125), ("k", 100), ("k", 125), ("state", 0)])
def test_delta_rule_in_chunks_keeps_other_columns(heads, D, V, columns, what, token):
    """As for the scan, half of the heads with fast decays."""
    from thintensor_b200.kernels import api

    assert delta_columns(heads, 2, D, V) == columns
    news, qk = [150, 70], heads * D
    tokens = sum(news)
    cu, slots = i32([0, news[0], tokens]), i32([1, 0])
    dt_bias, a_log = torch.full((heads,), 0.5413, device=DEV), torch.tensor([-3.0, 0.5], device=DEV).repeat(heads // 2)
    outs = []
    for poisoned, chunks in ((False, True), (True, True), (True, False)):
        qkv, raw, state = randn(tokens, 2 * qk + heads * V, seed=135), randn(1, tokens, 2 * heads, seed=136), randn(2, heads, V, D, seed=137)
        raw[:, :, heads:] *= 0.1
        if poisoned and what == "state":
            state[1, 1, 5, 1] = float("inf")
        elif poisoned:
            qkv[token, 2 * qk + V + 5 if what == "v" else qk + D + 2] = float("nan")
        out = torch.full((tokens, heads * V), 7.0, device=DEV)
        if chunks:
            scratch = torch.full(api.delta_chunks_scratch(tokens, 2, heads, D, V), float("nan"), device=DEV)
            api.delta_chunks(qkv, raw, 0, heads, dt_bias, a_log, state, out, cu, slots, 2, heads, heads, D, V, scratch)
        else:
            api.delta_scan(qkv, raw, 0, heads, dt_bias, a_log, state, out, cu, slots, 2, heads, heads, D, V)
        outs.append((out, state))
    (clean, clean_state), (out, state), (by_token, by_token_state) = outs
    assert torch.equal(out.isfinite(), by_token.isfinite()) and torch.equal(state.isfinite(), by_token_state.isfinite())
    reached = torch.zeros(tokens, heads * V, dtype=torch.bool, device=DEV)
    reached[token:news[0], slice(V, 2 * V) if what == "k" else V + 5] = True
    assert torch.equal(out[~reached], clean[~reached])
    keeps = torch.ones_like(state, dtype=torch.bool)
    keeps[1, 1, slice(0, V) if what == "k" else 5] = False
    assert torch.equal(state[keeps], clean_state[keeps])


@pytest.mark.parametrize("heads,D,V", [(4, 128, 128), (4, 64, 64)])
def test_delta_rule_in_chunks_is_as_close_as_token_by_token(heads, D, V):
    """As above: with lengths, factors and scores in float32 throughout the outputs were a seventh to a third further off."""
    from thintensor_b200.kernels import api

    tokens, qk = 900, heads * D
    qkv, raw = randn(tokens, 2 * qk + heads * V, seed=125), randn(1, tokens, 2 * heads, seed=126)
    a_log, dt_bias = randn(heads, seed=127), randn(heads, seed=128)
    cu, slots = i32([0, tokens]), i32([0])
    outs = []
    for chunks in (True, False):
        state, out = torch.zeros(1, heads, V, D, device=DEV), torch.empty(tokens, heads * V, device=DEV)
        if chunks:
            scratch = torch.empty(api.delta_chunks_scratch(tokens, 1, heads, D, V), device=DEV)
            api.delta_chunks(qkv, raw, 0, heads, dt_bias, a_log, state, out, cu, slots, 1, heads, heads, D, V, scratch)
        else:
            api.delta_scan(qkv, raw, 0, heads, dt_bias, a_log, state, out, cu, slots, 1, heads, heads, D, V)
        outs.append(out.double().reshape(tokens, heads, V))
    z = raw[0].double()
    beta, decay = torch.sigmoid(z[:, :heads]), torch.exp(-torch.exp(a_log.double()) * torch.nn.functional.softplus(z[:, heads:] + dt_bias.double()))
    unit = lambda y: y / (y.square().sum(-1, keepdim=True) + 1e-6).sqrt()
    q, k = (unit(part.double().reshape(tokens, heads, D)) for part in qkv[:, :2 * qk].split(qk, 1))
    v, S, want = qkv[:, 2 * qk:].double().reshape(tokens, heads, V), torch.zeros(heads, V, D, dtype=torch.float64, device=DEV), []
    for t in range(tokens):
        S = decay[t][:, None, None] * S
        S = S + (beta[t][:, None] * (v[t] - (S @ k[t][:, :, None])[..., 0]))[:, :, None] * k[t][:, None, :]
        want.append((S @ q[t][:, :, None])[..., 0] * D ** -0.5)
    want = torch.stack(want)
    chunked, by_token = (float((out - want).norm() / want.norm()) for out in outs)
    assert chunked <= 1.05 * by_token, (chunked, by_token)


DECAYS = [0.9999, 0.999, 0.99, 0.95, 0.9, 0.8, 0.7, 0.5, 0.3, 0.1, 0.05]


def closeness(outs, want, heads):
    """Relative errors [outputs, states] of every decay's heads, in chunks and token by token."""
    result = []
    for got, exact in zip(zip(*outs), want):
        exact = exact.reshape(-1, len(DECAYS), heads // len(DECAYS), exact[0, 0].numel())
        result.append([((o.reshape(exact.shape) - exact).square().sum((0, 2, 3)) / exact.square().sum((0, 2, 3))).sqrt().cpu() for o in got])
    return result


@pytest.mark.parametrize("tokens", [357, 130, 80])
@pytest.mark.parametrize("P,N", [(16, 128), (32, 100), (64, 128), (50, 70), (128, 128), (100, 128), (32, 64), (64, 64), (128, 40)])
def test_recurrence_in_chunks_of_every_decay(P, N, tokens):
    """Outputs and states of slow and of fast decays, each decay's heads by themselves, against 64 bits: no further off than token by token but for a twentieth.
    (States that hold only the last few tokens were up to 2.3 times as far off: the tensor cores truncate their sums.)"""
    from thintensor_b200.kernels import api

    copies = 12
    heads = copies * len(DECAYS)
    inner = heads * P
    assert scan_columns(heads, 1, P, N) == {(16, 128): 16, (32, 100): 32, (64, 128): 64, (50, 70): 64, (128, 128): 128, (100, 128): 128, (32, 64): 32, (64, 64): 64, (128, 40): 128}[P, N]
    rows, decays = randn(tokens, inner + 2 * heads * N, seed=170), torch.tensor(DECAYS, device=DEV).repeat_interleave(copies).contiguous()
    cu, slots, outs = i32([0, tokens]), i32([0]), []
    for chunks in (True, False):
        state, y = torch.zeros(1, heads, P, N, device=DEV), torch.empty(tokens, inner, device=DEV)
        if chunks:
            scratch = torch.full(api.scan_chunks_scratch(tokens, 1, heads, heads, N), float("nan"), device=DEV)
            api.scan_chunks(rows, 0, inner, inner + heads * N, state, y, cu, slots, 1, heads, P, N, heads, scratch, fixed_decay=decays)
        else:
            api.decay_scan(rows, decays, state, y, cu, slots, 1, heads, N, P)
        outs.append((y.double().reshape(tokens, heads, P), state[0].double().reshape(1, heads, P * N)))
    x, b, c = (z.double().reshape(tokens, heads, -1) for z in rows.split((inner, heads * N, heads * N), 1))
    S, want = torch.zeros(heads, P, N, dtype=torch.float64, device=DEV), torch.empty(tokens, heads, P, dtype=torch.float64, device=DEV)
    for t in range(tokens):
        S = torch.baddbmm(decays.double()[:, None, None] * S, x[t][:, :, None], b[t][:, None, :])
        want[t] = torch.bmm(S, c[t][:, :, None])[..., 0]
    for name, (chunked, by_token) in zip(("outputs", "states"), closeness(outs, (want, S.reshape(1, heads, P * N)), heads)):
        assert bool((chunked <= 1.05 * by_token).all()), (name, chunked / by_token)


@pytest.mark.parametrize("D,V", [(128, 16), (100, 32), (128, 64), (64, 16), (64, 32), (40, 50)])
def test_delta_rule_in_chunks_of_every_decay(D, V):
    """As above.  A state's error is mostly that of the last rows that went into it, a few numbers a head, so states of fast decays are compared in the mean over
    lengths and decays (0.83 to 1.02 at a length; 1.04 to 1.23 with their sums on the tensor cores)."""
    from thintensor_b200.kernels import api

    copies, fast = 12, []
    heads = copies * len(DECAYS)
    assert delta_columns(heads, 1, D, V) == {(128, 16): 16, (100, 32): 32, (128, 64): 64, (64, 16): 16, (64, 32): 32, (40, 50): 64}[D, V]
    qk = heads * D
    decays = torch.tensor(DECAYS, dtype=torch.float64, device=DEV).repeat_interleave(copies)
    a_log, dt_bias = torch.log(-torch.log(decays)).float(), torch.full((heads,), 0.5413248546, device=DEV)
    for tokens in (357, 130, 80):
        qkv, raw = randn(tokens, 2 * qk + heads * V, seed=175), randn(1, tokens, 2 * heads, seed=176)
        raw[:, :, heads:] = 0.0                            # softplus(0 + 0.5413) = 1: a decay is exp(-exp(a_log))
        cu, slots, outs = i32([0, tokens]), i32([0]), []
        for chunks in (True, False):
            state, out = torch.zeros(1, heads, V, D, device=DEV), torch.empty(tokens, heads * V, device=DEV)
            if chunks:
                scratch = torch.full(api.delta_chunks_scratch(tokens, 1, heads, D, V), float("nan"), device=DEV)
                api.delta_chunks(qkv, raw, 0, heads, dt_bias, a_log, state, out, cu, slots, 1, heads, heads, D, V, scratch)
            else:
                api.delta_scan(qkv, raw, 0, heads, dt_bias, a_log, state, out, cu, slots, 1, heads, heads, D, V)
            outs.append((out.double().reshape(tokens, heads, V), state[0].double().reshape(1, heads, V * D)))
        z = raw[0].double()
        beta, decay = torch.sigmoid(z[:, :heads]), torch.exp(-torch.exp(a_log.double()) * torch.nn.functional.softplus(z[:, heads:] + dt_bias.double()))
        unit = lambda y: y / (y.square().sum(-1, keepdim=True) + 1e-6).sqrt()
        q, k = (unit(part.double().reshape(tokens, heads, D)) for part in qkv[:, :2 * qk].split(qk, 1))
        v, S = qkv[:, 2 * qk:].double().reshape(tokens, heads, V), torch.zeros(heads, V, D, dtype=torch.float64, device=DEV)
        want = torch.empty(tokens, heads, V, dtype=torch.float64, device=DEV)
        for t in range(tokens):
            S = decay[t][:, None, None] * S
            S = torch.baddbmm(S, (beta[t][:, None] * (v[t] - torch.bmm(S, k[t][:, :, None])[..., 0]))[:, :, None], k[t][:, None, :])
            want[t] = torch.bmm(S, q[t][:, :, None])[..., 0] * D ** -0.5
        (chunked, by_token), (state_chunked, state_by_token) = closeness(outs, (want, S.reshape(1, heads, V * D)), heads)
        assert bool((chunked <= 1.1 * by_token).all()), (tokens, chunked / by_token)
        slow = [i for i, d in enumerate(DECAYS) if d >= 0.95]
        assert bool((state_chunked <= 1.1 * state_by_token)[slow].all()), (tokens, state_chunked / state_by_token)
        fast.append((state_chunked / state_by_token)[[i for i, d in enumerate(DECAYS) if d <= 0.7]])
    assert float(torch.stack(fast).mean()) <= 1.03, fast


# --------------------------------------------------------------------------------- experts' products of sorted tokens
@pytest.mark.parametrize("tokens,top,experts,hidden,inter", [(1, 1, 1, 64, 128), (300, 2, 3, 72, 128), (513, 4, 16, 256, 256), (1500, 1, 5, 264, 384), (200, 3, 70, 128, 128)])
def test_experts_of_sorted_tokens(tokens, top, experts, hidden, inter):
    """Experts without tokens, with one, with whole tiles of 256 and a remainder; choices that a token does not have; widths that end inside a tile."""
    from thintensor_b200.kernels import api

    g = torch.Generator(device=DEV).manual_seed(tokens + experts)
    order = torch.rand(tokens, experts, generator=g, device=DEV)
    order[:, 0] += 0.3                                     # an expert with most tokens
    if experts > 2:
        order[:, 1] = -1.0                                 # one that nobody chose
    chosen = order.topk(top, 1).indices.int()
    if top > 1:
        chosen[::7, top - 1] = -1
    x, w = randn(tokens, hidden, seed=140).bfloat16(), randn(2 * experts * inter, hidden, seed=141, scale=hidden ** -0.5).bfloat16()
    down, weights = randn(hidden, experts * inter, seed=142, scale=inter ** -0.5).bfloat16(), torch.rand(tokens, top, generator=g, device=DEV)
    weights[::5] = 0.0
    tiles = api.expert_tiles(tokens, top, experts)
    xs = torch.full((256 * tiles, hidden), 7.0, dtype=torch.bfloat16, device=DEV)
    place, table = torch.full((tokens, top), 99, dtype=torch.int32, device=DEV), torch.full((1 + experts + tiles,), 99, dtype=torch.int32, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    api.sort_tokens(x, chosen, experts, xs, place, table)
    counts = torch.stack([(chosen == e).sum() for e in range(experts)])
    padded = (counts + 255) // 256 * 256
    first = padded.cumsum(0) - padded
    assert int(table[0]) == int(padded.sum()) // 256 and torch.equal(table[1:1 + experts].long(), counts)
    assert torch.equal(table[1 + experts:1 + experts + int(table[0])].long(), torch.arange(experts, device=DEV).repeat_interleave(padded // 256))
    for e in range(experts):
        mine = chosen == e
        rows = first[e] + torch.arange(int(counts[e]), device=DEV)
        assert torch.equal(place[mine].long(), rows)       # in the tokens' order
        assert torch.equal(xs[rows], x[mine.any(1)])
    assert bool((place[chosen < 0] == -1).all())
    act = torch.full((256 * tiles, inter), float("nan"), dtype=torch.bfloat16, device=DEV)
    api.gemm_tcgen05_experts(xs, w, act, status, hidden, inter, experts, table, "silu", experts * inter)
    y = torch.full((256 * tiles, hidden), float("nan"), device=DEV)
    api.gemm_tcgen05_experts(act, down, y, status, inter, hidden, experts, table)
    out = randn(tokens, hidden, seed=143)
    want = out.double()
    api.combine_experts(y, place, weights, out)
    assert int(status) == 0
    gate, up = (m.double().view(experts, inter, hidden) for m in w.chunk(2))
    for t, c in ((t, c) for t in list(range(0, tokens, 61)) + [tokens - 1] for c in range(top)):
        e = int(chosen[t, c])
        if e < 0:
            continue
        z = gate[e] @ x[t].double()
        made = z * torch.sigmoid(z) * (up[e] @ x[t].double())
        got = act[place[t, c]].double()
        # one rounding to bfloat16 of a float32 sum, and the epilogue's fast exponential
        torch.testing.assert_close(got, made, rtol=2.0 ** -7, atol=2.0 ** -9 * float(made.abs().max()))
        product = down.double()[:, e * inter:(e + 1) * inter] @ got
        torch.testing.assert_close(y[place[t, c]].double(), product, rtol=1e-4, atol=1e-4 * float(product.abs().max()))
    for c in range(top):
        has = (chosen[:, c] >= 0) & (weights[:, c] != 0)
        want[has] += weights[has, c, None].double() * y[place[has, c].long()].double()
    torch.testing.assert_close(out.double(), want, rtol=1e-5, atol=1e-5)


def test_sorted_tokens_without_choices():
    """Nobody chose: no tiles, and the products' look at the first tile's expert finds one; the sums stay as they are."""
    from thintensor_b200.kernels import api

    tokens, top, experts, hidden, inter = 300, 2, 3, 128, 128
    x, chosen = randn(tokens, hidden, seed=145).bfloat16(), torch.full((tokens, top), -1, dtype=torch.int32, device=DEV)
    tiles = api.expert_tiles(tokens, top, experts)
    xs, place = torch.zeros(256 * tiles, hidden, dtype=torch.bfloat16, device=DEV), torch.full((tokens, top), 99, dtype=torch.int32, device=DEV)
    table, status = torch.full((1 + experts + tiles,), 99, dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    api.sort_tokens(x, chosen, experts, xs, place, table)
    assert table[:2 + experts].tolist() == [0] * (2 + experts) and bool((place == -1).all())
    act, y = torch.zeros(256 * tiles, inter, dtype=torch.bfloat16, device=DEV), torch.zeros(256 * tiles, hidden, device=DEV)
    w, down = randn(2 * experts * inter, hidden, seed=146).bfloat16(), randn(hidden, experts * inter, seed=147).bfloat16()
    api.gemm_tcgen05_experts(xs, w, act, status, hidden, inter, experts, table, "silu", experts * inter)
    api.gemm_tcgen05_experts(act, down, y, status, inter, hidden, experts, table)
    out = randn(tokens, hidden, seed=148)
    api.combine_experts(y, place, torch.rand(tokens, top, device=DEV), out)
    assert torch.equal(out, randn(tokens, hidden, seed=148)) and int(status) == 0


@pytest.mark.parametrize("which", range(4))
def test_sorted_tokens_refuse_tensors_elsewhere(which):
    from thintensor_b200.kernels import api

    tokens, top, experts, hidden = 40, 2, 3, 64
    tiles = api.expert_tiles(tokens, top, experts)
    operands = [randn(tokens, hidden, seed=149).bfloat16(), torch.zeros(tokens, top, dtype=torch.int32, device=DEV), torch.zeros(256 * tiles, hidden, dtype=torch.bfloat16, device=DEV),
                torch.zeros(tokens, top, dtype=torch.int32, device=DEV), torch.zeros(1 + experts + tiles, dtype=torch.int32, device=DEV)]
    at = (0, 1, 2, 4)[which]
    operands[at] = operands[at].cpu()
    x, chosen, xs, place, table = operands
    with pytest.raises(api.KernelError, match="CUDA tensors only"):
        api.sort_tokens(x, chosen, experts, xs, place, table)


@pytest.mark.parametrize("which", ["rows", "state", "y", "scratch", "decays"])
def test_recurrences_in_chunks_refuse_tensors_elsewhere(which):
    from thintensor_b200.kernels import api

    heads, P, N, tokens = 2, 16, 32, 70
    t = {"rows": randn(tokens, heads * (P + 2 * N), seed=150), "state": torch.zeros(1, heads, P, N, device=DEV), "y": torch.zeros(tokens, heads * P, device=DEV),
         "scratch": torch.zeros(api.scan_chunks_scratch(tokens, 1, heads, heads), device=DEV), "decays": torch.full((heads,), 0.9, device=DEV)}
    t[which] = t[which].cpu()
    with pytest.raises(api.KernelError, match="CUDA tensors only"):
        api.scan_chunks(t["rows"], 0, heads * P, heads * (P + N), t["state"], t["y"], i32([0, tokens]), i32([0]), 1, heads, P, N, heads, t["scratch"], fixed_decay=t["decays"])


@pytest.mark.parametrize("shared,residual", [(0, True), (0, False), (384, True), (384, False)])
@pytest.mark.parametrize("tokens", [640, 2100])
def test_mixture_of_sorted_tokens_is_the_mixture_of_columns(shared, residual, tokens, monkeypatch):
    """The layer both ways: tokens sorted by expert, and every expert's columns for every token with weights of zero."""
    from thintensor_b200.engine.context import StepContext, Workspace
    from thintensor_b200.parts import moe

    part = moe.MixtureOfExperts(hidden=256, experts=16, top=3, inter=128, groups=4, keep=2, shared_inter=shared)
    part.bind({name: (0.06 * randn(*decl.shape, seed=150 + i)).bfloat16() for i, (name, decl) in enumerate(part.weights().items())}, torch.bfloat16, torch.device(DEV))
    x = randn(tokens, 256, seed=149).bfloat16()
    outs = []
    for by_expert in (True, False):
        stream = randn(tokens, 256, seed=148)
        ctx = StepContext(n_tokens=tokens, sequences=1, decode=False, max_new=tokens, max_total=tokens, tokens=None, cu=i32([0, tokens]), len_before=i32([0]), slots=i32([0]),
                          tables=[], act_dtype=torch.bfloat16, workspace=Workspace(torch.device(DEV)), status=torch.zeros(1, dtype=torch.int32, device=DEV))
        ctx.residual = stream if residual else None
        part.sorted_takes = lambda rows: by_expert
        monkeypatch.setattr(moe, "sorted_experts_pay", lambda *sizes: True)
        delta = part.forward(ctx, x)
        outs.append((stream if delta.tensor is None else stream + delta.tensor.sum(0)).double() - randn(tokens, 256, seed=148).double())
        assert int(ctx.status) == 0
    # activations narrowed before and after the routing weight: two roundings of 2^-9 that the other form does not share
    assert float((outs[0] - outs[1]).norm() / outs[1].norm()) < 2.0 ** -8


# --------------------------------------------------------------------------------- differential attention of prompts
@pytest.mark.parametrize("heads,kv_heads", [(16, 4), (3, 3), (6, 2), (16, 1), (2, 1)])
@pytest.mark.parametrize("news,before", [([1, 63, 64, 65, 130], [0, 0, 5, 64, 127]), ([300], [0]), ([0, 40, 0, 129], [3, 200, 0, 1])])
def test_differential_attention_in_tiles(heads, kv_heads, news, before):
    """Tiles of 128 rows whole and in part, groups that do not divide 128, contexts from earlier steps, sequences without tokens; a map with scores of one size
    and one with a few large ones."""
    from thintensor_b200.kernels import api

    tokens, sequences, width = sum(news), len(news), 8
    g = torch.Generator(device=DEV).manual_seed(heads)
    table = torch.randperm(sequences * width, generator=g, device=DEV).int().view(sequences, width).contiguous()
    k_pool = torch.randn(sequences * width, kv_heads, 64, 128, generator=g, device=DEV).bfloat16()
    v_pool = torch.randn(sequences * width, kv_heads, 128, 64, generator=g, device=DEV).bfloat16()
    q = torch.randn(tokens, heads, 2, 64, generator=g, device=DEV)
    q[:, :, 1] *= 4.0
    q = q.bfloat16().view(tokens, heads * 128)
    cu = [sum(news[:i]) for i in range(sequences + 1)]
    out, maps = torch.full((tokens, heads * 128), 7.0, dtype=torch.bfloat16, device=DEV), torch.full((2, tokens, heads, 128), float("nan"), device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    scale, lam, gain, eps = 0.125, 0.3, 0.8, 1e-5
    api.differential_attention_tcgen05(q, k_pool, v_pool, table, i32(cu), i32(before), sequences, tokens, heads, kv_heads, scale, lam, gain, eps, maps, out, status)
    assert int(status) == 0
    group = heads // kv_heads
    for s in range(sequences):
        if not news[s]:
            continue
        span, seen = slice(cu[s], cu[s + 1]), before[s] + news[s]
        keys = k_pool[table[s].long()].double().permute(1, 0, 2, 3).reshape(kv_heads, -1, 128)[:, :seen].repeat_interleave(group, 0)
        values = v_pool[table[s].long()].double().permute(1, 0, 3, 2).reshape(kv_heads, -1, 128)[:, :seen].repeat_interleave(group, 0)
        hidden = torch.arange(seen, device=DEV)[None] > before[s] + torch.arange(news[s], device=DEV)[:, None]
        made = []
        for m in range(2):
            score = torch.einsum("ihd,hjd->hij", q[span].double().view(-1, heads, 128)[:, :, 64 * m:64 * m + 64], keys[:, :, 64 * m:64 * m + 64]) * scale
            made.append(torch.einsum("hij,hjd->ihd", torch.softmax(score.masked_fill(hidden, -float("inf")), -1), values))
            # probabilities narrowed to bfloat16 (2^-9 each) and summed in float32 over values of size one
            assert float((maps[m, span].double() - made[m]).abs().max()) <= 2.0 ** -8 * float(values.abs().max())
        o = made[0] - lam * made[1]
        # the errors of both maps, carried by the division by the root mean square, and one more rounding
        norm = o.square().mean(-1, keepdim=True).add(eps).sqrt()
        want = o / norm * gain
        error = (out[span].double().view(-1, heads, 128) - want).abs()
        assert bool((error <= gain * (2.0 ** -7 * float(values.abs().max()) / norm + 2.0 ** -8 * want.abs())).all())


@pytest.mark.parametrize("news,before", [([1, 15, 16, 17, 100], [0, 3, 16, 40, 60]), ([600], [127]), ([300, 0, 212], [0, 5, 64])])
@pytest.mark.parametrize("kv_heads,head_dim,value_dim,from_keys", [(1, 64, 64, False), (3, 40, 72, False), (2, 96, 96, True)])
@pytest.mark.parametrize("dtype,gain", [(torch.bfloat16, None), (torch.float32, None), (torch.bfloat16, (0.3, 100)), (torch.float32, (0.2, 64))])
def test_heads_and_values_of_prompts(news, before, kv_heads, head_dim, value_dim, from_keys, dtype, gain):
    """The plain copy (from 256 tokens in one slice on) and the general form: queries, keys and values where they belong, nothing else written; queries times
    1 + c ln(floor((position + 1) / every) + 1) where they have a gain, whose steps the positions straddle."""
    from thintensor_b200.kernels import api

    tokens, sequences, heads, width = sum(news), len(news), 7, 12
    cols = (heads + kv_heads) * head_dim + (0 if from_keys else kv_heads * value_dim)
    proj = randn(1, tokens, cols, seed=160)
    table = torch.randperm(sequences * width, device=DEV).int().view(sequences, width).contiguous()
    k_pool = torch.full((sequences * width, kv_heads, 64, head_dim), 7.0, dtype=dtype, device=DEV)
    v_pool = torch.full((sequences * width, kv_heads, value_dim, 64), 7.0, dtype=dtype, device=DEV)
    q, status = torch.empty(tokens, heads * head_dim, dtype=dtype, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    cu = [sum(news[:i]) for i in range(sequences + 1)]
    api.qk_norm_rope_append(proj, None, None, 0.0, torch.zeros(1, device=DEV), 0, False, 1.0, q, k_pool, v_pool, table, i32(cu), i32(before), sequences, tokens, heads,
                            kv_heads, head_dim, value_dim, status, q_gain=gain, **({"value_from_keys": True} if from_keys else {}))
    assert int(status) == 0
    want = torch.full_like(v_pool, 7.0)
    at = heads * head_dim + (0 if from_keys else kv_heads * head_dim)
    values = proj.sum(0)[:, at:at + kv_heads * value_dim].to(dtype).view(tokens, kv_heads, value_dim)
    for s in range(sequences):
        for i in range(news[s]):
            place = before[s] + i
            want[int(table[s, place // 64]), :, :, place % 64] = values[cu[s] + i]
    assert torch.equal(v_pool, want)
    keys = torch.full_like(k_pool, 7.0)
    made = proj.sum(0).to(dtype)
    if gain is None:
        assert torch.equal(q, made[:, :heads * head_dim])
    else:
        at = torch.cat([torch.arange(news[s], device=DEV) + before[s] for s in range(sequences)]).double()
        factor = 1.0 + gain[0] * torch.log(torch.floor((at + 1) / gain[1]) + 1)
        # the factor in float32 (a logarithm's error, a product and a sum), one product, and where queries are narrow one more rounding: half a unit of 8 bits, 2^-8
        want_q = proj[0][:, :heads * head_dim].double() * factor[:, None]
        assert bool(((q.double() - want_q).abs() <= (4 * 2.0 ** -24 + (2.0 ** -8 if dtype == torch.bfloat16 else 0.0)) * want_q.abs()).all())
    for s in range(sequences):
        for i in range(news[s]):
            place = before[s] + i
            keys[int(table[s, place // 64]), :, place % 64] = made[cu[s] + i, heads * head_dim:(heads + kv_heads) * head_dim].view(kv_heads, head_dim)
    assert torch.equal(k_pool, keys)
