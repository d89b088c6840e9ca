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
