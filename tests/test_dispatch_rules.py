"""Which form of a kernel takes a prompt: the rules at the sizes where their lines lie (no GPU)."""
from __future__ import annotations

import pytest
import torch

SMS = 148


@pytest.mark.parametrize("tokens,sequences,pays", [(2048, 1, True), (224, 1, True), (223, 1, False), (500, 5, False), (1000, 5, False), (1119, 5, False), (1120, 5, True), (1, 1, False)])
def test_maps_in_tiles(tokens, sequences, pays):
    """224 tokens a sequence on average."""
    from thintensor_b200.parts.attention_forms import tiled_maps_pay

    assert tiled_maps_pay(tokens, sequences) is pays


@pytest.mark.parametrize("tokens,experts,top,hidden,inter,pays", [
    (512, 16, 4, 2048, 1024, False), (700, 16, 4, 2048, 1024, True), (4096, 16, 4, 2048, 1024, True), (700, 16, 4, 1024, 1024, False), (2048, 16, 4, 1024, 1024, True),
    (300, 64, 6, 2048, 1024, False), (400, 64, 6, 2048, 1024, True), (1, 16, 4, 2048, 1024, False), (4096, 4, 4, 2048, 1024, False), (100000, 8, 8, 4096, 4096, False),
])
def test_experts_of_sorted_tokens(tokens, experts, top, hidden, inter, pays):
    """12 G multiply-adds saved in each matrix; never where every token chooses every expert."""
    from thintensor_b200.parts.moe import sorted_experts_pay

    assert sorted_experts_pay(tokens, experts, top, hidden, inter) is pays


def test_sorted_tokens_of_the_least_size_that_pays():
    """The line itself: tokens x experts less the rows of whole tiles, times the two widths."""
    from thintensor_b200.parts.moe import sorted_experts_pay

    least = next(tokens for tokens in range(1, 5000) if sorted_experts_pay(tokens, 16, 4, 2048, 1024))
    saved = lambda tokens: (tokens * 16 - max(tokens * 4 + 128 * 16, 256 * 16)) * 2048 * 1024
    assert saved(least - 1) < 12_000_000_000 <= saved(least) and all(sorted_experts_pay(tokens, 16, 4, 2048, 1024) for tokens in range(least, 5000))


@pytest.mark.parametrize("tokens,features,k,pays", [(16, 4096, 4096, False), (17, 1024, 1024, True), (17, 1024, 1023, False), (4000, 512, 2047, False), (193, 16384, 64, True), (193, 256, 2048, False)])
def test_products_in_parts(tokens, features, k, pays):
    from thintensor_b200.kernels import api

    assert api.gemm_split_pays(tokens, features, k) is pays


@pytest.mark.parametrize("tokens,sequences,ctas,pays", [
    (128, 1, 32, True), (127, 1, 32, False), (128, 1, 3 * SMS, True), (128, 1, 3 * SMS + 1, False), (349, 1, 3 * SMS + 1, False), (350, 1, 3 * SMS + 1, True),
    (5000, 1, 13 * SMS // 2, True), (5000, 1, 13 * SMS // 2 + 1, False), (640, 5, 64, True), (639, 5, 64, False), (64, 64, 4096, False),
])
def test_scans_in_chunks(tokens, sequences, ctas, pays):
    from thintensor_b200.parts.recurrent import scan_chunks_pay

    assert scan_chunks_pay(tokens, sequences, ctas, SMS) is pays


@pytest.mark.parametrize("tokens,sequences,ctas,keys,pays", [
    (127, 1, 64, 128, False), (128, 1, 64, 128, True), (128, 1, 64, 64, True), (128, 1, 3 * SMS, 64, True), (128, 1, 4 * SMS, 64, False), (320, 1, 4 * SMS, 64, True), (128, 1, 4 * SMS, 128, True),
    (4000, 1, 768, 128, False), (256, 1, 6 * SMS, 128, True), (255, 1, 6 * SMS, 128, False), (4000, 1, 6 * SMS, 64, False), (4000, 1, 14 * SMS, 128, True), (4000, 1, 15 * SMS, 128, False),
])
def test_delta_rule_in_chunks(tokens, sequences, ctas, keys, pays):
    from thintensor_b200.parts.recurrent import delta_chunks_pay

    assert delta_chunks_pay(tokens, sequences, ctas, keys, SMS) is pays


def test_tokens_are_sorted_where_the_kernels_take_them():
    """Rows side by side, bfloat16, whole tiles of 128 rows an expert, plainly gated experts; everything else multiplies every token as before."""
    from thintensor_b200.parts import moe

    def mixture(**changes):
        sizes = {"hidden": 256, "experts": 16, "top": 3, "inter": 128, "groups": 4, "keep": 2, "shared_inter": 0, **changes}
        part = moe.MixtureOfExperts(**sizes)
        part.bind({name: torch.zeros(*decl.shape, dtype=torch.bfloat16) for name, decl in part.weights().items()}, torch.bfloat16, torch.device("cpu"))
        return part

    wide = torch.zeros(40, 512, dtype=torch.bfloat16)
    x = torch.zeros(40, 256, dtype=torch.bfloat16)
    assert mixture().sorted_takes(x) and mixture(shared_inter=384).sorted_takes(x)
    for rows in (wide[:, :256], wide[:, 8:264], wide[::2, :256], x.float()):
        assert not mixture().sorted_takes(rows)
    assert not mixture(inter=96).sorted_takes(x) and not mixture(shared_inter=100).sorted_takes(x)
    assert not mixture(activation="clamped", limit=1.0).sorted_takes(x)
