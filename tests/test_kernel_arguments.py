"""What the entry points refuse before anything is launched, and the rules that choose between kernels (no GPU)."""
import pytest
import torch

from thintensor_b200.kernels import api


def off_by_one_number(count: int) -> torch.Tensor:
    """``count`` float32 numbers that do not start on a 16-byte boundary."""
    return torch.zeros(count + 4)[1:1 + count]


def test_scratch_that_is_copied_in_16_byte_pieces_is_aligned():
    tokens, heads, P, N = 70, 2, 8, 8
    cu, slots = torch.tensor([0, tokens], dtype=torch.int32), torch.zeros(1, dtype=torch.int32)
    rows, state, out = torch.zeros(tokens, heads * P + 2 * heads * N), torch.zeros(1, heads, P, N), torch.zeros(tokens, heads * P)
    scratch = off_by_one_number(api.scan_chunks_scratch(tokens, 1, heads, heads)[0])
    with pytest.raises(api.KernelError, match="16-byte boundary"):
        api.scan_chunks(rows, 0, heads * P, heads * (P + N), state, out, cu, slots, 1, heads, P, N, heads, scratch, fixed_decay=torch.ones(heads))
    qkv, proj, vector = torch.zeros(tokens, heads * (2 * N + P)), torch.zeros(1, tokens, 2 * heads), torch.zeros(heads)
    scratch = off_by_one_number(api.delta_chunks_scratch(tokens, 1, heads, N, P)[0])
    with pytest.raises(api.KernelError, match="16-byte boundary"):
        api.delta_chunks(qkv, proj, 0, heads, vector, vector, state, out, cu, slots, 1, heads, heads, N, P, scratch)


@pytest.mark.parametrize("sequences,each,ctas,chunks", [
    (1, 100, 64, False), (1, 160, 64, True), (4, 160, 256, True), (5, 160, 444, True),
    (8, 160, 512, False), (32, 160, 512, False), (32, 320, 512, False), (8, 640, 512, True), (4, 1024, 512, True), (16, 700, 1024, False),
])
def test_which_prompts_scan_in_chunks(sequences, each, ctas, chunks):
    """At sizes that were measured both ways the faster form is taken."""
    from thintensor_b200.parts.recurrent import scan_chunks_pay

    assert scan_chunks_pay(sequences * each, sequences, ctas, 148) == chunks


@pytest.mark.parametrize("sequences,each,ctas,key_dim,chunks", [
    (1, 127, 64, 128, False), (1, 128, 64, 128, True), (8, 128, 512, 128, True), (8, 128, 512, 64, False), (8, 320, 512, 64, True),
    (8, 128, 768, 128, False), (8, 320, 768, 128, False), (16, 320, 1024, 128, True), (16, 500, 1024, 64, False),
    (32, 256, 2048, 64, False), (64, 128, 4096, 128, False), (64, 200, 4096, 128, False), (64, 200, 4096, 64, False),
])
def test_which_prompts_take_the_delta_rule_in_chunks(sequences, each, ctas, key_dim, chunks):
    from thintensor_b200.parts.recurrent import delta_chunks_pay

    assert delta_chunks_pay(sequences * each, sequences, ctas, key_dim, 148) == chunks


@pytest.mark.parametrize("decay,chunks", [((0.9, 1.0), True), ((-1.0, 0.0), True), ((0.9, 1.0001), False), ((-8.0, 0.5), False), ((float("nan"), 0.5), False)])
def test_decays_beyond_one_go_token_by_token(decay, chunks):
    from thintensor_b200.parts.recurrent import DecayLinearAttention

    assert DecayLinearAttention(hidden=64, heads=2, key_dim=16, value_dim=16, decay=decay).chunks == chunks
