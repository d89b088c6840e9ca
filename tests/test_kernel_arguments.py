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
