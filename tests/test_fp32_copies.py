"""fp32 calls that multiply in 16 bits read fp16 copies of q, k and v: four 16-byte pieces per thread, 256 threads per block,
tensors of different lengths in one launch."""
import pytest
import torch

from kernels import flash_attention_v2, speculative_decode_attention

pytestmark = pytest.mark.gpu


# pieces of k and v (16 per key and KV head at D 64): one key, either side of a block's 1 024, several blocks and a remainder
@pytest.mark.parametrize("n", [1, 15, 63, 64, 65, 127, 129, 257, 1000, 4099])
def test_copies_of_every_length(n):
    g = torch.Generator(device="cuda").manual_seed(n)
    for qh, m in ((1, 7), (5, 64), (2, 200)):
        q, k, v = (torch.randn(s, generator=g, device="cuda") for s in ((1, qh, m, 64), (1, 1, n, 64), (1, 1, n, 64)))
        ref = torch.softmax(q.double() @ k.double().transpose(-1, -2) / 8, -1) @ v.double()
        # q, k, v and P rounded to fp16 (2^-12 each): scores off by O(2^-11), values |v| <= 5 by that much of themselves
        assert (flash_attention_v2(q, k, v).double() - ref).abs().max().item() < 4e-3
        if m <= 16:
            assert (speculative_decode_attention(q, k, v).double() - ref).abs().max().item() < 4e-3
