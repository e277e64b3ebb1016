"""The largest weight of a row against its exponent reference is exactly one where a pass starts from that weight's tile: it is the
one that rounding P to 16 bits would show most of.  fp32 calls, whose P is fp16 and whose output is not rounded: one key of the
first tile holds nearly all weight, another, alone among the columns a kernel looks at first, sets a lower reference, all
values are one.  A rounded weight would show as 2^-12, half a unit in fp16."""
import pytest
import torch

from kernels import flash_attention_v2, speculative_decode_attention

pytestmark = pytest.mark.gpu
D = 64


def _inputs(qh, m, n, key, above):
    """Scores in log2 units: 0 for key 0, ``above`` for ``key``, -40 for the others."""
    q = torch.zeros((3, qh, m, D), device="cuda")
    k = torch.zeros((3, 1, n, D), device="cuda")
    q[..., 0] = 1.0
    k[..., 0] = -40.0
    k[:, :, 0, 0] = 0.0
    # (a multiple of 1/64: exact in fp16; the scale 1/8 and log2(e) are what makes its exponential no round number)
    k[:, :, key, 0] = round(above * 0.6931472 * 8 * 64) / 64
    k[:, :, 1:, 0] = torch.where(k[:, :, 1:, 0] == -40.0, torch.tensor(-40 * 0.6931472 * 8, device="cuda").half().float(), k[:, :, 1:, 0])
    return q, k, torch.ones_like(k)


# (the weight of key 0 is 2^-above, rounded to 2^-12 of itself: 2^-12 / 2^above of the sum; the sums' own rounding is 2^-23)
@pytest.mark.parametrize("above", [5.3, 7.7, 9.1, 9.4])
@pytest.mark.parametrize("qh,m", [(5, 8), (8, 16)])
@pytest.mark.parametrize("key", [17, 40, 63])
def test_speculative_decode(above, qh, m, key):
    for n in (64, 300):
        out = speculative_decode_attention(*_inputs(qh, m, n, key, above))
        assert (out - 1).abs().max().item() <= 2.0 ** -(12 + above) * 1.1 + 2e-6


@pytest.mark.parametrize("above", [5.3, 7.7, 9.1, 9.4])
@pytest.mark.parametrize("key", [33, 70, 127])
def test_prefill(above, key):
    for n in (128, 500):
        out = flash_attention_v2(*_inputs(2, 100, n, key, above))
        assert (out - 1).abs().max().item() <= 2.0 ** -(12 + above) * 1.1 + 2e-6


@pytest.mark.parametrize("above", [2.3, 5.3, 7.7])
@pytest.mark.parametrize("key", [64, 70, 130])
def test_decode_cluster(above, key):
    """Key 0's warp meets the other key in a later tile."""
    q, k, v = _inputs(2, 4, 400, key, above)
    out = speculative_decode_attention(q[:1], k[:1], v[:1])
    assert (out - 1).abs().max().item() <= 2.0 ** -(12 + above) * 1.1 + 2e-6
