"""The exponent reference of a row in the prefill kernel: it stands as long as a tile's exponentials against it stay in
range and moves when they do not.  Rows whose maximum grows from tile to tile by amounts either side of every threshold,
rows whose first keys all score -inf, and rows in which both meet."""
import pytest
import torch

from kernels import flash_attention_v2

pytestmark = pytest.mark.gpu

# P is rounded to the 16-bit type (half a unit: 2^-9 bf16, 2^-12 fp16) and so is the output; with |v| = O(4) the largest
# difference stays below the bars that the other tests hold these types to
ATOL = {torch.bfloat16: 2e-2, torch.float16: 1e-2, torch.float32: 4e-3}


def _check(q, k, v, causal=False):
    out = flash_attention_v2(q, k, v, is_causal=causal)
    ref = torch.nn.functional.scaled_dot_product_attention(
        q.double(), k.double().repeat_interleave(q.shape[1] // k.shape[1], 1),
        v.double().repeat_interleave(q.shape[1] // k.shape[1], 1), is_causal=causal)
    assert torch.isfinite(out).all()
    assert (out.double() - ref).abs().max().item() < ATOL[q.dtype]


def _rising(dtype, d, n, step, rows=130, growing_rows=None):
    """Scores of tile t lie step * t (log2 units) above those of tile 0, for all rows or for a few of them."""
    g = torch.Generator(device="cuda").manual_seed(int(step * 8) + n)
    q = torch.randn((1, 2, rows, d), generator=g, device="cuda")
    k = torch.randn((1, 1, n, d), generator=g, device="cuda")
    v = torch.randn((1, 1, n, d), generator=g, device="cuda")
    # the last dimension carries the offset: q there is 1 (0 for rows that do not grow), k there the offset
    q[..., -1] = 1.0
    if growing_rows is not None:
        q[..., -1] = 0.0
        q[:, :, growing_rows, -1] = 1.0
    offset = step * (torch.arange(n, device="cuda") // 128) * 0.6931472 * d ** 0.5
    k[..., -1] = offset
    return q.to(dtype), k.to(dtype), v.to(dtype)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32], ids=["bf16", "fp16", "fp32"])
@pytest.mark.parametrize("step", [0, 1, 2.9, 3.1, 5, 7.9, 8.1, 9.9, 10.1, 12, 15.5, 16.5, 40])
def test_growing_maximum(dtype, step):
    _check(*_rising(dtype, 64, 5 * 128 + 33, step))
    _check(*_rising(dtype, 128, 4 * 128, step, growing_rows=[3, 77]))


@pytest.mark.parametrize("step", [2, 6, 20])
def test_growing_maximum_causal(step):
    q, k, v = _rising(torch.bfloat16, 128, 700, step, rows=700)
    _check(q, k, v, causal=True)


def test_falling_maximum():
    q, k, v = _rising(torch.bfloat16, 128, 6 * 128, 7)
    _check(q, k.flip(2).contiguous(), v)


@pytest.mark.parametrize("first", [1, 127, 128, 129, 256, 300])
@pytest.mark.parametrize("step", [0, 4, 12])
def test_first_keys_at_minus_infinity(first, step):
    q, k, v = _rising(torch.bfloat16, 128, 512, step)
    q[..., 0] = 1e20
    k[..., 0] = 0.0
    k[:, :, :first, 0] = -1e20      # products of -1e40: -inf in the fp32 accumulator
    out = flash_attention_v2(q, k, v)
    # (in 64 bits the product is finite and the weight 0 all the same)
    ref = torch.nn.functional.scaled_dot_product_attention(q.double(), k.double().expand(-1, 2, -1, -1), v.double().expand(-1, 2, -1, -1))
    assert torch.isfinite(out).all()
    assert (out.double() - ref).abs().max().item() < ATOL[q.dtype]
