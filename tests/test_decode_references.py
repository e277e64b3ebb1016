"""The exponent reference of a row in the tcgen05 decode kernel (more than sixteen rows per KV head): it stands as long as a
tile's exponentials against it stay in range, and moves, with the accumulator in tensor memory rescaled, when they do not.
Rows whose maximum grows from tile to tile by amounts either side of every threshold, or within a unit's first tile behind the
sixteen columns that the first reference comes from; all rows or a few of one warp; falling maxima; keys at -inf; draft-causal
tails; sequences cut into parts whose references lie far apart."""
import pytest
import torch

from kernels import speculative_decode_attention

pytestmark = pytest.mark.gpu

# P and the output are rounded to the 16-bit type (half a unit: 2^-9 bf16, 2^-12 fp16; fp32 calls multiply in fp16), the values
# are |v| <= 5: an output, an average of them, is off by at most 2 * 2^-9 * 5 = 2e-2 and 2 * 2^-12 * 5 = 2.5e-3.  A row that was
# not rescaled, or twice, is off by O(1).
ATOL = {torch.bfloat16: 2e-2, torch.float16: 2.5e-3, torch.float32: 2.5e-3}
DTYPES = pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32], ids=["bf16", "fp16", "fp32"])
# (q heads, KV heads, drafts): 40 rows (two softmax warps), 24 (one), 128 (all four)
SHAPES = pytest.mark.parametrize("qh,kvh,m", [(16, 2, 5), (6, 1, 4), (16, 1, 8)])


def _check(q, k, v, causal=False):
    out = speculative_decode_attention(q, k, v, causal=causal)
    g, m, n = q.shape[1] // k.shape[1], q.shape[2], k.shape[2]
    s = q.double() @ k.double().repeat_interleave(g, 1).transpose(-1, -2) / q.shape[-1] ** 0.5
    if causal:
        hidden = torch.arange(n, device="cuda")[None] > torch.arange(n - m, n, device="cuda")[:, None]
        s = s.masked_fill(hidden, float("-inf"))
    ref = torch.softmax(s, -1) @ v.double().repeat_interleave(g, 1)
    assert torch.isfinite(out).all()
    assert (out.double() - ref).abs().max().item() <= ATOL[q.dtype]


def _rising(dtype, batch, qh, kvh, m, d, n, step, block=64, rows=None):
    """Scores of block t of `block` keys lie step * t (log2 units) above those of block 0, for all rows or for some."""
    g = torch.Generator(device="cuda").manual_seed(int(step * 8) + n + block)
    q, k, v = (torch.randn(s, generator=g, device="cuda") for s in ((batch, qh, m, d), (batch, kvh, n, d), (batch, kvh, n, d)))
    v = v.clamp(-5, 5)
    # the last dimension carries the offset: q there is 1 (0 for rows that do not grow), k there the offset
    q[..., -1] = 1.0
    if rows is not None:
        q[..., -1] = 0.0
        q.view(batch, kvh, -1, d)[:, :, rows, -1] = 1.0
    k[..., -1] = step * (torch.arange(n, device="cuda") // block) * 0.6931472 * d ** 0.5
    # (fp32 calls round to fp16: their inputs are numbers that this leaves as they are)
    return [t.half().float() if dtype == torch.float32 else t.to(dtype) for t in (q, k, v)]


@DTYPES
@SHAPES
@pytest.mark.parametrize("step", [0, 1, 2.9, 3.1, 3.9, 4.1, 5, 7.9, 9.9, 10.1, 12, 16.5, 40])
def test_growing_maximum(dtype, qh, kvh, m, step):
    _check(*_rising(dtype, 40, qh, kvh, m, 64, 12 * 64 + 33, step))                       # whole sequences
    _check(*_rising(dtype, 40, qh, kvh, m, 128, 10 * 64, step, rows=[3, 17]))             # two rows of one warp
    _check(*_rising(dtype, 1, qh, kvh, m, 128, 4096, step))                               # cut into parts


@DTYPES
@SHAPES
@pytest.mark.parametrize("step", [2.9, 5.1, 9.9, 11, 30])
def test_maximum_behind_the_first_columns(dtype, qh, kvh, m, step):
    """The first reference is the maximum of sixteen columns; the next sixteen lie above it."""
    for d in (64, 128):
        _check(*_rising(dtype, 3, qh, kvh, m, d, 64, step, block=16))
        _check(*_rising(dtype, 3, qh, kvh, m, d, 200, step, block=16, rows=[0, 5, 20]))


@DTYPES
@SHAPES
def test_falling_maximum(dtype, qh, kvh, m):
    for step in (3.5, 7, 20):
        q, k, v = _rising(dtype, 40, qh, kvh, m, 128, 8 * 64, step)
        _check(q, k.flip(2).contiguous(), v)


@SHAPES
@pytest.mark.parametrize("first", [1, 15, 16, 17, 63, 64, 65, 128, 200])
@pytest.mark.parametrize("step", [0, 4, 12])
def test_first_keys_at_minus_infinity(qh, kvh, m, first, step):
    q, k, v = _rising(torch.bfloat16, 20, qh, kvh, m, 128, 500, step)
    q[..., 0] = 1e20
    k[..., 0] = 0.0
    k[:, :, :first, 0] = -1e20      # products of -1e40: -inf in the fp32 accumulator (in 64 bits the weight is 0 all the same)
    _check(q, k, v)


@DTYPES
@SHAPES
@pytest.mark.parametrize("n", [9, 16, 63, 64, 65, 70, 129, 1000, 5000])
def test_draft_causal_tail(dtype, qh, kvh, m, n):
    for batch, step in ((2, 0), (2, 6), (40, 11)):
        if batch * n <= 50000:
            _check(*_rising(dtype, batch, qh, kvh, m, 64, n, step), causal=True)
