"""Decode calls whose (sequence, KV head) pairs are short run without a plan: a cluster of CTAs shares a pair.  Every cluster
size, every layout, both kernels (16-bit rows, fp32), parts that are empty, ragged tile ends, rows up to a whole row tile."""
import pytest
import torch

from helpers import assert_close_both
from test_decode_without_planner import _call, _problem, _reference

pytestmark = pytest.mark.gpu

# (batch, q heads, KV heads): 8, 4, 2 and 1 CTAs per pair on 148 SMs
SHAPES = [(1, 8, 1), (1, 32, 8), (6, 32, 8), (13, 32, 8), (25, 32, 8), (60, 8, 8)]


def _lens(batch, layout, longest):
    if layout == "dense":
        return [longest] * batch
    base = [longest, 1, 63, 64, 65, 0, 129, longest // 2, longest - 1]
    return [min(longest, base[i % len(base)]) for i in range(batch)]


@pytest.mark.parametrize("batch,qh,kvh", SHAPES)
@pytest.mark.parametrize("layout,page", [("dense", 0), ("ragged", 0), ("paged", 16), ("paged", 64), ("paged", 24)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32], ids=["bf16", "fp16", "fp32"])
@pytest.mark.parametrize("d", [64, 128])
def test_sizes_and_layouts(batch, qh, kvh, layout, page, dtype, d):
    gen = torch.Generator().manual_seed(batch * 977 + qh + d)
    for longest in (5, 64, 200, 511, 1000, 2048):
        lens = _lens(batch, layout, longest)
        qs, ks, vs = _problem(gen, lens, qh, kvh, d, dtype)
        out = _call(qs, ks, vs, layout, 0, page or 16)
        keep = [i for i, n in enumerate(lens) if n > 0]
        ref = _reference([qs[i] for i in keep], [ks[i] for i in keep], [vs[i] for i in keep], qh, kvh, 0)
        assert_close_both(out[keep], ref, dtype, longest, f"{layout} {batch}x{kvh} {longest}")
        assert not out[[i for i in range(batch) if i not in keep]].any()


@pytest.mark.parametrize("batch,qh,kvh,m", [(2, 8, 8, 16), (4, 8, 2, 4), (3, 4, 4, 2), (1, 8, 1, 2), (2, 15, 3, 3)])
@pytest.mark.parametrize("layout,page", [("ragged", 0), ("paged", 16)])
def test_draft_rows(batch, qh, kvh, m, layout, page):
    """Up to sixteen rows per KV head: the owners' shares cut rows anywhere."""
    gen = torch.Generator().manual_seed(batch * 31 + m)
    lens = [max(m, n) for n in _lens(batch, layout, 700)]
    for d in (64, 128):
        for dtype in (torch.bfloat16, torch.float16):
            qs, ks, vs = _problem(gen, lens, qh, kvh, d, dtype, m)
            out = _call(qs, ks, vs, layout, m, page or 16)
            assert_close_both(out, _reference(qs, ks, vs, qh, kvh, m), dtype, max(lens), f"{layout} m{m} d{d}")


def test_one_long_among_short():
    """Packed sequences of which one holds nearly all keys."""
    gen = torch.Generator().manual_seed(4)
    lens = [3, 9000, 17, 1, 64, 200, 5, 40]
    qs, ks, vs = _problem(gen, lens, 8, 2, 64, torch.float16)
    out = _call(qs, ks, vs, "ragged", 0)
    assert_close_both(out, _reference(qs, ks, vs, 8, 2, 0), torch.float16, max(lens), "one long")


def test_nan_reaches_the_rows_that_saw_it():
    gen = torch.Generator().manual_seed(5)
    qs, ks, vs = _problem(gen, [600, 600], 8, 2, 64, torch.bfloat16)
    vs[1][100, 1, 3] = float("nan")
    out = _call(qs, ks, vs, "dense", 0)
    assert torch.isfinite(out[0]).all() and torch.isfinite(out[1, :4]).all()
    assert torch.isnan(out[1, 4:, 3]).all() and torch.isfinite(out[1, 4:, 4:]).all()


def test_calls_in_a_row_and_in_a_graph():
    """Back to back without a synchronisation, and replayed: nothing is left over from a call."""
    from kernels import decode_attention

    gen = torch.Generator(device="cuda").manual_seed(6)
    q, k, v = (torch.randn(s, generator=gen, device="cuda", dtype=torch.bfloat16) for s in ((4, 8, 128), (4, 2, 900, 128), (4, 2, 900, 128)))
    first = decode_attention(q, k, v)
    outs = [decode_attention(q, k, v) for _ in range(50)]
    assert all(torch.equal(first, o) for o in outs)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = decode_attention(q, k, v)
    for _ in range(20):
        g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, first)


@pytest.mark.parametrize("qh,kvh", [(16, 1), (17, 1), (64, 1), (128, 1), (96, 2)])
def test_fp32_rows_either_side_of_the_line(qh, kvh):
    """fp32 decode takes any number of q rows per KV head; up to sixteen of them share a cluster."""
    gen = torch.Generator().manual_seed(qh)
    for d in (64, 128):
        lens = [300, 40]
        qs, ks, vs = _problem(gen, lens, qh, kvh, d, torch.float32)
        out = _call(qs, ks, vs, "ragged", 0)
        assert_close_both(out, _reference(qs, ks, vs, qh, kvh, 0), torch.float32, 300, f"fp32 {qh}/{kvh} d{d}")
