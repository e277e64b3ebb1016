"""Short calls of the tcgen05 decode kernel (more than sixteen q rows per KV head) go without the planner's launch: both sides of the
lines that part them from the rest (96 pairs of sequence and KV head; 1 024 keys less 8 for every sequence for each of two CTAs an SM),
at the edges of tiles and of items, with the merge tickets of a header word's both halves, and calls of either kind in turn."""
import pytest
import torch

from helpers import assert_close_both, spec_strict
from test_decode_planned import _route
from test_decode_routes import INLINE, PLANNER, route
from test_decode_without_planner import DEV, _call, _problem, _reference


# (8 q heads a KV head: with five drafts 40 rows.  fp32 drafts are multiplied as fp16 copies.)
@pytest.mark.parametrize("sms", [108, 148])
@pytest.mark.parametrize("dtype", ["bf16", "fp16", "fp32"])
@pytest.mark.parametrize("layout", ["dense", "ragged", "paged"])
def test_route_on_either_side_of_the_lines(layout, dtype, sms):
    def way(batch, kvh, keys, m=5, static=False):
        return route(layout, dtype, batch, 8 * kvh, kvh, 128, keys, m=m, page=1, sms=sms, static=static)

    for batch, kvh in ((96, 1), (12, 8), (1, 96), (2, 48)):
        assert way(batch, kvh, 100) == INLINE
        assert way(batch, kvh, 100, static=True) == PLANNER
    for batch, kvh in ((97, 1), (13, 8), (1, 97), (7, 14)):
        assert way(batch, kvh, 100) == PLANNER
    for batch, kvh in ((1, 1), (1, 8), (3, 2), (10, 8), (60, 1), (90, 1)):
        line = _line(batch, kvh, sms)
        assert way(batch, kvh, line) == INLINE
        assert way(batch, kvh, line + 1) == PLANNER
        from utils.launch_config import tcgen05_plans_itself

        assert tcgen05_plans_itself(sms, batch, kvh, batch * line) and not tcgen05_plans_itself(sms, batch, kvh, batch * (line + 1))
    # sixteen rows are another kernel's, without a line of keys
    assert way(1, 8, 100000, m=2) == INLINE


def _line(batch, kvh, sms):
    """The most keys of a sequence, all of one length."""
    return (1024 - 8 * batch) * 2 * sms // kvh // batch


def _check(lens, qh, kvh, d, m, dtype, layout, page=16, calls=2, want=None):
    if want is not None:
        assert _route(lens, layout, dtype, qh, kvh, d, m, page) == want
    gen = torch.Generator().manual_seed(len(lens) * 31 + m)
    problem = _problem(gen, lens, qh, kvh, d, dtype, m)
    ref = _reference(*problem, qh, kvh, m)
    for _ in range(calls):
        out = _call(*problem, layout, m, page)
        # (fp32 is multiplied with ten mantissa bits here: the bound for that)
        assert_close_both(out, ref, dtype, max(lens), f"{layout} {len(lens)}x{kvh} m{m}", strict=spec_strict(dtype, qh, kvh, m))


# (8 q heads a KV head: 24, 40, 72 and 128 rows; items of 192 to 1 024 keys)
@pytest.mark.gpu
@pytest.mark.parametrize("batch,kvh", [(1, 1), (3, 1), (12, 8), (13, 8), (96, 1), (97, 1), (1, 96), (1, 97)])
@pytest.mark.parametrize("m,d", [(3, 64), (5, 128), (9, 128), (16, 64)])
@pytest.mark.parametrize("layout,page", [("dense", 0), ("ragged", 0), ("paged", 16), ("paged", 24)])
def test_pairs_and_layouts(batch, kvh, m, d, layout, page):
    base = [330] if layout == "dense" else [16, 63, 64, 65, 129, 321, 640, 1000, 2500]
    if layout == "paged" and batch >= 96:        # (a table of 2 500 keys would be beyond the line of keys)
        base = base[:7]
    lens = [base[i % len(base)] for i in range(batch)] if batch > 1 else [1500]
    _check(lens, 8 * kvh, kvh, d, m, torch.bfloat16, layout, page or 16, calls=1, want=INLINE if batch * kvh <= 96 else PLANNER)


@pytest.mark.gpu
@pytest.mark.parametrize("off", [-64, 0, 1])
@pytest.mark.parametrize("batch,kvh", [(1, 2), (5, 8)])
def test_line_of_keys(batch, kvh, off):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    _check([_line(batch, kvh, sms) + off] * batch, 8 * kvh, kvh, 64, 4, torch.float16, "dense", want=INLINE if off <= 0 else PLANNER)


@pytest.mark.gpu
def test_two_passes():
    """160 rows per KV head are two launches of 80, which draw and reset the same tickets."""
    _check([700, 64, 1300], 64, 2, 128, 5, torch.bfloat16, "ragged", want=INLINE)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32], ids=["fp16", "fp32"])
def test_one_long_sequence_and_empty_ones(dtype):
    _check([5, 9000, 5, 5, 64, 5], 16, 2, 128, 5, dtype, "ragged", want=INLINE)
    from kernels import speculative_decode_attention
    gen = torch.Generator().manual_seed(2)
    q = torch.randn((4, 8, 5, 64), generator=gen).to(dtype).to(DEV)
    k, v = (torch.randn((700, 1, 64), generator=gen).to(dtype).to(DEV) for _ in range(2))
    indptr = torch.tensor([0, 0, 700, 700, 700], dtype=torch.int32, device=DEV)
    out = speculative_decode_attention(q, k, v, kv_indptr=indptr, causal=False)
    assert not out[[0, 2, 3]].any() and bool(out[1].isfinite().all()) and bool(out[1].any())


@pytest.mark.gpu
def test_calls_of_either_kind_in_turn():
    """Planned and unplanned calls on one workspace, and unplanned ones of the warp-level kernel, whose tickets share the header."""
    gen = torch.Generator().manual_seed(8)
    shapes = [([1500, 90, 3000], 8, 1, 5), ([9000] * 14, 64, 8, 4), ([2000, 17, 640], 16, 2, 9), ([20000, 700, 3], 8, 2, 0)]
    assert [_route(lens, "ragged", torch.bfloat16, qh, kvh, 64, max(1, m)) for lens, qh, kvh, m in shapes] == [INLINE, PLANNER, INLINE, INLINE]
    problems = [(_problem(gen, lens, qh, kvh, 64, torch.bfloat16, m), qh, kvh, m, max(lens)) for lens, qh, kvh, m in shapes]
    refs = [_reference(*pr, qh, kvh, m) for pr, qh, kvh, m, _ in problems]
    for _ in range(3):
        outs = [_call(*pr, "ragged", m) for pr, qh, kvh, m, _ in problems]
        for out, ref, (_, qh, kvh, m, longest) in zip(outs, refs, problems):
            assert_close_both(out, ref, torch.bfloat16, longest, f"{qh}/{kvh} m{m}")
