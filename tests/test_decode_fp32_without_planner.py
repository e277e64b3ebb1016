"""fp32 decode calls of 97 to 192 (sequence, KV head) pairs plan inside the kernel too, with merge tickets of eight bits: either side of
the line, pairs at every place of a header word, pairs of more than 128 items, calls with tickets of either width in turn."""
import pytest
import torch

from helpers import assert_close_both
from test_decode_planned import _route
from test_decode_routes import INLINE, PLANNER, route
from test_decode_without_planner import DEV, _call, _problem, _reference


@pytest.mark.parametrize("batch,kvh,want", [(12, 8, INLINE), (13, 8, INLINE), (24, 8, INLINE), (25, 8, PLANNER), (97, 1, PLANNER),
                                            (33, 3, PLANNER), (8, 13, INLINE), (96, 2, PLANNER)])
def test_route(batch, kvh, want):
    """Two bytes a ticket up to 96 pairs, one up to 192 unless a pair may be cut into more than 255 items."""
    assert route("ragged", "fp32", batch, kvh, kvh, 64, 0, total=batch * 2000) == want
    assert route("ragged", "fp32", batch, kvh, kvh, 64, 0, total=batch * 2000, static=True) == PLANNER


def test_route_of_much_data():
    assert route("dense", "fp32", 20, 8, 8, 64, 3000) == INLINE
    assert route("dense", "fp32", 20, 8, 8, 64, 6000) == PLANNER       # 469 MiB of keys and values


@pytest.mark.gpu
@pytest.mark.parametrize("batch,qh,kvh,d", [(13, 8, 8, 64), (24, 8, 8, 64), (16, 32, 8, 64), (13, 8, 8, 128), (8, 13, 13, 64)])
@pytest.mark.parametrize("layout", ["ragged", "paged"])
def test_tickets_of_eight_bits(batch, qh, kvh, d, layout):
    gen = torch.Generator().manual_seed(batch * 7 + d)
    base = [1, 63, 64, 65, 129, 2500, 640, 1500]
    lens = [base[i % len(base)] for i in range(batch)]
    lens[-1] = 9000 if layout == "ragged" else 2900          # a pair of many items (a table of 9 000 keys would be beyond 300 MiB)
    page = 16
    keys = -(-max(lens) // page) * page
    assert _route(lens, layout, torch.float32, qh, kvh, d, page=page) == INLINE
    qs, ks, vs = _problem(gen, lens, qh, kvh, d, torch.float32)
    small = _problem(gen, [700, 90, 3000], 8, 2, d, torch.float32)     # sixteen bits
    ref, small_ref = _reference(qs, ks, vs, qh, kvh, 0), _reference(*small, 8, 2, 0)
    for _ in range(2):
        out = _call(qs, ks, vs, layout, 0, page)
        other = _call(*small, layout, 0, page)
        assert_close_both(out, ref, torch.float32, keys, f"{layout} {batch}x{kvh}")
        assert_close_both(other, small_ref, torch.float32, 3000, layout)


@pytest.mark.gpu
@pytest.mark.parametrize("place", [0, 13, 27])
def test_tickets_beyond_half_of_eight_bits(place):
    """Pairs of more than 128 items, so that the highest bit of their tickets is drawn: the KV heads of one sequence, whose tickets are
    neighbours in the header."""
    from utils.launch_config import decode_items, decode_plan

    gen = torch.Generator().manual_seed(place)
    lens = [20] * 28
    lens[place] = 67000
    assert _route(lens, "ragged", torch.float32, 5, 5, 64) == INLINE
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    items = decode_items(decode_plan(sms, len(lens), 5, 5, 1, fp32=True), lens)
    assert 128 < items[place] <= 255
    qs, ks, vs = _problem(gen, lens, 5, 5, 64, torch.float32)
    ref = _reference(qs, ks, vs, 5, 5, 0)
    for _ in range(2):
        assert_close_both(_call(qs, ks, vs, "ragged", 0), ref, torch.float32, max(lens))
