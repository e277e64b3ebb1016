"""Which planned calls go to the kernel whose tensor-core tiles have keys as their rows: what the library says
(``b200attn_decode_keys_as_rows``, the function that the launch uses) against ``utils/launch_config.keyrows_suit``, by which the tests of that
kernel choose their sizes.  Host arithmetic; no GPU."""
import ctypes as C

import pytest

from test_decode_routes import PLANNER, SMS


def _args(layout, dtype, batch, qh, kvh, d, keys, m, page=16, cache=None):
    from kernels import _native

    a = _native.DecodeArgs()
    a.layout = {"dense": _native.DENSE, "ragged": _native.RAGGED, "paged": _native.PAGED}[layout]
    a.dtype = {"fp16": _native.F16, "bf16": _native.BF16, "fp32": _native.F32}[dtype]
    a.batch, a.q_heads, a.kv_heads, a.head_dim, a.q_len = batch, qh, kvh, d, m
    a.max_kv = keys
    a.page_size, a.table_stride = page, -(-keys // page)
    a.total_kv = batch * keys if cache is None else cache
    return a


def _ask(a, static=False, sms=SMS):
    from kernels import _native

    lib = _native.lib()
    return lib.b200attn_decode_route(C.byref(a), sms, int(static)), lib.b200attn_decode_keys_as_rows(C.byref(a), sms, int(static))


def _says(layout, a, sms=SMS):
    from utils.launch_config import decode_pass_group, keyrows_suit

    keys = a.total_kv if layout == "ragged" else a.batch * (a.max_kv if layout == "dense" else a.table_stride * a.page_size)
    rows = decode_pass_group(a.q_heads // a.kv_heads, a.q_len) * a.q_len
    return keyrows_suit(sms, a.batch, a.kv_heads, rows, keys, a.head_dim, *((a.page_size, a.total_kv) if layout == "paged" else ()),
                        equal=layout == "dense")


@pytest.mark.parametrize("layout", ["dense", "ragged", "paged"])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("g,m", [(1, 16), (17, 1), (8, 3), (8, 5), (20, 2), (8, 8), (13, 5), (16, 8)])
def test_the_rule_is_the_librarys(layout, d, g, m):
    """Either side of each line: rows, sequences for the SMs, keys of a sequence and of an SM, boxes of pages."""
    chosen = 0
    for kvh in (1, 2, 8):
        for batch in (1, 13, 18, 19, 60, 73, 74, 75, 97, 100, 148, 149, 200, 400):
            for keys in (20, 250, 511, 512, 513, 1000, 1023, 1024, 1025, 1500, 2047, 2048, 2049, 4100, 9000, 20000):
                for page in (4, 8, 12, 16, 24, 256) if layout == "paged" else (16,):
                    for sms in (148, 132):
                        a = _args(layout, "bf16", batch, g * kvh, kvh, d, keys, m, page)
                        route, key_rows = _ask(a, sms=sms)
                        assert key_rows == (route == PLANNER and _says(layout, a, sms)), (kvh, batch, keys, page, sms)
                        chosen += key_rows
    assert (chosen > 0) == (16 < g * m <= 64)


@pytest.mark.parametrize("rows,d,keys", [((20, 2), 128, 1000), ((8, 5), 128, 1280), ((8, 8), 64, 1569)])
def test_other_types_and_arrays(rows, d, keys):
    g, m = rows
    for dtype, static, want in (("bf16", False, 1), ("fp16", False, 1), ("fp32", False, 1), ("bf16", True, 1), ("fp32", True, 0)):
        a = _args("dense", dtype, 100, g, 1, d, keys, m)       # (fp32 drafts are copied to fp16, but not for the library's own array)
        assert _ask(a, static) == (PLANNER, want), (dtype, static)


def test_calls_that_plan_for_themselves_or_mean_nothing():
    route, key_rows = _ask(_args("dense", "bf16", 10, 64, 8, 128, 2590, 5))
    assert route != PLANNER and key_rows == 0
    assert _ask(_args("dense", "bf16", 10, 64, 8, 128, 2590, 5), static=True) == (PLANNER, 0)       # the same call's plan, by a launch
    for bad in (dict(kv_heads=0), dict(q_len=0), dict(head_dim=0), dict(head_dim=96)):
        a = _args("dense", "bf16", 100, 40, 1, 128, 2000, 1)
        for name, value in bad.items():
            setattr(a, name, value)
        assert _ask(a)[1] < 0, bad


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("kvh,batch", [(8, 16), (8, 64), (8, 256), (2, 64), (2, 256), (1, 320)])
def test_a_cache_holds_no_more_keys_than_it_has_rows(kvh, batch, d):
    """Wide tables in front of a cache that only has room for short sequences: what counts is the cache, to a key."""
    line = (192 if batch * kvh <= SMS else 384) * 128 // d * batch
    never = d == 64 and batch * kvh <= SMS
    if batch * kvh > SMS:
        line = max(line, -(-1536 * 128 * SMS // (kvh * d)))
    for cache in (0, batch * 20, line - 1, line, batch * 8192):
        a = _args("paged", "bf16", batch, 8 * kvh, kvh, d, 8192, 5, cache=cache)
        route, key_rows = _ask(a)
        assert route == PLANNER and key_rows == _says("paged", a) == (cache >= line and not never), cache
    # a longer table does not make such sequences longer
    assert _ask(_args("paged", "bf16", batch, 8 * kvh, kvh, d, 1 << 20, 5, cache=batch * 20)) == (PLANNER, 0)


@pytest.mark.parametrize("kvh", [1, 2])
def test_short_heads_want_a_sequence_for_an_sm(kvh):
    """At head_dim 64, up to one pair an SM: only sequences of one length that two thirds of the SMs have one of."""
    for batch in (96 // kvh, 98 // kvh, 100 // kvh, 148 // kvh, 150 // kvh):
        for layout in ("dense", "ragged", "paged"):
            route, key_rows = _ask(_args(layout, "bf16", batch, 8 * kvh, kvh, 64, 9000, 5))
            pairs = batch * kvh
            assert route == PLANNER and key_rows == (pairs > SMS or (layout == "dense" and 3 * pairs >= 2 * SMS)), (batch, layout)
