"""Which way a prefill call goes: items whole, shared by the CTAs of a cluster, or cut into parts of the workspace.  The rule is host
arithmetic of the library and is checked without a GPU."""
import ctypes as C

import pytest

WHOLE, WORKSPACE = 1, 32          # include/b200attn.h
SMS = 148


def route(layout, dtype, batch, qh, kvh, lq, lkv, causal, d, page=16, sms=SMS):
    """``lkv``: keys of a sequence (dense, ragged) or of the block table (paged)."""
    from kernels import _native

    a = _native.PrefillArgs()
    a.layout = {"dense": _native.DENSE, "ragged": _native.RAGGED, "paged": _native.PAGED}[layout]
    a.dtype = {"fp16": _native.F16, "bf16": _native.BF16, "fp32": _native.F32}[dtype]
    a.batch, a.q_heads, a.kv_heads, a.head_dim, a.max_q, a.max_kv = batch, qh, kvh, d, lq, lkv
    a.total_q, a.total_kv, a.page_size, a.table_stride = batch * lq, batch * lkv, page, -(-lkv // page)
    a.is_causal = int(causal)
    return _native.lib().b200attn_prefill_route(C.byref(a), sms)


def test_arguments_that_mean_nothing_are_refused():
    assert route("dense", "bf16", 1, 8, 0, 128, 128, False, 64) < 0
    assert route("dense", "bf16", 1, 7, 2, 128, 128, False, 64) < 0
    assert route("dense", "bf16", 1, 8, 2, 128, 128, False, 64, sms=0) < 0
    assert route("dense", "bf16", 0, 8, 2, 128, 128, False, 64) == WHOLE


@pytest.mark.parametrize("sms", [74, 108, 148, 160])
@pytest.mark.parametrize("d", [64, 128])
def test_clusters_are_all_resident_and_worth_it(d, sms):
    """One CTA to an SM: of 148 SMs 74, 33 and 15 clusters of two, four and eight; no part is empty when the longest item is cut."""
    held = {2: 74, 4: 33, 8: 15}
    taken = set()
    for batch in (1, 2, 3, 5, 8, 15, 16, 33, 34, 74, 75):
        for qh, kvh in ((2, 1), (2, 2), (8, 2), (32, 8)):
            for lq in (1, 100, 128, 129, 256, 700):
                for lkv in (128, 384, 512, 640, 760, 900, 1024, 1500, 4096):
                    for causal in (False, True):
                        if causal and lq != 700:
                            continue
                        for layout in ("dense", "paged"):
                            c = route(layout, "bf16", batch, qh, kvh, lq, lkv, causal, d, sms=sms)
                            items = batch * (-(-lq // 128) * qh // 2 if qh != kvh else -(-lq // 256) * qh)
                            if c <= 8:
                                assert c in (1, 2, 4, 8)
                                if c > 1:
                                    taken.add(c)
                                    assert items <= held[c] * sms // 148
                                    tiles = -(-lkv // 128) if not causal else min(-(-lkv // 128), -(-lq // 128))
                                    assert tiles >= c and tiles >= 4
                            else:
                                assert WORKSPACE + 2 <= c <= WORKSPACE + 8
                        assert route("ragged", "bf16", batch, qh, kvh, lq, lkv, causal, d, sms=sms) == WHOLE
    assert taken == ({2, 4, 8} if d == 64 else {4, 8})      # (at head_dim 128 two parts in the workspace are cheaper than in a cluster)
