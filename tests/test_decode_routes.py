"""Which way a decode call goes: clusters, items that the CTAs plan for themselves, or items behind the planner.  The rule is
host arithmetic of the library; what it may not do is checked without a GPU."""
import ctypes as C

import pytest

PLANNER, INLINE = 0, 16           # include/b200attn.h
SMS = 148


def route(layout, dtype, batch, qh, kvh, d, keys, m=1, total=None, static=False, page=16, sms=SMS):
    """``keys``: per sequence (dense), on average (ragged), of the block table (paged)."""
    from kernels import _native

    a = _native.DecodeArgs()
    a.layout = {"dense": _native.DENSE, "ragged": _native.RAGGED, "paged": _native.PAGED}[layout]
    a.dtype = {"fp16": _native.F16, "bf16": _native.BF16, "fp32": _native.F32}[dtype]
    a.batch, a.q_heads, a.kv_heads, a.head_dim, a.q_len = batch, qh, kvh, d, m
    a.max_kv = keys
    a.page_size, a.table_stride = page, -(-keys // page)
    a.total_kv = total if total is not None else batch * keys
    return _native.lib().b200attn_decode_route(C.byref(a), sms, int(static))


def test_arguments_that_mean_nothing_are_refused():
    assert route("dense", "bf16", 1, 8, 0, 64, 100) < 0
    assert route("dense", "bf16", 1, 7, 2, 64, 100) < 0
    assert route("dense", "bf16", 1, 8, 2, 64, 100, sms=0) < 0
    assert route("dense", "bf16", 0, 8, 2, 64, 100) in (PLANNER, INLINE)


# A CTA takes about 0.5 us per tile of 64 keys and 64 elements of a head in 16 bits; in fp32 0.8, 1.5, 3 and 6 us at 1, 4, 8 and 16
# rows.  A call behind the planner takes 15 to 20 us with one long sequence, one without a planner launch 10 to 15, and its
# shortest items are two tiles.  A table of pages says how long a sequence can be; that one of a packed batch has all keys is
# rare, and may cost such a call half its time.
def _tile_us(dtype, d, rows):
    if dtype != "fp32":
        return 0.46 if d == 64 else 0.8
    return (0.83 if rows == 1 else 1.1 if rows == 2 else 1.5 if rows <= 4 else 3.0 if rows <= 8 else 6.0) * d / 64


@pytest.mark.parametrize("dtype", ["bf16", "fp32"])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("rows", [1, 2, 4, 8, 16])
def test_parts_of_clusters_are_bounded(dtype, d, rows):
    """Where one packed sequence holds all keys, and where one of a paged batch fills the table."""
    for batch, kvh in ((1, 1), (2, 1), (4, 1), (16, 1), (4, 2), (16, 2), (4, 8), (13, 8), (32, 8), (100, 8)):
        for keys in (1, 20, 64, 100, 128, 250, 500, 1000, 2000, 4000, 8000):
            own = 2 * _tile_us(dtype, d, rows) if dtype == "fp32" else 0
            for layout, longest in (("ragged", batch * keys), ("paged", keys)):
                c = route(layout, dtype, batch, rows * kvh, kvh, d, keys)
                if 1 <= c <= 8:
                    part = -(--(-longest // 64) // c) * _tile_us(dtype, d, rows)
                    if layout == "paged":
                        bound = 7.5
                    elif dtype == "fp32":
                        bound = 22 if batch * kvh > 96 else 9
                    else:
                        bound = 26 if batch * kvh > 96 else 15
                    assert part <= bound + own, (layout, batch, kvh, keys, c, part)


def test_one_long_sequence_among_short_ones_is_planned():
    # 16 packed fp32 sequences, 8 rows per KV head, 8 000 keys in all: eight CTAs would take 50 us for the one that may have them
    # all; of 2 000 keys they take as long as a plan, two CTAs took 50
    for total in (4000, 8000):
        assert route("ragged", "fp32", 16, 8, 1, 64, 0, total=total) in (PLANNER, INLINE)
        assert route("ragged", "fp32", 16, 8, 2, 128, 0, total=total) in (PLANNER, INLINE)
    assert route("ragged", "fp32", 16, 8, 1, 64, 0, total=2000) in (PLANNER, INLINE, 8)
    assert route("ragged", "fp16", 16, 8, 8, 128, 0, total=8000) in (PLANNER, INLINE)
    # ... and short ones still share clusters
    assert 1 <= route("ragged", "fp16", 16, 8, 2, 64, 0, m=4, total=8300) <= 8
    assert 1 <= route("ragged", "fp32", 16, 8, 1, 64, 0, total=500) <= 8
    # ... and so do ordinary batches of them: 13, 25 and 40 sequences of 625, 190 and 60 keys on average (planned 15, 14 and 12 us, in
    # clusters 7.5, 6.7 and 5.4)
    for batch, total in ((13, 8200), (25, 4700), (40, 2500)):
        assert 1 <= route("ragged", "bf16", batch, 8, 8, 64, 0, total=total) <= 8


@pytest.mark.parametrize("sms", [1, 108, 132, 148, 160])
def test_clusters_take_what_they_can_hold(sms):
    """More than sixteen rows never share a cluster; the library's own array never brings tickets along."""
    for layout in ("dense", "ragged", "paged"):
        for batch in (1, 3, 50, 97):
            for keys in (0, 1, 100, 3000):
                for qh, m in ((8, 1), (16, 1), (24, 1), (8, 4), (8, 16)):
                    for dtype in ("bf16", "fp32"):
                        c = route(layout, dtype, batch, qh, 1, 64, keys, m=m, sms=sms)
                        assert c in (PLANNER, INLINE, 1, 2, 4, 8)
                        if keys and qh * m > 16 and (dtype == "bf16" or m > 1):
                            assert c in (PLANNER, INLINE)
                        if batch > 96:
                            assert c != INLINE
                        if 1 < c <= 8:
                            assert batch * c <= 3 * sms
                        s = route(layout, dtype, batch, qh, 1, 64, keys, m=m, static=True, sms=sms)
                        assert s != INLINE
                        if m == 1:
                            assert s == (PLANNER if c == INLINE else c)


# From shared memory: 16-bit calls at D 128 fit three CTAs to an SM up to ten rows per KV head, fp32 calls up to seven; of 148 SMs,
# clusters of eight leave SMs over in every processing cluster: 15, 33 and 48 are resident at one, two and three CTAs per SM.
@pytest.mark.parametrize("dtype,rows,per_sm", [("bf16", 4, 3), ("bf16", 10, 3), ("bf16", 12, 2), ("bf16", 16, 2), ("fp32", 4, 3),
                                               ("fp32", 8, 2), ("fp32", 16, 2)])
def test_all_clusters_of_a_call_are_resident(dtype, rows, per_sm):
    held = {2: (74, 148, 222), 4: (33, 71, 104), 8: (15, 33, 48)}
    for pairs in range(1, 230):
        for layout in ("dense", "paged"):
            for keys in (200, 500):
                c = route(layout, dtype, pairs, rows, 1, 128, keys)
                if 1 < c <= 8:
                    assert pairs <= held[c][per_sm - 1], (pairs, c)
    assert route("dense", dtype, held[8][per_sm - 1], rows, 1, 128, 500) == 8
