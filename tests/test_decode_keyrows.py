"""Planned calls of 17 to 64 q rows per KV head over long sequences: the decode kernel whose tensor-core tiles have keys as their rows
(128 to a tile, columns padded to a multiple of sixteen, in chunks of eight over four groups of warps).  Row counts either side of every
chunk and padding, lengths either side of a tile and of its steps of sixteen keys, empty and one-tile sequences between long ones, drafts
that hide keys, pages of whole groups of eight keys, references that move, hostile rows behind the sequences' ends."""
import pytest
import torch

from kernels import speculative_decode_attention
from oracle import sdpa_ref
from test_decode_references import _check, _rising

pytestmark = pytest.mark.gpu
# bf16 output and probabilities: half a unit, 2^-9, each, of values up to 5
ATOL = {torch.bfloat16: 2e-2, torch.float16: 2.5e-3}


def _takes_it(batch, kvh, rows, keys, d, page=None):
    from test_decode_routes import PLANNER, route
    from utils.launch_config import keyrows_suit

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    layout = "dense" if page is None else "paged"
    assert route(layout, "bf16", batch, rows * kvh, kvh, d, keys // batch, page=page or 16, sms=sms) == PLANNER
    assert keyrows_suit(sms, batch, kvh, rows, keys, d, page)


def _reference(q, k, v, causal):
    """One sequence: q [H, M, D], k and v [N, KVH, D]; zeros where there is no key."""
    n, g, m = k.shape[0], q.shape[0] // k.shape[1], q.shape[1]
    if n == 0:
        return torch.zeros_like(q, dtype=torch.float64)
    kk, vv = (x.double().transpose(0, 1).repeat_interleave(g, 0) for x in (k, v))
    s = q.double() @ kk.transpose(-1, -2) / q.shape[-1] ** 0.5
    if causal:
        s = s.masked_fill(torch.arange(n, device=q.device)[None] > torch.arange(n - m, n, device=q.device)[:, None], float("-inf"))
    return torch.softmax(s, -1).nan_to_num(0.0) @ vv


def _run(layout, dtype, qh, kvh, m, d, lens, causal, page=16, seed=0, width=0, again=0, cache=0):
    """`width`: keys that the tables have room for, where that is more than the longest sequence; `cache`: rows of the cache, where that
    is more than the sequences'; `again`: further calls, of which the same bits are expected."""
    g = torch.Generator(device="cuda").manual_seed(seed + qh + m)
    q = torch.randn((len(lens), qh, m, d), generator=g, device="cuda").to(dtype)
    ks, vs = ([torch.randn((n, kvh, d), generator=g, device="cuda").clamp(-5, 5).to(dtype) for n in lens] for _ in range(2))
    if layout == "dense":
        k, v = (torch.stack(x).transpose(1, 2).contiguous() for x in (ks, vs))
        call = lambda: speculative_decode_attention(q, k, v, causal=causal)
    elif layout == "ragged":
        # NaN behind the last sequence; a tile that ends in one sequence holds the next one's rows
        pad = torch.full((130, kvh, d), float("nan"), device="cuda", dtype=dtype)
        k, v = (torch.cat(x + [pad])[: sum(lens)] for x in (ks, vs))
        indptr = torch.tensor([0] + lens).cumsum(0).to(torch.int32).cuda()
        call = lambda: speculative_decode_attention(q, k, v, causal=causal, kv_indptr=indptr)
    else:
        spare = max(2, cache // page - sum(-(-n // page) for n in lens))
        kc, kt, ln = sdpa_ref.pack_paged(ks, page, permute_seed=1, extra_pages=spare, pad_value=-1, poison=float("nan"))
        vc, vt, _ = sdpa_ref.pack_paged(vs, page, permute_seed=2, extra_pages=spare, pad_value=-1, poison=float("nan"))
        kt, vt = (torch.nn.functional.pad(t, (0, max(0, width // page - t.shape[1])), value=-1).cuda() for t in (kt, vt))
        ln = ln.cuda()
        from test_decode_keyrows_rule import _args, _ask

        asked = _args("paged", "bf16", len(lens), qh, kvh, d, kt.shape[1] * page, m, page, kc.shape[0])
        assert _ask(asked, sms=torch.cuda.get_device_properties(0).multi_processor_count)[1] == 1
        call = lambda: speculative_decode_attention(q, kc, vc, causal=causal, kv_indptr=ln, k_block_table=kt, v_block_table=vt,
                                                    kv_page_size=page)
    out = call()
    for _ in range(again):
        assert torch.equal(call(), out)
    assert torch.isfinite(out).all()
    for i, n in enumerate(lens):
        ref = _reference(q[i], ks[i], vs[i], causal)
        assert (out[i].double() - ref).abs().max().item() <= ATOL[dtype], (i, n)


@pytest.mark.parametrize("rows", [17, 23, 24, 25, 31, 32, 33, 40, 47, 48, 49, 56, 57, 63, 64])
@pytest.mark.parametrize("d", [64, 128])
def test_row_counts(rows, d):
    """`rows` heads with one draft would be plain decode: one KV head and `rows` q heads, or 4 drafts of rows / 4 heads."""
    heads, m = (rows // 4, 4) if rows % 4 == 0 else (rows, 1)
    batch = 100
    _takes_it(batch, 1, rows, batch * 1100, d)
    _run("dense", torch.bfloat16, heads, 1, m, d, [1100] * batch, m > 1)


LENS = [0, 1, 3, 15, 16, 17, 63, 64, 65, 111, 112, 113, 127, 128, 129, 143, 144, 145, 255, 256, 257, 300, 383, 385]


@pytest.mark.parametrize("layout,page", [("ragged", None), ("paged", 8), ("paged", 16), ("paged", 24), ("paged", 64), ("paged", 256)])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("causal", [False, True])
def test_lengths_and_pages(layout, page, d, causal):
    lens = [n for n in LENS if n == 0 or n >= 3 or not causal] + [(2600 if d == 128 else 5700) + 7 * i for i in range(78)]
    keys = sum(lens) if layout == "ragged" else len(lens) * -(-max(lens) // page) * page
    _takes_it(len(lens), 2, 24, keys, d, page)
    _run(layout, torch.bfloat16, 16, 2, 3, d, lens, causal, page=page or 16)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("layout", ["dense", "ragged", "paged"])
def test_long_sequences_are_cut_and_merged(dtype, layout):
    lens = [20000] * 13 if layout == "dense" else [3, 70000, 128, 9000, 33333, 20001, 64, 15000, 500, 40000, 7, 25000, 1]
    _takes_it(13, 8, 40, sum(lens), 128, 16 if layout == "paged" else None)
    _run(layout, dtype, 64, 8, 5, 128, lens, causal=False, seed=1)


def _with_empty(batch, empty, order, length):
    """Lengths of `batch` sequences, `empty` tenths of them zero, in runs or scattered; the others length(i)."""
    blank = [i % 10 < empty for i in range(batch)]
    if order == "scattered":
        blank = [blank[p] for p in torch.randperm(batch, generator=torch.Generator().manual_seed(empty)).tolist()]
    return [0 if b else length(i) for i, b in enumerate(blank)]


def _cache_for(batch, qh, kvh, m, d, width, page=16):
    """Rows of the smallest cache, in units of 4 096, before which the library takes such a call to the kernel."""
    from test_decode_keyrows_rule import _args, _ask

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for cache in range(4096, batch * width + 1, 4096):
        if _ask(_args("paged", "bf16", batch, qh, kvh, d, width, m, page, cache), sms=sms)[1] == 1:
            return cache
    raise AssertionError("not that kernel's, whatever the cache")


def _run_with_empty(lens, kvh, d, dealt, page=None, width=0):
    from kernels._native import check_device_errors
    from utils.launch_config import decode_cuts, decode_plan

    from test_decode_keyrows_rule import _args, _ask

    keys = sum(lens) if page is None else len(lens) * width
    _takes_it(len(lens), kvh, 24, keys, d, page)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    plan = decode_plan(sms, len(lens), 8 * kvh, kvh, 3, keys=keys, head_dim=d, page_size=page, equal=False)
    assert page is not None or _ask(_args("ragged", "bf16", len(lens), 8 * kvh, kvh, d, 0, 3, cache=keys), sms=sms)[1] == 1
    assert (decode_cuts(plan, lens) is not None) == dealt
    _run("ragged" if page is None else "paged", torch.bfloat16, 8 * kvh, kvh, 3, d, lens, causal=False, width=width, again=20,
         cache=0 if page is None else _cache_for(len(lens), 8 * kvh, kvh, 3, d, width, page))
    check_device_errors()


# what the sequences with keys are, in tables of 16 384: several tiles, one tile, mostly one tile and a few that are cut
KEYS = {"long": [700, 1300, 640], "one tile": [20, 128, 100, 7], "cut": [30, 9000, 100, 64, 128]}


@pytest.mark.parametrize("empty", [3, 6, 9])
@pytest.mark.parametrize("order", ["runs", "scattered"])
@pytest.mark.parametrize("kind", ["long", "one tile", "cut", "packed"])
@pytest.mark.parametrize("kvh,d", [(1, 128), (2, 64), (8, 128)])
def test_empty_sequences(empty, order, kind, kvh, d):
    """Longest-first order hands the units of sequences without keys out behind all others, `kvh` for each."""
    batch, lengths = 320 // kvh, KEYS["cut" if kind == "packed" else kind]
    lens = _with_empty(batch, empty, order, lambda i: lengths[i // 3 % len(lengths)])
    if kind == "packed":       # as many keys as the call needs to go there, most of them in the last sequence
        lens[-1] += max(0, 1100 * 128 // d * batch - sum(lens))
    _run_with_empty(lens, kvh, d, False, *(() if kind == "packed" else (16, 16384)))


@pytest.mark.parametrize("order", ["runs", "scattered"])
@pytest.mark.parametrize("kvh,d,empty", [(1, 128, 6), (2, 64, 3), (2, 64, 6), (8, 128, 3)])
def test_empty_sequences_dealt_out(kvh, d, empty, order):
    """A CTA's units are those of its stretch of the batch: a run of empty sequences comes one behind the other."""
    lens = _with_empty(60 // kvh + 20 if d == 128 else 80, empty, order, lambda i: 1000 + i * 7919 % 33000)
    _run_with_empty(lens, kvh, d, True)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("heads,m", [(8, 3), (8, 5), (8, 8)])
@pytest.mark.parametrize("kvh", [1, 2, 8])
def test_short_ends_of_cut_sequences(kvh, heads, m, d):
    """Every sequence is a chunk of the shortest and twenty keys.  Those ends come last, and a CTA finishes one after the other: a pair's
    ticket may be drawn when all four output warps have written the unit's rows (at head_dim 64 two of them have none to write)."""
    from kernels._native import check_device_errors
    from utils.launch_config import decode_chunk_tokens, decode_cuts, decode_plan

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    batch, width = 3 * sms // kvh // 2, 16384
    plan = decode_plan(sms, batch, heads * kvh, kvh, m, keys=batch * width, head_dim=d, page_size=16)
    lens = [plan.min_chunk + 20] * batch
    assert decode_cuts(plan, lens) is None and decode_chunk_tokens(plan, lens) == plan.min_chunk
    _takes_it(batch, kvh, heads * m, batch * width, d, 16)
    _run("paged", torch.bfloat16, heads * kvh, kvh, m, d, lens, causal=False, width=width, again=40,
         cache=_cache_for(batch, heads * kvh, kvh, m, d, width))
    check_device_errors()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32], ids=["bf16", "fp16", "fp32"])
@pytest.mark.parametrize("qh,kvh,m", [(16, 2, 5), (6, 2, 7), (32, 4, 8)])
@pytest.mark.parametrize("step", [0, 2.9, 3.1, 9.9, 10.1, 16.5, 40])
def test_growing_maximum(dtype, qh, kvh, m, step):
    """Blocks of 64 keys whose scores lie ever higher: references that stand, move, and move by more than P can hold."""
    batch = -(-100 // kvh)
    for d, n, rows in ((64, 12 * 128 + 33, None), (128, 10 * 128, [3, 17])):
        _takes_it(batch, kvh, qh // kvh * m, batch * n, d)
        _check(*_rising(dtype, batch, qh, kvh, m, d, n, step, rows=rows))
        q, k, v = _rising(dtype, batch, qh, kvh, m, d, n, step, block=16, rows=rows)
        _check(q, k.flip(2).contiguous(), v)


@pytest.mark.parametrize("first", [1, 16, 127, 128, 129, 300])
def test_first_keys_at_minus_infinity(first):
    q, k, v = _rising(torch.bfloat16, 100, 20, 1, 2, 128, 1000, 4)
    _takes_it(100, 1, 40, 100 * 1000, 128)
    q[..., 0] = 1e20
    k[..., 0] = 0.0
    k[:, :, :first, 0] = -1e20      # products of -1e40: -inf in the fp32 accumulator (in 64 bits the weight is 0 all the same)
    _check(q, k, v)


def test_nan_stays_in_its_row_and_sequence():
    q, k, v = _rising(torch.bfloat16, 100, 20, 1, 2, 128, 1000, 0)
    q[7, 3, 1] = float("nan")
    k[9, 0, 500] = float("nan")
    out = speculative_decode_attention(q, k, v, causal=False)
    bad = torch.isnan(out).all(-1)
    assert bad[7, 3, 1] and bad[7].sum() == 1 and bad[9].all()
    assert torch.isfinite(out[[i for i in range(100) if i not in (7, 9)]]).all()
