"""Prefill launches of few work items whose KV range is cut over the CTAs of a cluster: two, four and eight parts, parts that see no key
(beyond the diagonal, behind a short sequence), rows that no part sees, query blocks that are not full, both element widths."""
import pytest
import torch

from helpers import assert_close_both
from oracle import sdpa_ref
from test_prefill_routes import route

pytestmark = pytest.mark.gpu
DEV = "cuda"


# (batch, q heads, kv heads, queries, keys, causal, head_dim); items of one or two q heads x 128 rows: up to 15 for eight parts, 33 for
# four, 74 for two
SHAPES = [(1, 8, 2, 100, 600, False, 64), (1, 2, 1, 128, 1024, False, 64), (2, 8, 1, 1, 1500, False, 128), (3, 8, 2, 130, 700, False, 64),
          (16, 8, 2, 128, 760, False, 64), (1, 8, 2, 512, 512, True, 64), (1, 8, 8, 700, 700, True, 64), (1, 4, 4, 300, 1600, False, 128),
          (2, 6, 2, 257, 1537, False, 128), (1, 2, 2, 1400, 1400, True, 128), (1, 4, 2, 1500, 1500, True, 128)]


def _route(layout, dtype, *shape):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return route(layout, {torch.bfloat16: "bf16", torch.float16: "fp16", torch.float32: "fp32"}[dtype], *shape, sms=sms)


@pytest.mark.parametrize("layout", ["dense", "paged"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: f"b{s[0]}-{s[1]}-{s[2]}-q{s[3]}-kv{s[4]}-{'c' if s[5] else 'f'}-d{s[6]}")
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32], ids=["fp16", "fp32"])
def test_parts(layout, shape, dtype):
    from test_attention import run_prefill

    b, qh, kvh, lq, lkv, causal, d = shape
    assert 1 < _route(layout, dtype, *shape) <= 8
    gen = torch.Generator().manual_seed(lq + 3 * lkv + qh)
    lens = [lkv] * b if causal or layout == "dense" else [max(1, lkv - 190 * i - 64 * (i % 2)) for i in range(b)]
    qs = [torch.randn((lq, qh, d), generator=gen).to(dtype).to(DEV) for _ in range(b)]
    ks = [torch.randn((n, kvh, d), generator=gen).to(dtype).to(DEV) for n in lens]
    vs = [torch.randn((n, kvh, d), generator=gen).to(dtype).to(DEV) for n in lens]
    refs = sdpa_ref.prefill_reference(qs, ks, vs, qh, kvh, causal)
    for _ in range(2):
        outs = run_prefill(layout, qs, ks, vs, causal, permute=5, pad=-1, poison=float("nan"))
        for i in range(b):
            assert_close_both(outs[i], refs[i], dtype, lens[i], f"seq {i}", strict=4e-3 if dtype == torch.float32 else None)


@pytest.mark.parametrize("d", [64, 128])
def test_a_part_of_nan_shows(d):
    """One NaN key makes every row NaN, also in a part none of whose scores is a number; values of -inf scores weigh nothing."""
    from kernels import flash_attention_v2

    assert 1 < _route("dense", torch.bfloat16, 1, 2, 2, 128, 1500, False, d) <= 8
    gen = torch.Generator().manual_seed(d)
    q, k, v = (torch.randn((1, 2, n, d), generator=gen).to(torch.bfloat16).to(DEV) for n in (128, 1500, 1500))
    ref = flash_attention_v2(q, k, v)
    assert torch.isfinite(ref.float()).all()
    for lo, hi in ((700, 701), (384, 1500)):
        bad = k.clone()
        bad[:, :, lo:hi] = float("nan")
        assert torch.isnan(flash_attention_v2(q, bad, v).float()).all()


@pytest.mark.parametrize("d", [64, 128])
def test_rows_keep_to_themselves(d):
    """A row that is NaN changes no other row: a thread holds two, eight rows apart, and one whose scores are all -inf has no sum."""
    from kernels import flash_attention_v2

    assert 1 < _route("dense", torch.bfloat16, 1, 2, 2, 128, 1500, False, d) <= 8
    gen = torch.Generator().manual_seed(d + 1)
    q, k, v = (torch.randn((1, 2, n, d), generator=gen).to(torch.bfloat16).to(DEV) for n in (128, 1500, 1500))
    k[..., 0] = 1.0
    q[:, :, 3, 0] = float("-inf")
    q[:, :, 12, 0] = float("-inf")
    want = flash_attention_v2(q, k, v)
    q[:, :, [11, 4, 77], 1] = float("nan")
    out = flash_attention_v2(q, k, v)
    nan = torch.zeros(128, dtype=torch.bool, device=DEV)
    nan[[11, 4, 77]] = True
    assert torch.isnan(out[:, :, nan].float()).all()
    assert not out[:, :, [3, 12]].any() and not want[:, :, [3, 12]].any()
    # (a warp with such a row takes its tiles in two passes: P and the output rounded to eight bits around another reference)
    torch.testing.assert_close(out[:, :, ~nan].float(), want[:, :, ~nan].float(), atol=2**-7, rtol=2**-7)


@pytest.mark.parametrize("queries,longest,d,causal", [(100, 760, 64, False), (100, 1500, 64, False), (100, 1500, 128, False),
                                                      (700, 760, 64, True), (1500, 1500, 128, True)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32], ids=["bf16", "fp32"])
def test_sequences_shorter_than_the_table(queries, longest, d, causal, dtype):
    """An item of fewer tiles than the parts are worth is the first CTA's alone: every number of tiles up to the widest, also none."""
    from kernels import flash_attention_v2

    gen = torch.Generator().manual_seed(longest + d)
    b, page = (13, 16) if queries == 100 else (2, 16)
    lens = ([0, longest] + [n for t in range(1, 12) for n in (128 * t, 128 * t + 1) if n <= longest])[:b]
    assert 1 < _route("paged", dtype, len(lens), 2, 1, queries, longest, causal, d) <= 8
    qs = [torch.randn((queries, 2, d), generator=gen).to(dtype).to(DEV) for _ in lens]
    ks, vs = ([torch.randn((n, 1, d), generator=gen).to(dtype).to(DEV) for n in lens] for _ in range(2))
    (kc, kt, n), (vc, vt, _) = (sdpa_ref.pack_paged(x, page, permute_seed=3, extra_pages=2, pad_value=-1, poison=float("nan")) for x in (ks, vs))
    q = torch.stack([x.transpose(0, 1) for x in qs]).contiguous()
    out = flash_attention_v2(q, kc, vc, is_causal=causal, kv_indptr=n, k_block_table=kt, v_block_table=vt, kv_page_size=page)
    assert not out[0].any()
    refs = sdpa_ref.prefill_reference(qs[1:], ks[1:], vs[1:], 2, 1, causal)
    for i, ref in enumerate(refs, 1):
        assert_close_both(out[i].transpose(0, 1), ref, dtype, max(1, lens[i]), f"{lens[i]} keys", strict=4e-3 if dtype == torch.float32 else None)
