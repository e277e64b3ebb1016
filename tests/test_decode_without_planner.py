"""Decode calls with few (sequence, KV head) pairs plan inside the kernel; the fp32 kernel's row blocks; calls that follow
one another on a stream without a synchronisation in between."""
import pytest
import torch

from helpers import assert_close_both
from oracle import sdpa_ref

pytestmark = pytest.mark.gpu
DEV = "cuda"
PAIRS = 96                    # csrc/decode_launch.h kInlinePairs


def _problem(gen, lens, qh, kvh, d, dtype, m=0):
    shape = (qh, d) if m == 0 else (qh, m, d)
    qs = [torch.randn(shape, generator=gen).to(dtype).to(DEV) for _ in lens]
    ks = [torch.randn((n, kvh, d), generator=gen).to(dtype).to(DEV) for n in lens]
    vs = [torch.randn((n, kvh, d), generator=gen).to(dtype).to(DEV) for n in lens]
    return qs, ks, vs


def _call(qs, ks, vs, layout, m, page=16, index=torch.int32):
    from kernels import decode_attention, speculative_decode_attention

    q = torch.stack(qs)
    if layout == "ragged":
        (k, ip), (v, _) = sdpa_ref.pack_ragged(ks, index), sdpa_ref.pack_ragged(vs, index)
        kw = {"kv_indptr": ip}
    elif layout == "dense":
        k, v = (torch.stack([x.transpose(0, 1) for x in t]).contiguous() for t in (ks, vs))
        kw = {}
    else:
        k, kt, n = sdpa_ref.pack_paged(ks, page, permute_seed=1, extra_pages=2, pad_value=-1, poison=float("nan"))
        v, vt, _ = sdpa_ref.pack_paged(vs, page, permute_seed=2, extra_pages=2, pad_value=-1, poison=float("nan"))
        kw = {"kv_indptr": n, "k_block_table": kt, "v_block_table": vt, "kv_page_size": page}
    return decode_attention(q, k, v, **kw) if m == 0 else speculative_decode_attention(q, k, v, causal=True, **kw)


def _reference(qs, ks, vs, qh, kvh, m):
    f = [[t.float() for t in x] for x in (qs, ks, vs)]
    refs = sdpa_ref.decode_reference(*f, qh, kvh) if m == 0 else sdpa_ref.spec_decode_reference(*f, qh, kvh, True)
    return torch.stack(refs)


# batch x KV heads on both sides of the line; one KV head (most items per pair); lengths around tiles, one key, long
@pytest.mark.parametrize("batch,qh,kvh", [(1, 8, 1), (1, 32, 8), (12, 8, 8), (13, 8, 8), (48, 4, 2), (49, 4, 2), (96, 2, 1),
                                          (97, 2, 1), (1, 96, 96), (1, 97, 97)])
@pytest.mark.parametrize("layout,page,index", [("dense", 0, None), ("ragged", 0, torch.int32), ("ragged", 0, torch.int64),
                                               ("paged", 16, None), ("paged", 24, None)])
def test_both_plans_over_layouts(batch, qh, kvh, layout, page, index):
    gen = torch.Generator().manual_seed(batch * 131 + qh)
    base = [300] if layout == "dense" else [1, 63, 64, 65, 127, 129, 640, 1000, 2500]
    lens = [base[i % len(base)] for i in range(batch)] if batch > 1 else [5000]
    for m in (0, 2):
        qs, ks, vs = _problem(gen, lens, qh, kvh, 64, torch.bfloat16, m)
        out = _call(qs, ks, vs, layout, m, page or 16, index or torch.int32)
        assert_close_both(out, _reference(qs, ks, vs, qh, kvh, m), torch.bfloat16, max(lens), f"{layout} {batch}x{kvh} m{m}")


def test_empty_sequences_without_planner():
    gen = torch.Generator().manual_seed(5)
    lens = [0, 700, 0, 3, 0]
    for dtype in (torch.float16, torch.float32):
        qs, ks, vs = _problem(gen, lens, 8, 2, 64, dtype)
        out = _call(qs, ks, vs, "ragged", 0)
        live = [i for i, n in enumerate(lens) if n]
        ref = _reference([qs[i] for i in live], [ks[i] for i in live], [vs[i] for i in live], 8, 2, 0)
        assert_close_both(out[live], ref, dtype, 700)
        assert (out[[0, 2, 4]] == 0).all()


# q rows per KV head: blocks of 1, 2 and 4 rows, blocks with rows left over, three blocks (no key split); more than 16 rows
# multiply in 16 bits, on another kernel
@pytest.mark.parametrize("group", [1, 2, 3, 4, 5, 8, 9, 16])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("layout", ["ragged", "paged"])
def test_fp32_row_blocks(group, d, layout):
    gen = torch.Generator().manual_seed(group * 7 + d)
    lens = [1, 31, 64, 65, 200, 1111]
    qs, ks, vs = _problem(gen, lens, 2 * group, 2, d, torch.float32)
    out = _call(qs, ks, vs, layout, 0)
    # 64-bit reference.  A score is a sum of d products of N(0, 1) numbers, a weight its exponential, an output a sum of
    # weighted values: relative errors of a few d * 2^-24 (scores of up to 5 / sqrt(d) * d) - 2e-5 covers them.
    f = [[t.double().cpu() for t in x] for x in (qs, ks, vs)]
    for i, n in enumerate(lens):
        k = f[1][i].repeat_interleave(group, 1)
        w = torch.softmax(torch.einsum("hd,nhd->hn", f[0][i], k) / d ** 0.5, -1)
        want = torch.einsum("hn,nhd->hd", w, f[2][i].repeat_interleave(group, 1))
        torch.testing.assert_close(out[i].double().cpu(), want, atol=2e-5, rtol=2e-5)


@pytest.mark.parametrize("qh,m", [(8, 0), (64, 5)], ids=["decode", "speculative"])   # warp-level and tcgen05 kernel
def test_calls_in_a_row_see_each_other(qh, m):
    """Each call reads what the one before it wrote (cache rows, scores, fp16 copies), each has its launch set up while
    that one is still running: the outputs are those of the same calls one at a time."""
    from kernels import append_paged_kv, decode_attention, flash_attention_v2, softmax, speculative_decode_attention

    gen = torch.Generator().manual_seed(9)
    batch, kvh, d, page, steps = 4, 8, 128, 16, 24
    pages = 20
    table = torch.randperm(batch * pages, generator=gen).to(torch.int32).view(batch, pages).to(DEV)
    q0 = torch.randn((batch, qh, d) if m == 0 else (batch, qh, m, d), generator=gen).to(torch.bfloat16).to(DEV)
    new = torch.randn((batch * 8, kvh, d), generator=gen).to(torch.bfloat16).to(DEV)
    indptr = torch.arange(0, 8 * batch + 1, 8, dtype=torch.int32, device=DEV)
    pq = torch.randn((1, 8, 128, d), generator=gen).to(DEV)

    def run(sync):
        wait = torch.cuda.synchronize if sync else (lambda: None)
        k = torch.zeros((batch * pages * page, kvh, d), dtype=torch.bfloat16, device=DEV)
        v = torch.zeros_like(k)
        x, y, outs = q0, pq, []
        for s in range(steps):
            pos = torch.full((batch,), 8 * s, dtype=torch.int32, device=DEV)
            lens = pos + 8
            wait()
            append_paged_kv(k, table, new, indptr, page, dst_pos=pos)
            wait()
            append_paged_kv(v, table, softmax(new), indptr, page, dst_pos=pos)
            wait()
            kw = dict(kv_indptr=lens, k_block_table=table, v_block_table=table, kv_page_size=page)
            x = decode_attention(x, k, v, **kw) if m == 0 else speculative_decode_attention(x, k, v, causal=True, **kw)
            wait()
            x = softmax(x)
            wait()
            y = flash_attention_v2(y, y, y, is_causal=True)
            wait()
            y = softmax(y)
            wait()
            outs += [x, y]
        torch.cuda.synchronize()
        return [*outs, k, v]

    for a, b in zip(run(True), run(False)):
        assert torch.equal(a, b)
