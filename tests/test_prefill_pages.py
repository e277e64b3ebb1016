"""Paged prefill by page size: pages of whole groups of eight keys come in one copy per page at head_dim 128, others one 64-column
block at a time; tails, spare pages and the rows behind the last whole group hold NaN."""
import pytest
import torch

from helpers import assert_close_both
from oracle import sdpa_ref

DEV = "cuda"


@pytest.mark.gpu
@pytest.mark.parametrize("page", [1, 2, 4, 5, 8, 12, 16, 24, 64, 128, 192])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("causal", [False, True], ids=["full", "causal"])
def test_prefill_page_sizes(page, d, causal):
    from kernels import flash_attention_v2

    qh, kvh = 4, 2
    kv_lens = [301, 301, 301] if causal else [301, 7, 128]
    lq = kv_lens[0] if causal else 133
    gen = torch.Generator().manual_seed(page * 1000 + d)
    qs = [torch.randn((lq, qh, d), generator=gen).to(torch.bfloat16).to(DEV) for _ in kv_lens]
    ks, vs = ([torch.randn((n, kvh, d), generator=gen).to(torch.bfloat16).to(DEV) for n in kv_lens] for _ in range(2))
    kc, kt, lens = sdpa_ref.pack_paged(ks, page, permute_seed=1, extra_pages=1, pad_value=-1, poison=float("nan"))
    vc, vt, _ = sdpa_ref.pack_paged(vs, page, permute_seed=2, extra_pages=1, pad_value=-1, poison=float("nan"))
    q = torch.stack([x.transpose(0, 1) for x in qs]).contiguous()
    out = flash_attention_v2(q, kc, vc, is_causal=causal, kv_indptr=lens.to(DEV), k_block_table=kt.to(DEV), v_block_table=vt.to(DEV),
                             kv_page_size=page)
    refs = sdpa_ref.prefill_reference(qs, ks, vs, qh, kvh, causal)
    for i, n in enumerate(kv_lens):
        assert_close_both(out[i].transpose(0, 1), refs[i], torch.bfloat16, n, f"seq {i}")
