"""Calls of few (sequence, KV head) pairs without a planner launch, whose many chunks are merged in groups: tickets of eight bits, a pair's in
bytes of its own.  Pairs at every place of a header word and at the line, groups that do not come out even, long pairs beside short ones that
are merged in one step, every kernel, the same call again (tickets are left at zero) and calls of the other ticket forms in between."""
import pytest
import torch

from kernels import decode_attention, speculative_decode_attention
from test_decode_routes import INLINE, route

pytestmark = pytest.mark.gpu
# outputs are averages of |v| <= 5 rounded to 16 bits, as are the probabilities; fp32 decode is 32-bit arithmetic (sums of up to 40 000 terms)
ATOL = {torch.bfloat16: 2e-2, torch.float16: 2.5e-3, torch.float32: 1e-4}


def _call(dtype, qh, kvh, m, d, lens, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed + sum(lens))
    k, v = (torch.randn((sum(lens), kvh, d), generator=g, device="cuda").clamp(-5, 5).to(dtype) for _ in range(2))
    indptr = torch.tensor([0] + lens).cumsum(0).to(torch.int32).cuda()
    shape = (len(lens), qh, d) if m == 1 else (len(lens), qh, m, d)
    q = torch.randn(shape, generator=g, device="cuda").to(dtype)
    run = (lambda: decode_attention(q, k, v, kv_indptr=indptr)) if m == 1 else (
        lambda: speculative_decode_attention(q, k, v, kv_indptr=indptr, causal=False))
    at, refs = 0, []
    for i, n in enumerate(lens):
        kk, vv = (x[at:at + n].double().transpose(0, 1).repeat_interleave(qh // kvh, 0) for x in (k, v))
        s = q[i].double().view(qh, m, d) @ kk.transpose(-1, -2) / d ** 0.5
        refs.append((torch.softmax(s, -1) @ vv).view(q[i].shape))
        at += n
    return run, torch.stack(refs)


CASES = [  # dtype, q heads, KV heads, drafts, head_dim, lengths
    (torch.bfloat16, 8, 1, 1, 128, [30000]),
    (torch.bfloat16, 1, 1, 1, 64, [40001]),
    (torch.float16, 16, 1, 1, 128, [9999, 20, 3000]),
    (torch.bfloat16, 32, 8, 1, 128, [9000]),
    (torch.bfloat16, 6, 3, 1, 64, [20000, 1, 7000, 129, 15000]),
    (torch.bfloat16, 8, 8, 1, 64, [12000, 100, 3000, 5000, 600, 2]),          # 48 pairs: the line
    (torch.bfloat16, 7, 7, 1, 64, [12000, 100, 3000, 5000, 600, 2, 9]),       # 49
    (torch.float32, 8, 1, 1, 64, [30000]),
    (torch.float32, 8, 4, 1, 128, [8000, 50, 6000]),
    (torch.bfloat16, 8, 1, 5, 128, [6607, 14000, 26430]),                     # 40 rows
    (torch.float16, 24, 2, 4, 64, [20000, 64]),                               # 48
    (torch.bfloat16, 16, 1, 8, 128, [30000]),                                 # 128
]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_groups_of_chunks(case):
    dtype, qh, kvh, m, d, lens = CASES[case]
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    name = {torch.bfloat16: "bf16", torch.float16: "fp16", torch.float32: "fp32"}[dtype]
    assert route("ragged", name, len(lens), qh, kvh, d, 0, m=m, total=sum(lens), sms=sms) == INLINE
    run, refs = _call(dtype, qh, kvh, m, d, lens)
    first = run()
    assert (first.double() - refs).abs().max().item() <= ATOL[dtype]
    other, other_refs = _call(torch.bfloat16, 32, 8, 1, 64, [3000] * 10, seed=1)          # 80 pairs: tickets of sixteen bits
    assert (other().double() - other_refs).abs().max().item() <= ATOL[torch.bfloat16]
    for _ in range(3):
        assert torch.equal(run(), first)


def test_groups_in_a_recorded_call():
    run, refs = _call(torch.bfloat16, 8, 1, 1, 128, [30000])
    run()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = run()
    for _ in range(3):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert (out.double() - refs).abs().max().item() <= ATOL[torch.bfloat16]


@pytest.mark.parametrize("qh,kvh,m,d", [(8, 1, 1, 128), (16, 1, 1, 64), (8, 1, 5, 128), (24, 1, 1, 64)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32], ids=["bf16", "fp16", "fp32"])
@pytest.mark.parametrize("batch", [1, 5, 60])
def test_an_infinite_value_stays_infinite(batch, dtype, qh, kvh, m, d):
    """One key of each sequence has an infinite element of V: the weight of every key is positive, and so the output's element is that
    infinity, whatever number of chunks the sequence is merged from."""
    for n in (1500, 2500, 3000, 4000, 7000, 12000):
        g = torch.Generator(device="cuda").manual_seed(n)
        k, v = (torch.randn((batch, kvh, n, d), generator=g, device="cuda").to(dtype) for _ in range(2))
        q = torch.randn((batch, qh, d) if m == 1 else (batch, qh, m, d), generator=g, device="cuda").to(dtype)
        at = torch.arange(batch, device="cuda")
        v[at, 0, at * 977 % n, 7] = float("inf")
        v[at, 0, at * 977 % n, 9] = float("-inf")
        out = decode_attention(q, k, v) if m == 1 else speculative_decode_attention(q, k, v, causal=False)
        assert (out[..., 7] == float("inf")).all() and (out[..., 9] == float("-inf")).all(), n
        assert torch.isfinite(out[..., [i for i in range(d) if i not in (7, 9)]]).all(), n


@pytest.mark.parametrize("dtype,qh,kvh,m,d", [(torch.bfloat16, 8, 1, 1, 64), (torch.float32, 8, 2, 1, 128), (torch.float16, 32, 8, 1, 128),
                                              (torch.bfloat16, 8, 1, 2, 128), (torch.bfloat16, 8, 1, 4, 128)])
@pytest.mark.parametrize("chunks", [25, 26, 27, 39, 40, 41])
def test_either_side_of_the_lines(chunks, dtype, qh, kvh, m, d):
    """Pairs of as many chunks as are merged in one step and in groups: 26 are the first where a thread has more than one element of the
    output, 40 where it has one."""
    from utils.launch_config import decode_items, decode_plan

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for n in range(1500, 40000, 128):
        lens = [n, 700]
        plan = decode_plan(sms, 2, qh, kvh, m, fp32=dtype == torch.float32, keys=sum(lens), head_dim=d)
        if decode_items(plan, lens)[0] == chunks:
            break
    else:
        pytest.skip("no length of that many chunks")
    run, refs = _call(dtype, qh, kvh, m, d, lens)
    first = run()
    assert (first.double() - refs).abs().max().item() <= ATOL[dtype]
    assert torch.equal(run(), first)
