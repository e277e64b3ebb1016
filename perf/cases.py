"""The work that programs have this package do, as timed cases: attention prefill, decode and speculative decode over
dense, ragged and paged KV, the paged-cache append that precedes them in a server, and row softmax / log-softmax.

A case is a dict of plain values.  ``kind`` is ``prefill``, ``decode``, ``spec`` or ``softmax``; sequence lengths are
drawn between ``lo`` and ``hi`` with the generator seeded by ``lengths`` (they belong to the case, not to its inputs),
and ``append`` rows per sequence are written into the paged cache before the attention call, as a server does with the
keys and values of the tokens it is about to attend from.  Tensor values are N(0, 1); softmax rows are N(0, 3)."""
import os
import sys

import torch

_PKG = os.path.join(os.getcwd(), "triton-kernels_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from kernels import (  # noqa: E402
    append_paged_kv,
    decode_attention,
    flash_attention_v2,
    log_softmax,
    softmax,
    speculative_decode_attention,
)

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}
SIZE = {"fp16": 2, "bf16": 2, "fp32": 4}


def _attention(name, kind, layout, dtype, batch, heads, head_dim, lo, hi, lengths=0, drafts=1, q_len=0, causal=False,
               page=16, append=0):
    """``q_len`` 0: as many queries as keys (self attention)."""
    return {"name": name, "kind": kind, "layout": layout, "dtype": dtype, "batch": batch, "q_heads": heads[0],
            "kv_heads": heads[1], "head_dim": head_dim, "lo": lo, "hi": hi, "lengths": lengths, "drafts": drafts,
            "q_len": q_len, "causal": causal, "page": page if layout == "paged" else 0, "append": append}


def listed():
    return [
        # one user's next token: the smallest call of a server, the new K and V rows go into the cache first
        _attention("decode_one_user", "decode", "paged", "bf16", 1, (32, 8), 128, 1500, 1500, append=1),
        # a small equal-length batch over plain tensors, the middle of the decode grid in benchmarks/sweeps.py
        _attention("decode_dense_batch", "decode", "dense", "fp16", 16, (8, 2), 64, 2048, 2048),
        # a serving batch of mixed contexts: the paged decode workload of bench.py
        _attention("decode_paged_serving", "decode", "paged", "bf16", 64, (32, 8), 128, 512, 8192),
        # full-precision decode over packed sequences of odd lengths (evaluation, numerics checks)
        _attention("decode_fp32_ragged", "decode", "ragged", "fp32", 16, (8, 8), 64, 100, 4096, lengths=1),
        # a few drafts for a small batch of short packed sequences: the tests' speculative-decode range
        _attention("spec_ragged_small", "spec", "ragged", "fp16", 16, (8, 2), 64, 17, 1024, drafts=4, causal=True),
        # drafts over long contexts: the paged speculative-decode workload of bench.py (contexts + 5 drafts)
        _attention("spec_paged_serving", "spec", "paged", "bf16", 32, (64, 8), 128, 1024 + 5, 32768 + 5, drafts=5,
                   causal=True),
        # one short fp32 prompt: the CPU-sized configuration of the benchmark
        _attention("prefill_fp32_prompt", "prefill", "dense", "fp32", 1, (8, 2), 64, 512, 512, causal=True),
        # two equal prompts: the dense prefill workload of bench.py
        _attention("prefill_dense_causal", "prefill", "dense", "bf16", 2, (32, 8), 128, 2048, 2048, causal=True),
        # packed prompts of 128 to 4096 tokens: the ragged prefill workload of bench.py
        _attention("prefill_ragged_causal", "prefill", "ragged", "bf16", 16, (32, 8), 128, 128, 4096, causal=True),
        # a chunk of 128 new tokens per sequence over cached keys: cross 128 x 2048 of the prefill grid in
        # benchmarks/sweeps.py, the chunk's K and V appended first
        _attention("prefill_paged_chunk", "prefill", "paged", "fp16", 16, (8, 2), 128, 2048, 2048, q_len=128, append=128),
        # scores of a hand-written attention: a shape of the softmax benchmark
        {"name": "softmax_scores", "kind": "softmax", "dtype": "bf16", "rows": 4096, "cols": 4096, "log": False},
        # token log-probabilities over a vocabulary whose size is not a multiple of anything
        {"name": "log_softmax_logits", "kind": "softmax", "dtype": "fp32", "rows": 2000, "cols": 50001, "log": True},
    ]


# No drawn case does more than the largest listed ones: bytes of keys and values (fp32 decode multiplies on the FMA
# pipes and gets less), tensor-core work (short heads reach half the rate), bytes of a softmax.
_MAX_KV_BYTES = {"fp16": 1.6e9, "bf16": 1.6e9, "fp32": 2.5e8}
_MAX_FLOPS = {64: 4e11, 128: 9e11}
_MAX_SOFTMAX_BYTES = 1.6e9


def _log_uniform(rng, lo, hi):
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "spec", "spec", "prefill", "prefill", "prefill", "softmax"])
    dtype = rng.choice(["bf16", "bf16", "bf16", "fp16", "fp16", "fp32"])
    if kind == "softmax":
        cols = _log_uniform(rng, 128, 262144)
        if rng.random() < 0.6:
            cols = max(128, cols // 64 * 64)
        rows = _log_uniform(rng, 1, 65536)
        rows = max(1, min(rows, int(_MAX_SOFTMAX_BYTES / (2 * SIZE[dtype] * cols))))
        return {"kind": kind, "dtype": dtype, "rows": rows, "cols": cols, "log": rng.random() < 0.5}
    layout = rng.choice(["dense", "ragged", "paged", "paged"])
    heads = rng.choice([(8, 8), (8, 2), (8, 1), (32, 8), (32, 8), (64, 8)])
    head_dim = rng.choice([64, 128, 128])
    lengths = rng.randrange(1 << 20)
    page = rng.choice([16, 16, 16, 32, 64, 128])
    if kind == "prefill":
        batch = _log_uniform(rng, 1, 32)
        hi = _log_uniform(rng, 16, 8192)
        q_len = 0 if layout == "ragged" or rng.random() < 0.6 else _log_uniform(rng, 16, 1024)
        causal = q_len == 0 and rng.random() < 0.75
        drafts, append = 1, 0
    else:
        batch = _log_uniform(rng, 1, 256)
        hi = _log_uniform(rng, 16, 32768)
        q_len, drafts = 0, rng.randint(2, 10) if kind == "spec" else 1
        causal = kind == "spec" and rng.random() < 0.75
        append = drafts if layout == "paged" and rng.random() < 0.5 else 0
    # a paged prefill call with as many queries as keys has queries of one length for all sequences, like a dense one
    uniform = layout == "dense" or (kind == "prefill" and layout == "paged")
    hi = max(hi, drafts)
    lo = hi if uniform else max(drafts, hi // rng.choice([1, 4, 16, 32]))
    if kind == "prefill" and layout == "paged" and rng.random() < 0.5:
        append = min(q_len or hi, hi)
    case = _attention("", kind, layout, dtype, batch, heads, head_dim, lo, hi, lengths, drafts, q_len, causal, page, append)
    del case["name"]
    while case["batch"] > 1 and _too_large(case):
        case["batch"] = max(1, case["batch"] * 3 // 4)
    while _too_large(case):
        case["hi"] = max(drafts, case["hi"] * 3 // 4)
        case["lo"] = case["hi"] if uniform else min(case["lo"], case["hi"])
        case["append"] = min(case["append"], case["hi"])
    return case


def _too_large(case):
    kv = 2.0 * sum(_lengths(case)) * case["kv_heads"] * case["head_dim"] * SIZE[case["dtype"]]
    return kv > _MAX_KV_BYTES[case["dtype"]] or (
        case["kind"] == "prefill" and work(case)["flops"] > _MAX_FLOPS[case["head_dim"]])


def _lengths(case):
    g = torch.Generator().manual_seed(case["lengths"])
    return torch.randint(case["lo"], case["hi"] + 1, (case["batch"],), generator=g).tolist()


def _q_lengths(case):
    if case["kind"] == "prefill":
        return [case["q_len"] or n for n in _lengths(case)]
    return [case["drafts"]] * case["batch"]


def _prefix(lens):
    return torch.tensor([0] + lens, dtype=torch.int64).cumsum(0).to(torch.int32).cuda()


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype = DTYPES[case["dtype"]]

    def normal(*shape):
        return torch.randn(shape, generator=gen, device="cuda").to(dtype)

    if case["kind"] == "softmax":
        return {"case": case, "x": (3 * torch.randn((case["rows"], case["cols"]), generator=gen, device="cuda")).to(dtype)}
    batch, qh, kvh, d = case["batch"], case["q_heads"], case["kv_heads"], case["head_dim"]
    lens, q_lens = _lengths(case), _q_lengths(case)
    s = {"case": case, "kw": {}}
    if case["kind"] == "decode":
        s["q"] = normal(batch, qh, d)
    elif case["kind"] == "spec" or case["layout"] != "ragged":
        s["q"] = normal(batch, qh, q_lens[0], d)
    else:
        s["q"] = normal(sum(q_lens), qh, d)
        s["kw"]["q_indptr"] = _prefix(q_lens)
    if case["kind"] != "decode":
        s["kw"]["is_causal" if case["kind"] == "prefill" else "causal"] = case["causal"]

    if case["layout"] == "dense":
        s["k"], s["v"] = (normal(batch, kvh, lens[0], d) for _ in range(2))
    elif case["layout"] == "ragged":
        s["k"], s["v"] = (normal(sum(lens), kvh, d) for _ in range(2))
        s["kw"]["kv_indptr"] = _prefix(lens)
    else:
        # one pool of pages, each sequence's pages anywhere in it; K and V have tables of their own
        page = case["page"]
        blocks = [-(-n // page) for n in lens]
        s["k"], s["v"] = (normal(sum(blocks) * page, kvh, d) for _ in range(2))
        s["kw"]["kv_indptr"] = torch.tensor(lens, dtype=torch.int32).cuda()
        s["kw"]["kv_page_size"] = page
        host = torch.Generator().manual_seed(seed)
        for name in ("k_block_table", "v_block_table"):
            perm = torch.randperm(sum(blocks), generator=host).to(torch.int32)
            table, at = torch.full((batch, max(blocks)), -1, dtype=torch.int32), 0
            for i, n in enumerate(blocks):
                table[i, :n] = perm[at:at + n]
                at += n
            s["kw"][name] = table.cuda()
        if case["append"]:
            s["k_new"], s["v_new"] = (normal(batch * case["append"], kvh, d) for _ in range(2))
            s["new_indptr"] = _prefix([case["append"]] * batch)
            s["new_pos"] = torch.tensor([n - case["append"] for n in lens], dtype=torch.int32).cuda()
    return s


def run(state):
    case = state["case"]
    if case["kind"] == "softmax":
        return log_softmax(state["x"]) if case["log"] else softmax(state["x"])
    q, k, v, kw = state["q"], state["k"], state["v"], state["kw"]
    if case["append"]:
        append_paged_kv(k, kw["k_block_table"], state["k_new"], state["new_indptr"], case["page"], dst_pos=state["new_pos"])
        append_paged_kv(v, kw["v_block_table"], state["v_new"], state["new_indptr"], case["page"], dst_pos=state["new_pos"])
    if case["kind"] == "prefill":
        out = flash_attention_v2(q, k, v, **kw)
    elif case["kind"] == "decode":
        out = decode_attention(q, k, v, **kw)
    else:
        out = speculative_decode_attention(q, k, v, **kw)
    return (out, k, v) if case["append"] else out


def work(case):
    size = SIZE[case["dtype"]]
    if case["kind"] == "softmax":
        n = case["rows"] * case["cols"]
        return {"bytes": 2 * n * size, "flops": 5 * n}
    lens, q_lens = _lengths(case), _q_lengths(case)
    row_q, row_kv = case["q_heads"] * case["head_dim"] * size, case["kv_heads"] * case["head_dim"] * size
    if case["kind"] == "prefill" and case["causal"]:
        pairs = sum(n * (n + 1) // 2 for n in lens)
    else:
        pairs = sum(m * n for m, n in zip(q_lens, lens))
    moved = 2 * sum(q_lens) * row_q + 2 * sum(lens) * row_kv
    # an appended row is read once and written once; the attention call then reads it with the rest of the cache
    moved += 2 * 2 * case["append"] * case["batch"] * row_kv
    if case["layout"] == "paged":
        moved += 2 * 4 * sum(-(-n // case["page"]) for n in lens)
    return {"bytes": moved, "flops": 4 * case["head_dim"] * case["q_heads"] * pairs}


def tolerance(case):
    """Relative errors of another correct implementation at the same precision: the probabilities and the output are
    rounded to the 16-bit type.  fp32 prefill and speculative decode multiply in 16 bits with ten mantissa bits, as the
    kernels that they stand in for do; fp32 decode and softmax are 32-bit arithmetic throughout."""
    if case["dtype"] == "bf16":
        return {"rel": 1e-2}
    if case["dtype"] == "fp16" or case["kind"] in ("prefill", "spec"):
        return {"rel": 2e-3}
    return {"rel": 1e-5}
