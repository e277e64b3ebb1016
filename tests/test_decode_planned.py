"""Decode calls that are cut into items, by the CTAs themselves or by the planner, at sizes where clusters do not take them: each
test asks the library which way its call goes before it makes it."""
import threading

import pytest
import torch

from helpers import assert_close_both
from oracle import sdpa_ref
from test_decode_routes import INLINE, PLANNER, route
from test_decode_without_planner import _call, _problem, _reference

pytestmark = pytest.mark.gpu
DEV = "cuda"
NAMES = {torch.bfloat16: "bf16", torch.float16: "fp16", torch.float32: "fp32"}


def _route(lens, layout, dtype, qh, kvh, d, m=1, page=16):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return route(layout, NAMES[dtype], len(lens), qh, kvh, d, max(lens), m=m, total=sum(lens), page=page, sms=sms)


# either side of the line between the two plans (96 pairs of sequence and KV head), every layout, lengths around tiles
@pytest.mark.parametrize("layout,page", [("dense", 0), ("ragged", 0), ("paged", 16), ("paged", 24)])
@pytest.mark.parametrize("batch,qh,kvh,want", [(1, 8, 1, INLINE), (4, 32, 8, INLINE), (12, 8, 8, INLINE), (13, 8, 8, PLANNER),
                                               (97, 2, 1, PLANNER)])
def test_planned_layouts(layout, page, batch, qh, kvh, want):
    gen = torch.Generator(device=DEV).manual_seed(batch * 17 + qh)
    longest = 20000 if batch <= 4 else 9000
    base = [longest, 1, 63, 64, 65, 127, 129, 640, 1000, 2500]
    lens = [longest] * batch if layout == "dense" else [base[i % len(base)] for i in range(batch)]
    for m in (0, 2):
        shape = (qh, 64) if m == 0 else (qh, m, 64)
        qs = [torch.randn(shape, generator=gen, device=DEV).bfloat16() for _ in lens]
        ks, vs = ([torch.randn((max(n, m), kvh, 64), generator=gen, device=DEV).bfloat16() for n in lens] for _ in range(2))
        assert _route([len(k) for k in ks], layout, torch.bfloat16, qh, kvh, 64, max(1, m), page or 16) == want
        out = _call(qs, ks, vs, layout, m, page or 16)
        assert_close_both(out, _reference(qs, ks, vs, qh, kvh, m), torch.bfloat16, longest, f"{layout} {batch}x{kvh} m{m}")


@pytest.mark.parametrize("batch,want", [(5, INLINE), (50, PLANNER)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32], ids=["fp16", "fp32"])
def test_empty_sequences(batch, want, dtype):
    gen = torch.Generator().manual_seed(5)
    lens = ([0, 20000, 0, 3, 0] * batch)[:batch]
    assert _route(lens, "ragged", dtype, 8, 2, 64) == want
    qs, ks, vs = _problem(gen, lens, 8, 2, 64, dtype)
    out = _call(qs, ks, vs, "ragged", 0)
    live = [i for i, n in enumerate(lens) if n]
    ref = _reference([qs[i] for i in live], [ks[i] for i in live], [vs[i] for i in live], 8, 2, 0)
    assert_close_both(out[live], ref, dtype, 20000)
    assert (out[[i for i, n in enumerate(lens) if not n]] == 0).all()


def _jobs(seed, sizes, kvh=8, d=64):
    """Packed decode calls of ``sizes`` = (batch, longest): the calls and the routes that they take."""
    from kernels import decode_attention

    gen = torch.Generator(device=DEV).manual_seed(seed)
    jobs, routes = [], []
    for batch, longest in sizes:
        lens = [longest // (1 + i % 5) for i in range(batch)]
        q = torch.randn((batch, 8, d), generator=gen, device=DEV).bfloat16()
        k, v = (torch.randn((sum(lens), kvh, d), generator=gen, device=DEV).bfloat16() for _ in range(2))
        indptr = torch.tensor([0] + lens, device=DEV).cumsum(0).int()
        routes.append(_route(lens, "ragged", torch.bfloat16, 8, kvh, d))
        jobs.append(lambda q=q, k=k, v=v, indptr=indptr: decode_attention(q, k, v, kv_indptr=indptr))
    return jobs, routes


def test_plans_of_two_streams_do_not_meet():
    """Planner tables, partials and tickets belong to a stream's workspace: calls of two streams overlap on the GPU."""
    (a, b), routes = _jobs(1, [(40, 3000), (20, 5000)])
    assert routes == [PLANNER, PLANNER]
    (c, e), routes = _jobs(2, [(4, 9000), (7, 7000)])
    assert routes == [INLINE, INLINE]
    want = [[j() for j in pair] for pair in ((a, c), (b, e))]
    torch.cuda.synchronize()
    streams, got = [torch.cuda.Stream(), torch.cuda.Stream()], [[], []]
    for _ in range(40):
        for s, (stream, pair) in enumerate(zip(streams, ((a, c), (b, e)))):
            with torch.cuda.stream(stream):
                got[s].append([j() for j in pair])
    torch.cuda.synchronize()
    for outs, refs in zip(got, want):
        for pair in outs:
            assert all(torch.equal(x, y) for x, y in zip(pair, refs))


def test_plans_of_two_threads_on_one_stream_do_not_mix():
    """Planner and kernel of a call stay together."""
    jobs, routes = _jobs(3, [(13, 3000), (40, 1000)])
    assert routes == [PLANNER, PLANNER]
    want = [job() for job in jobs]
    torch.cuda.synchronize()
    wrong = []

    def run(job, ref):
        for i in range(300):
            out = job()
            if i % 10 == 9 and not torch.equal(out, ref):
                wrong.append(i)

    threads = [threading.Thread(target=run, args=a) for a in zip(jobs, want)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not wrong


@pytest.mark.parametrize("kvh,want", [(8, INLINE), (32, PLANNER)])
def test_calls_in_a_row_see_each_other(kvh, want):
    """A table much wider than the sequences are: planned, and every call reads rows that the append before it wrote."""
    from kernels import append_paged_kv, decode_attention, softmax

    gen = torch.Generator().manual_seed(9)
    batch, d, page, steps, pages = 4, 128, 16, 24, 700
    assert _route([pages * page] * batch, "paged", torch.bfloat16, kvh, kvh, d, page=page) == want
    table = torch.full((batch, pages), -1, dtype=torch.int32)
    table[:, :20] = torch.randperm(batch * 20, generator=gen).to(torch.int32).view(batch, 20)
    table = table.to(DEV)
    q0 = torch.randn((batch, kvh, d), generator=gen).bfloat16().to(DEV)
    new = torch.randn((batch * 8, kvh, d), generator=gen).bfloat16().to(DEV)
    indptr = torch.arange(0, 8 * batch + 1, 8, dtype=torch.int32, device=DEV)

    def run(sync):
        wait = torch.cuda.synchronize if sync else (lambda: None)
        k = torch.zeros((batch * 20 * page, kvh, d), dtype=torch.bfloat16, device=DEV)
        v = torch.zeros_like(k)
        x, outs = q0, []
        for s in range(steps):
            pos = torch.full((batch,), 8 * s, dtype=torch.int32, device=DEV)
            lens = pos + 8
            wait()
            append_paged_kv(k, table, new, indptr, page, dst_pos=pos)
            wait()
            append_paged_kv(v, table, softmax(new), indptr, page, dst_pos=pos)
            wait()
            x = decode_attention(x, k, v, kv_indptr=lens, k_block_table=table, v_block_table=table, kv_page_size=page)
            wait()
            x = softmax(x)
            wait()
            outs.append(x)
        torch.cuda.synchronize()
        return [*outs, k, v]

    for a, b in zip(run(True), run(False)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("dtype,qh,kvh,m,batch,width", [("fp32", 8, 8, 1, 24, 3200), ("fp32", 4, 4, 1, 26, 5888), ("bf16", 64, 8, 5, 12, 2848),
                                                        ("fp16", 8, 1, 5, 90, 992), ("bf16", 8, 8, 1, 12, 8000)])
def test_tables_wider_than_the_sequences(dtype, qh, kvh, m, batch, width):
    """Grids are as large as the table's width asks for, and most CTAs of a call that plans for itself find that these lengths leave
    nothing for them: no sequence at all, one key, items that end on and around the shortest (128 to 320 keys), one long sequence."""
    kind = {v: k for k, v in NAMES.items()}[dtype]
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert route("paged", dtype, batch, qh, kvh, 64, width, m=m, sms=sms) == INLINE
    gen = torch.Generator().manual_seed(width)
    for base in ([m], [128], [129, 127], [320, 321, 640, 639], [m + 1] * (batch - 1) + [width]):
        lens = [base[i % len(base)] for i in range(batch)]
        qs, ks, vs = _problem(gen, lens, qh, kvh, 64, kind, m if m > 1 else 0)
        k, kt, n = sdpa_ref.pack_paged(ks, 16, permute_seed=1, extra_pages=2, pad_value=-1, poison=float("nan"))
        v, vt, _ = sdpa_ref.pack_paged(vs, 16, permute_seed=2, extra_pages=2, pad_value=-1, poison=float("nan"))
        kt, vt = (torch.nn.functional.pad(t, (0, width // 16 - t.shape[1]), value=-1).contiguous() for t in (kt, vt))
        kw = dict(kv_indptr=n, k_block_table=kt, v_block_table=vt, kv_page_size=16)
        from kernels import decode_attention, speculative_decode_attention

        q = torch.stack(qs)
        out = decode_attention(q, k, v, **kw) if m == 1 else speculative_decode_attention(q, k, v, causal=True, **kw)
        ref = _reference(qs, ks, vs, qh, kvh, m if m > 1 else 0)
        assert_close_both(out, ref, kind, max(lens), f"{base[:4]}")
