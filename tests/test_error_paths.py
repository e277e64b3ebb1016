"""The bounded waits, made to run out without hanging anything: a self-test kernel of the library waits on a barrier
that nothing completes, with the kernels' own wait loop and a small try limit, gives up, records the error code the
attention kernels would record and returns.  The host then reads the code and the context stays usable."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_wait_expiry_is_reported_and_the_context_survives():
    from kernels import _native, flash_attention_v2

    lib = _native.lib()
    dev = torch.device("cuda")
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    ws = torch.zeros(256, dtype=torch.uint8, device=dev)
    _native.check(lib.b200attn_selftest_wait_expiry(torch.cuda.current_device(), C.c_void_p(ws.data_ptr()), 1 << 12, stream),
                  "b200attn_selftest_wait_expiry")
    code = C.c_int32(0)
    rc = lib.b200attn_check_workspace(C.c_void_p(ws.data_ptr()), stream, C.byref(code))
    assert rc == -6 and code.value == 1, (rc, code.value, _native.last_error())
    assert "bounded wait expired" in _native.last_error()
    # the word was cleared, and a second check is clean
    assert lib.b200attn_check_workspace(C.c_void_p(ws.data_ptr()), stream, C.byref(code)) == 0 and code.value == 0
    # the context is intact: a following attention call runs and is right
    g = torch.Generator().manual_seed(0)
    q = torch.randn((1, 4, 40, 64), generator=g).half().to(dev)
    k = torch.randn((1, 4, 40, 64), generator=g).half().to(dev)
    v = torch.randn((1, 4, 40, 64), generator=g).half().to(dev)
    out = flash_attention_v2(q, k, v, is_causal=True)
    ref = torch.nn.functional.scaled_dot_product_attention(q.float(), k.float(), v.float(), is_causal=True)
    torch.testing.assert_close(out.float(), ref, atol=1e-2, rtol=1e-2)


def test_wait_expiry_selftest_rejects_unbounded_limits():
    from kernels import _native

    lib = _native.lib()
    ws = torch.zeros(256, dtype=torch.uint8, device="cuda")
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert lib.b200attn_selftest_wait_expiry(torch.cuda.current_device(), C.c_void_p(ws.data_ptr()), 0, stream) == -1
    assert lib.b200attn_selftest_wait_expiry(torch.cuda.current_device(), C.c_void_p(ws.data_ptr()), (1 << 20) + 1, stream) == -1
    assert lib.b200attn_selftest_wait_expiry(torch.cuda.current_device(), None, 16, stream) == -1


@pytest.mark.parametrize("late", [0, 1])
def test_cluster_waits_for_a_late_cta_before_it_leaves(late):
    """A decode CTA that gave up on a peer's part reports it, and is still there when the part arrives."""
    from kernels import _native

    lib = _native.lib()
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    ws = torch.zeros(256, dtype=torch.uint8, device="cuda")
    out = torch.full((65,), -1.0, device="cuda")
    _native.check(lib.b200attn_selftest_cluster_expiry(torch.cuda.current_device(), C.c_void_p(ws.data_ptr()),
                                                       C.c_void_p(out.data_ptr()), 1 << 10, late, stream),
                  "b200attn_selftest_cluster_expiry")
    code = C.c_int32(0)
    rc = lib.b200attn_check_workspace(C.c_void_p(ws.data_ptr()), stream, C.byref(code))
    assert (rc, code.value) == ((-6, 1) if late else (0, 0))
    assert out[64] == 1, "the first CTA left while the second still had stores on the way to it"
    assert (out[32:64] == 1.5).all()                 # the second CTA's half: the mean of 1 and 2
    assert torch.isnan(out[:32]).all() if late else (out[:32] == 1.5).all()


def test_cluster_selftest_rejects_what_it_cannot_bound():
    from kernels import _native

    lib = _native.lib()
    stream, dev = C.c_void_p(torch.cuda.current_stream().cuda_stream), torch.cuda.current_device()
    ws, out = torch.zeros(256, dtype=torch.uint8, device="cuda"), torch.zeros(65, device="cuda")
    w, o = C.c_void_p(ws.data_ptr()), C.c_void_p(out.data_ptr())
    for args in ((w, o, 0), (w, o, (1 << 14) + 1), (None, o, 16), (w, None, 16)):
        assert lib.b200attn_selftest_cluster_expiry(dev, *args, 1, stream) == -1


@pytest.mark.parametrize("ended", [0, 1])
@pytest.mark.parametrize("published", [1, 2, 4, 5, 6, 7, 8, 9, 13])
@pytest.mark.parametrize("abort_round", [0, 3, 6, 1 << 30])
def test_every_unfinished_unit_of_a_cta_that_gave_up_is_nan(published, ended, abort_round):
    """A persistent decode CTA holds the last four entries of its list, the end mark among them; which of those units are finished
    is known from `abort_round` on (0: of none)."""
    from kernels import _native

    out = torch.zeros((64, 64), device="cuda")
    _native.check(_native.lib().b200attn_selftest_abandoned_units(torch.cuda.current_device(), C.c_void_p(out.data_ptr()), published, ended,
                                                                  abort_round, C.c_void_p(torch.cuda.current_stream().cuda_stream)),
                  "b200attn_selftest_abandoned_units")
    want = torch.zeros(64, dtype=torch.bool)
    want[max(0, published - 4, abort_round): published - ended] = True
    assert torch.equal(torch.isnan(out).all(1).cpu(), want) and (out[~want.cuda()] == 0).all()
