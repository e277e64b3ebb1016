"""A process whose very first attention call is recorded into a CUDA graph: what the library asks the driver once (attributes of its
kernels, clusters that the GPU holds) it asks while the stream records."""
import subprocess
import sys

import pytest

from test_decode_routes import route
from test_prefill_routes import route as prefill_route

CODE = """
import sys
sys.path[:0] = [{pkg!r}]
import torch
from kernels import decode_attention, flash_attention_v2
g = torch.Generator(device="cuda").manual_seed(1)
q, k, v = (torch.randn(s, generator=g, device="cuda", dtype=torch.bfloat16) for s in {shapes!r})
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph, capture_error_mode={mode!r}):
    out = decode_attention(q, k, v) if q.dim() == 3 else flash_attention_v2(q, k, v)
graph.replay()
torch.cuda.synchronize()
k, v = (t.double().repeat_interleave(4, 1) for t in (k, v))
q4 = q.double().unsqueeze(2) if q.dim() == 3 else q.double()
ref = torch.softmax((q4 @ k.transpose(-1, -2)) / q.shape[-1] ** 0.5, -1) @ v
assert (out.double().view(ref.shape) - ref).abs().max().item() < 2e-2
print("ok")
"""


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["global", "thread_local"])
@pytest.mark.parametrize("shapes", [((4, 32, 128), (4, 8, 300, 128), (4, 8, 300, 128)), ((1, 8, 100, 64), (1, 2, 600, 64), (1, 2, 600, 64))],
                         ids=["decode", "prefill"])
def test_first_call_is_recorded(shapes, mode):
    """Both calls go in clusters."""
    from kernels import _native

    assert route("dense", "bf16", 4, 32, 8, 128, 300) == 8
    assert prefill_route("dense", "bf16", 1, 8, 2, 100, 600, False, 64) == 4
    done = subprocess.run([sys.executable, "-c", CODE.format(pkg=_native._PKG_ROOT, mode=mode, shapes=shapes)], capture_output=True,
                          text=True, timeout=300)
    assert done.returncode == 0 and "ok" in done.stdout, done.stderr[-2000:]
