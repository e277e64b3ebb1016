"""A process whose very first decode call is recorded into a CUDA graph: what the library asks the driver once (attributes of its
kernels, clusters that the GPU holds) it asks while the stream records."""
import subprocess
import sys

import pytest

from test_decode_routes import route

CODE = """
import sys
sys.path[:0] = [{pkg!r}]
import torch
from kernels import decode_attention
g = torch.Generator(device="cuda").manual_seed(1)
q, k, v = (torch.randn(s, generator=g, device="cuda", dtype=torch.bfloat16) for s in ((4, 32, 128), (4, 8, 300, 128), (4, 8, 300, 128)))
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph, capture_error_mode={mode!r}):
    out = decode_attention(q, k, v)
graph.replay()
torch.cuda.synchronize()
k, v = (t.double().repeat_interleave(4, 1) for t in (k, v))
ref = torch.softmax((q.double().unsqueeze(2) @ k.transpose(-1, -2)) / 128 ** 0.5, -1) @ v
assert (out.double() - ref.squeeze(2)).abs().max().item() < 2e-2
print("ok")
"""


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["global", "thread_local"])
def test_first_call_is_recorded(mode):
    from kernels import _native

    assert route("dense", "bf16", 4, 32, 8, 128, 300) == 8
    done = subprocess.run([sys.executable, "-c", CODE.format(pkg=_native._PKG_ROOT, mode=mode)], capture_output=True, text=True,
                          timeout=300)
    assert done.returncode == 0 and "ok" in done.stdout, done.stderr[-2000:]
