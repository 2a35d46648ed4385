"""The first call of a process inside a stream capture: whatever the library sets up once per device must not disturb it.
Each case is a process of its own, since an earlier call would have done the set-up."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = """
import sys; sys.path.insert(0, {root!r})
import torch, monarch_attention_b200 as ma
E, H, N, D, B, T = {shape}
g = torch.Generator().manual_seed(1)
dt = torch.{dtype}
q, k, v = (torch.randn(E, H, N, D, generator=g).to(dt).cuda() for _ in range(3))
mod = ma.MonarchAttention(B, T, "post")
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    out = mod(q, k, v)
graph.replay()
torch.cuda.synchronize()
assert torch.equal(out, mod(q, k, v))
print("family ok")
"""


@pytest.mark.parametrize("shape,dtype", [
    ((4, 12, 3000, 64, 60, 2), "float16"),      # tile kernels, one launch
    ((1, 4, 200 * 180, 64, 200, 2), "bfloat16"),  # tile kernels, a launch per stage
    ((1, 4, 4096, 64, 64, 2), "bfloat16"),      # fused kernel
    ((2, 12, 197, 64, 15, 2), "bfloat16"),      # head-resident kernel
    ((1, 2, 40 * 60, 80, 40, 2), "bfloat16"),   # warp-level kernels
    ((2, 12, 256, 64, 16, 2), "float32"),       # fp32 tensor path, one launch
    ((2, 13, 576, 64, 24, 2), "float32"),       # ... where a query decides whether the heads fit
    ((20, 8, 256, 64, 16, 2), "float32"),       # ... a launch per stage
    ((1, 2, 250, 20, 16, 2), "float32")])       # generic kernels
def test_first_call_of_a_process_can_be_captured(shape, dtype):
    run = subprocess.run([sys.executable, "-c", SCRIPT.format(root=ROOT, shape=shape, dtype=dtype)], capture_output=True, text=True,
                         timeout=300)
    assert run.returncode == 0 and "family ok" in run.stdout, run.stderr[-2000:]
