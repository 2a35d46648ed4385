"""Gradients where the stage inputs are recomputed by one launch of the head-resident kernel: heads in parts of some columns with a smaller
last one, one CTA a head, both tile sizes on either side, every width that has tiles of its own, and beside the line to a launch
per stage (148 SMs)."""
import pytest
import torch
from test_backward_gpu import _exact

pytestmark = pytest.mark.gpu

SHAPES = [  # heads, N, D, B, T, pad
    (3, 32 * 31 - 5, 64, 32, 2, "pre"), (48, 21 * 20, 72, 21, 3, "post"), (74, 32 * 17, 32, 32, 2, "post"), (75, 32 * 17, 32, 32, 2, "post"),
    (20, 16 * 29 - 2, 80, 16, 2, "pre"), (149, 12 * 30, 64, 12, 2, "post"), (149, 30 * 12 - 7, 72, 30, 2, "pre"), (150, 15 * 13, 80, 15, 3, "post")]


@pytest.mark.parametrize("dtype,tol", [(torch.bfloat16, 1.5e-2), (torch.float16, 2e-3)])
@pytest.mark.parametrize("H,N,D,B,T,pad", SHAPES)
def test_gradients_match_float64(H, N, D, B, T, pad, dtype, tol):
    import monarch_attention_b200 as ma
    g = torch.Generator(device="cuda").manual_seed(N + H)
    q, k, v, w = (torch.randn(1, N, H, D, generator=g, device="cuda").to(dtype).permute(0, 2, 1, 3) for _ in range(4))
    m = torch.rand(1, N, generator=g, device="cuda") > 0.25
    m[:, B:2 * B] = False
    exact = [t.double().requires_grad_(True) for t in (q, k, v)]
    want = torch.autograd.grad(_exact(*exact, m, T, B, pad == "pre"), exact, w.double())
    for t in (q, k, v):
        t.requires_grad_(True)
    runs = [torch.autograd.grad(ma.MonarchAttention(B, T, pad)(q, k, v, m), (q, k, v), w) for _ in range(2)]
    for name, a, again, b in zip(("dq", "dk", "dv"), *runs, want):
        err = ((a.double() - b).norm() / b.norm()).item()
        assert err <= tol and torch.equal(a, again), (name, err)
