"""Warp-level kernels, forward and backward, at the edges of every tile width (key columns padded to 16, 32, 48, 64, 80, 96, 112, 128)."""
import pytest
import torch
from test_backward_gpu import _exact

pytestmark = pytest.mark.gpu

SIDES = [(33, 48), (48, 33), (49, 64), (65, 80), (80, 66), (81, 96), (97, 112), (112, 98), (113, 17), (47, 128)]  # B, M


def _inputs(B, M, D, dtype, count):
    g = torch.Generator().manual_seed(B * 131 + M)
    N = B * M - 3
    x = [torch.randn(1, 2, N, D, generator=g).to(dtype) for _ in range(count)]
    m = torch.rand(1, N, generator=g) > 0.2
    m[:, :B] = False
    m[:, -1] = True
    return x, m


@pytest.mark.parametrize("B,M", SIDES)
@pytest.mark.parametrize("dtype,impl,D,tol", [(torch.float32, "b200-tf32x3", 72, 5e-6), (torch.bfloat16, "b200-warp-mma", 80, 1e-2),
                                              (torch.float16, "b200-warp-mma", 40, 2e-3)])
def test_forward_matches_the_oracle(B, M, dtype, impl, D, tol):
    import monarch_attention_b200 as ma
    from oracle.monarch_oracle import monarch_attention_oracle
    (q, k, v), m = _inputs(B, M, D, dtype, 3)
    dev = torch.device("cuda:0")
    out = ma.MonarchAttention(B, 2, "pre", impl=impl)(q.to(dev), k.to(dev), v.to(dev), m.to(dev)).cpu().float()
    ref = monarch_attention_oracle(q, k, v, m, 2, B, True).float()
    assert ((out - ref).norm() / ref.norm()).item() <= tol


@pytest.mark.parametrize("B,M", SIDES)
@pytest.mark.parametrize("dtype,D,tol", [(torch.float32, 32, 1e-5), (torch.bfloat16, 64, 1.5e-2), (torch.float16, 80, 2e-3)])
def test_gradients_match_float64(B, M, dtype, D, tol):
    import monarch_attention_b200 as ma
    if dtype == torch.float32 and max(B, M) > 64:
        pytest.skip("fp32 backward kernels end at blocks of 64")
    dev = torch.device("cuda:0")
    x, m = _inputs(B, M, D, dtype, 4)
    (q, k, v, w), m = [t.to(dev) for t in x], m.to(dev)
    exact = [t.double().requires_grad_(True) for t in (q, k, v)]
    want = torch.autograd.grad(_exact(*exact, m, 2, B, True), exact, w.double())
    for t in (q, k, v):
        t.requires_grad_(True)
    got = torch.autograd.grad(ma.MonarchAttention(B, 2, "pre")(q, k, v, m), (q, k, v), w)
    for name, a, b in zip(("dq", "dk", "dv"), got, want):
        err = ((a.double() - b).norm() / b.norm()).item()
        assert err <= tol, (name, err)
