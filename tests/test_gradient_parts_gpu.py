"""A head's gradients have the same bits whatever is beside it in the call: some heads alone, fewer than the GPU has places for and more,
as in a batch shard or a micro-batch of a training step."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(32, 32, 64, 2), (30, 31, 72, 2), (17, 20, 80, 3), (32, 32, 32, 2), (16, 16, 64, 3), (13, 30, 64, 2), (32, 9, 32, 3), (28, 16, 72, 2),
          (16, 25, 80, 2), (11, 12, 80, 2), (24, 24, 40, 2)]  # B, M, D, T


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,M,D,T", SHAPES)
def test_gradients_of_some_heads_are_those_of_the_whole_call(B, M, D, T, dtype):
    import monarch_attention_b200 as ma
    H, N = 160, B * M - 2
    g = torch.Generator(device="cuda").manual_seed(B * M + D)
    x = [torch.randn(1, H, N, D, generator=g, device="cuda").to(dtype) for _ in range(4)]
    m = torch.rand(1, N, generator=g, device="cuda") > 0.2
    mod = ma.MonarchAttention(B, T, "pre")

    def gradients(lo, hi):
        q, k, v, w = (t[:, lo:hi].contiguous() for t in x)
        for t in (q, k, v):
            t.requires_grad_(True)
        return torch.autograd.grad(mod(q, k, v, m), (q, k, v), w)

    whole = gradients(0, H)
    for lo, hi in ((0, 1), (5, 42), (31, 105), (7, 157)):
        for name, a, b in zip(("dq", "dk", "dv"), gradients(lo, hi), whole):
            assert torch.equal(a, b[:, lo:hi]), (name, lo, hi)
