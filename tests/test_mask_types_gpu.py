"""Masks are read in the type they come in: every type gives the bits of the boolean mask, in every kernel family."""
import pytest
import torch

pytestmark = pytest.mark.gpu

TYPES = [torch.uint8, torch.int8, torch.int16, torch.int32, torch.int64, torch.float16, torch.bfloat16, torch.float32, torch.float64]


@pytest.mark.parametrize("shape", [(2, 3, 200, 64, 15, 2, torch.bfloat16), (2, 2, 2000, 64, 45, 2, torch.bfloat16),
                                   (2, 2, 200, 72, 40, 2, torch.float16), (2, 2, 250, 64, 16, 2, torch.float32),
                                   (2, 2, 250, 20, 16, 2, torch.float32)],
                         ids=["head-resident", "tile", "warp-mma", "tf32x3", "generic"])
def test_mask_types_are_equivalent(shape):
    import monarch_attention_b200 as ma
    E, H, N, D, B, T, dt = shape
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(1)
    q, k, v = (torch.randn(E, H, N, D, generator=g, device=dev).to(dt).requires_grad_(D != 20) for _ in range(3))
    keep = torch.rand(E, N, generator=g, device=dev) > 0.3
    keep[:, 0] = True
    mod = ma.MonarchAttention(B, T, "pre")
    want = mod(q, k, v, keep)
    for t in TYPES:
        mask = keep.to(t)
        if t.is_floating_point:
            mask = torch.where(keep, mask * 0.25, torch.full_like(mask, -0.0))
        out = mod(q, k, v, mask)
        assert torch.equal(out, want), t
        if D != 20 and t in (torch.int64, torch.float32):
            w = torch.ones_like(out)
            a = torch.autograd.grad(out, (q, k, v), w)
            b = torch.autograd.grad(mod(q, k, v, keep), (q, k, v), w)
            assert all(torch.equal(x, y) for x, y in zip(a, b)), t
    wide = keep.to(torch.int64).repeat_interleave(2, dim=1)[:, ::2]    # inner stride 2
    assert torch.equal(mod(q, k, v, wide), want)
