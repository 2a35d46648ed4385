"""Few heads are shared out by columns over CTAs: with parts of one column, of some, of 16, a smaller last one, and beside the line
to one CTA a head, every head has the bits it has among many."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [  # heads, N, D, B, T, pad; 148 SMs: parts x columns (last)
    (1, 20 * 9, 64, 20, 2, "post"),        # 20 x 1
    (10, 31 * 30 - 7, 72, 31, 2, "pre"),   # 11 x 3 (1)
    (48, 32 * 32, 64, 32, 3, "post"),      # 3 x 11 (10)
    (60, 29 * 17 - 5, 80, 29, 1, "pre"),   # 2 x 15 (14)
    (74, 32 * 20, 40, 32, 2, "post"),      # 2 x 16
    (75, 32 * 20, 40, 32, 2, "post"),      # one CTA a head
    (148, 16 * 13, 32, 16, 2, "pre"),      # 1 x 16
    (149, 16 * 13, 64, 16, 2, "pre"),      # one CTA a head
    (3, 5 * 32 - 1, 24, 5, 2, "post")]     # 5 x 1


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("H,N,D,B,T,pad", SHAPES)
def test_parts_of_a_head_have_the_bits_of_the_whole(H, N, D, B, T, pad, masked, dtype):
    import monarch_attention_b200 as ma
    g = torch.Generator(device="cuda").manual_seed(N + D)
    many = 300  # one CTA a head
    q, k, v = (torch.randn(1, many, N, D, generator=g, device="cuda").to(dtype) for _ in range(3))
    m = (torch.rand(1, N, generator=g, device="cuda") > 0.3) if masked else None
    mod = ma.MonarchAttention(B, T, pad, impl="b200-head-resident")
    want = mod(q, k, v, m)
    some = [t[:, 100:100 + H].permute(0, 2, 1, 3).contiguous().permute(0, 2, 1, 3) for t in (q, k, v)]
    assert torch.equal(mod(*some, m), want[:, 100:100 + H])
    assert torch.isfinite(want.float()).all()
