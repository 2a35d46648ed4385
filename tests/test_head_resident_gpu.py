"""Head-resident kernel at the edges of its tiles and of its launch shapes (state in shared memory, y in the workspace,
clusters of CTAs), against the CPU oracle; and the bits do not depend on how many heads share a launch."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [  # E, H, N, D, B, T, pad, mask
    (1, 1, 1, 8, 1, 1, "post", "none"), (1, 2, 225, 64, 15, 1, "pre", "rand"), (2, 12, 197, 64, 15, 2, "pre", "none"),
    (1, 3, 256, 64, 16, 3, "post", "none"), (2, 2, 17 * 16 - 3, 40, 17, 2, "post", "block"),
    (1, 12, 512, 64, 32, 1, "post", "tail"), (3, 4, 1024, 72, 32, 2, "pre", "none"), (1, 1, 1023, 80, 32, 3, "pre", "rand"),
    (2, 1, 32 * 7, 32, 7, 2, "post", "block"), (1, 5, 33, 16, 32, 2, "pre", "none"), (40, 4, 31 * 32, 64, 31, 2, "post", "none"),
    (30, 10, 200, 24, 14, 2, "pre", "rand")]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("E,H,N,D,B,T,pad,mask", SHAPES)
def test_head_resident_kernel_matches_the_oracle(E, H, N, D, B, T, pad, mask, dtype):
    import monarch_attention_b200 as ma
    from oracle.monarch_oracle import monarch_attention_oracle
    g = torch.Generator().manual_seed(N * 7 + D)
    q, k, v = (torch.randn(E, H, N, D, generator=g).to(dtype) for _ in range(3))
    m = None
    if mask != "none":
        m = torch.rand(E, N, generator=g) > (0.3 if mask == "rand" else 0.0)
        if mask == "block":
            m[:, B:3 * B] = False
        if mask == "tail":
            m[0, N // 3:] = False
        m[:, 0] = True
    dev = torch.device("cuda:0")
    args = [t.to(dev) for t in (q, k, v)] + [None if m is None else m.to(dev)]
    mod = ma.MonarchAttention(B, T, pad, impl="b200-head-resident")
    out = mod(*args)
    ref = monarch_attention_oracle(q, k, v, m, T, B, pad == "pre").float()
    err = ((out.cpu().float() - ref).norm() / ref.norm()).item()
    assert torch.isfinite(out.float()).all() and err <= (1e-2 if dtype == torch.bfloat16 else 2e-3), err
    assert torch.equal(mod(*args), out)
    one = mod(*(t[:1, :1] for t in args[:3]), None if m is None else args[3][:1])
    assert torch.equal(one, out[:1, :1])
