"""fp32 tensor-core stage kernels (operands split into two tf32 parts) at the edges of their tiles, against the CPU
oracle in fp32."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [  # E, H, N, D, B, T, pad, masked
    (1, 1, 1, 24, 1, 1, "post", False), (2, 3, 250, 64, 16, 2, "pre", True), (1, 2, 289, 72, 17, 3, "post", False),
    (1, 2, 33 * 31 - 5, 32, 33, 2, "pre", True), (1, 1, 65 * 64, 80, 65, 1, "post", False),
    (1, 1, 128 * 128 - 77, 40, 128, 2, "post", True), (2, 1, 16 * 128, 80, 16, 2, "pre", False)]


@pytest.mark.parametrize("E,H,N,D,B,T,pad,masked", SHAPES)
def test_fp32_tensor_core_kernels_match_the_oracle(E, H, N, D, B, T, pad, masked):
    import monarch_attention_b200 as ma
    from oracle.monarch_oracle import monarch_attention_oracle
    g = torch.Generator().manual_seed(N)
    q, k, v = (torch.randn(E, H, N, D, generator=g) for _ in range(3))
    mask = None
    if masked:
        mask = torch.rand(E, N, generator=g) > 0.3
        mask[:, B:2 * B] = False         # a key block without valid keys
        mask[:, 0] = True
    dev = torch.device("cuda:0")
    out = ma.MonarchAttention(B, T, pad, impl="b200-tf32x3")(q.to(dev), k.to(dev), v.to(dev),
                                                             None if mask is None else mask.to(dev)).cpu()
    ref = monarch_attention_oracle(q, k, v, mask, T, B, pad == "pre")
    assert ((out - ref).norm() / ref.norm()).item() <= 5e-6
    assert (out - ref).abs().max().item() <= 2e-5 * ref.abs().max().item()
