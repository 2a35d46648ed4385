"""The single launch of the fp32 tensor path (few heads, blocks up to 32) against the CPU oracle, and against the launch per
stage that a call of more heads takes: the same bits, so that parts of a call agree with the whole."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("few,many,N,D,B,T,pad,masked", [
    (1, 150, 256, 72, 16, 3, "post", False), (100, 150, 15 * 14 - 3, 64, 15, 2, "pre", True), (3, 2100, 1, 24, 1, 1, "post", False),
    (2, 300, 9 * 16 - 8, 80, 9, 2, "post", False), (129, 160, 16 * 16, 32, 16, 1, "pre", True),
    (1, 16, 1024, 64, 32, 2, "post", False), (3, 30, 17 * 30 - 9, 72, 17, 3, "pre", True), (5, 40, 32 * 10 - 1, 40, 32, 2, "post", True),
    (140, 150, 256, 64, 16, 3, "post", False), (30, 40, 24 * 23 - 5, 64, 24, 2, "pre", True)])
def test_single_launch_returns_the_bits_of_the_stage_kernels(few, many, N, D, B, T, pad, masked):
    import monarch_attention_b200 as ma
    from oracle.monarch_oracle import monarch_attention_oracle
    g = torch.Generator().manual_seed(N + D)
    q, k, v = (torch.randn(many, 1, N, D, generator=g) for _ in range(3))
    mask = None
    if masked:
        mask = torch.rand(many, N, generator=g) > 0.3
        mask[:, B:2 * B] = False         # a key block without valid keys
        mask[:, 0] = True
    mod = ma.MonarchAttention(B, T, pad, impl="b200-tf32x3")
    whole = mod(q.cuda(), k.cuda(), v.cuda(), None if mask is None else mask.cuda())
    part = mod(q[:few].cuda(), k[:few].cuda(), v[:few].cuda(), None if mask is None else mask[:few].cuda())
    assert torch.equal(part, whole[:few])
    n = min(few, 3)
    ref = monarch_attention_oracle(q[:n], k[:n], v[:n], None if mask is None else mask[:n], T, B, pad == "pre")
    assert ((part[:n].cpu() - ref).norm() / ref.norm()).item() <= 5e-6  # as for the stage kernels
