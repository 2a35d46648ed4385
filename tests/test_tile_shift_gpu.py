"""Column tiles with missing columns take the shift of their exponentials from the first 16 columns and raise it where later
ones are far larger (masked_column_exps in csrc/ma_tile_common.cuh): rows whose logits grow by some 60 powers of two from the
first block to the last, or fall, or do both, against the CPU oracle."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape", ["rising", "falling", "peak"])
@pytest.mark.parametrize("B,M,T", [(64, 121, 2), (40, 60, 1), (40, 200, 2), (100, 33, 2)])
def test_shift_follows_the_largest_logit(B, M, T, shape, dtype):
    import monarch_attention_b200 as ma
    from oracle.monarch_oracle import monarch_attention_oracle
    D, N = 64, B * M
    g = torch.Generator().manual_seed(B + M)
    x = torch.linspace(0, 1, M)
    size = {"rising": x, "falling": 1 - x, "peak": 1 - (2 * x - 1).abs()}[shape]
    # q = 1 and the keys of block m multiples of 1/8 up to 5.5: logits of 0 to 44, that is 63 powers of two, and (all but)
    # exact, since a logit of 44 that rounds the other way moves its exponential by a quarter
    q = torch.ones(1, 2, N, D)
    k = ((5.5 * 8 * size).round() / 8).repeat_interleave(B).view(1, 1, N, 1).expand(1, 2, N, D).contiguous()
    v = torch.randn(1, 2, N, D, generator=g)
    q, k, v = (t.to(dtype) for t in (q, k, v))
    out = ma.MonarchAttention(B, T, "post", impl="b200-tile")(q.cuda(), k.cuda(), v.cuda()).cpu().float()
    ref = monarch_attention_oracle(q, k, v, None, T, B, False).float()
    # (the tolerance of the other comparisons of these kernels with the oracle: roundings of the storage type)
    assert (out - ref).norm() <= (1e-2 if dtype == torch.bfloat16 else 2e-3) * ref.norm()
