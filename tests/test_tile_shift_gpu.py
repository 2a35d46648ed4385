"""Column tiles with missing columns take the shift of their exponentials from the first 16 columns and raise it where later
ones are far larger (masked_column_exps in csrc/ma_tile_common.cuh): rows whose logits grow by some 60 powers of two from the
first block to the last, or fall, or do both, and rows with logits beyond the range of the storage type, against the CPU oracle."""
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


# Logits of a column that are below the range of the storage type in a row's first columns, and 0 in the others.
# The first M1 blocks have q = 0 and k = -300, the others q = 300 and k = 0: every logit of a right-factor stage is 0, and in a
# column stage the rows from M1 on have 300 * -37.5 * 64 = -720000 for the first M1 columns, -inf in half precision.
@pytest.mark.parametrize("pre", [False, True])
@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("N,B,M1,T", [(7683, 64, 16, 1), (7683, 64, 16, 2), (40 * 60 - 3, 40, 32, 1), (40 * 60 - 3, 40, 20, 2), (7683, 64, 1, 2),
                                      (200 * 150 - 9, 200, 16, 1), (200 * 150 - 9, 200, 140, 2), (100 * 33, 100, 16, 2)])
def test_rows_whose_first_logits_overflow_stay_finite(N, B, M1, T, masked, pre):
    import monarch_attention_b200 as ma
    from oracle.monarch_oracle import monarch_attention_oracle
    D, M = 64, -(-N // B)
    off = M * B - N if pre else 0
    late = ((torch.arange(N) + off) // B >= M1).view(1, 1, N, 1)
    g = torch.Generator().manual_seed(N + M1)
    q = torch.where(late, 300.0, 0.0).expand(1, 2, N, D).half()
    k = torch.where(late, 0.0, -300.0).expand(1, 2, N, D).half()
    v = torch.randn(1, 2, N, D, generator=g).half()
    mask = torch.rand(1, N, generator=g) > 0.2 if masked else None
    out = ma.MonarchAttention(B, T, "pre" if pre else "post", impl="b200-tile")(q.cuda(), k.cuda(), v.cuda(), None if mask is None else mask.cuda())
    ref = monarch_attention_oracle(q, k, v, mask, T, B, pre).float()
    assert ref.isfinite().all()
    assert (out.cpu().float() - ref).norm() <= 2e-3 * ref.norm()


@pytest.mark.parametrize("far", [0, 20])  # the logits that overflow begin in the first columns of their row, or behind them
@pytest.mark.parametrize("value", [60000.0, float("nan")])
@pytest.mark.parametrize("N,B", [(7683, 64), (40 * 60 - 3, 40), (200 * 150 - 9, 200)])
def test_a_row_that_overflows_leaves_the_others_alone(N, B, value, far):
    """One query whose logits in the output stage are +inf, or NaN.  Its own block has k = 0, so a value of 60000 changes nothing
    but that row: all other tokens keep their bits.  A query that is NaN reaches its own column, and the other one of its tile where
    two columns share one (their sums take 0 * NaN from each other)."""
    import monarch_attention_b200 as ma
    D, M = 64, -(-N // B)
    l, j = M - 2, 5
    g = torch.Generator().manual_seed(N)
    q, k, v = (torch.randn(1, 2, N, D, generator=g) for _ in range(3))
    k[:, :, :far * B] = 0
    k[:, :, far * B:] = k[:, :, far * B:].abs()
    k[:, :, l * B:(l + 1) * B] = 0
    module = ma.MonarchAttention(B, 1, "post", impl="b200-tile")
    outs = []
    for x in (0.0, value):
        q[:, :, l * B + j] = x
        outs.append(module(*(t.half().cuda() for t in (q, k, v))).cpu())
    gone = torch.zeros(N, dtype=torch.bool)
    if value == value:
        gone[l * B + j] = True
    else:
        gone[j::B] = True
    apart = gone if value == value or M > 64 else gone | gone.roll(-1)  # (columns 4 and 5)
    assert outs[0].isfinite().all()
    assert outs[1][:, :, gone].isnan().all()
    assert torch.equal(outs[1][:, :, ~apart].view(torch.int16), outs[0][:, :, ~apart].view(torch.int16))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("N,B,T,masked,pre", [(64 * 61 - 7, 64, 2, False, False), (7683, 64, 1, True, False), (40 * 60 - 3, 40, 3, True, True),
                                              (200 * 70 - 9, 200, 2, True, False), (100 * 33 - 50, 100, 2, False, True)])
def test_missing_columns_leave_the_precision_of_the_reference(N, B, T, masked, pre, dtype):
    """The shift that is not the maximum costs no precision: against float64 the kernels are where the reference's own 16-bit result
    is.  Both round at the same points and keep sums and exponentials in fp32; what differs (order of the sums, last bits of
    exponentials and quotients, some 2^-21) moves one in 2^10 or fewer of the values that are rounded to 11 or 8 bits to the other
    neighbour, and a few of these are carried through the next softmax: the quotient of the two errors is 0.996 to 1.014 over the
    cases here, and a shift that lost one bit of a row would be far above 1.05.  Activation-scale inputs."""
    import monarch_attention_b200 as ma
    from oracle.monarch_oracle import monarch_attention_dense_f64, monarch_attention_oracle
    g = torch.Generator().manual_seed(N + T)
    q, k = ((1.5 * torch.randn(1, 2, N, 64, generator=g) + 0.3 * torch.randn(1, 2, 1, 64, generator=g)).to(dtype) for _ in range(2))
    v = torch.randn(1, 2, N, 64, generator=g).to(dtype)
    mask = torch.rand(1, N, generator=g) > 0.2 if masked else None
    exact = torch.from_numpy(monarch_attention_dense_f64(*(t.double().numpy() for t in (q, k, v)), None if mask is None else mask.numpy(), T, B, pre))
    ref = monarch_attention_oracle(q, k, v, mask, T, B, pre).double()
    mod = ma.MonarchAttention(B, T, "pre" if pre else "post", impl="b200-tile")
    out = mod(q.cuda(), k.cuda(), v.cuda(), None if mask is None else mask.cuda()).cpu().double()
    err_out, err_ref = (out - exact).norm() / exact.norm(), (ref - exact).norm() / exact.norm()
    assert err_out <= 1.05 * err_ref, (err_out.item(), err_ref.item())
