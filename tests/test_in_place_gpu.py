"""A result that takes the place of the queries, keys or values: every family reads what it needs of a head before it writes there."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [  # E, H, N, D, B, T
    (1, 1, 32 * 32, 64, 32, 1), (1, 12, 197, 64, 15, 1), (2, 24, 31 * 30 - 4, 72, 31, 2), (1, 80, 17 * 20, 64, 17, 2), (1, 90, 16 * 22, 40, 16, 1),
    (4, 40, 20 * 9, 32, 20, 3), (1, 4, 40 * 60, 80, 40, 2), (1, 2, 4096, 64, 64, 2), (4, 12, 3000, 64, 60, 1), (1, 2, 200 * 150, 64, 200, 1)]


@pytest.mark.parametrize("where", [0, 1, 2])
@pytest.mark.parametrize("tokens", [False, True])
@pytest.mark.parametrize("E,H,N,D,B,T", SHAPES)
def test_result_in_the_place_of_an_input(E, H, N, D, B, T, tokens, where):
    import monarch_attention_b200 as ma
    g = torch.Generator(device="cuda").manual_seed(N)
    shape = (E, N, H, D) if tokens else (E, H, N, D)
    x = [torch.randn(shape, generator=g, device="cuda").to(torch.bfloat16) for _ in range(3)]
    x = [t.permute(0, 2, 1, 3) if tokens else t for t in x]
    want = ma.monarch_attention_b200(*x, None, T, B, False)
    for _ in range(3):
        y = [t.clone() for t in x]
        got = ma.monarch_attention_b200(*y, None, T, B, False, out=y[where])
        assert got.data_ptr() == y[where].data_ptr() and torch.equal(got, want)
