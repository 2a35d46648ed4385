"""The three forms of the head-resident kernel (one CTA a head, parts of its columns, a cluster) give a head the same bits: beside both lines
to the clusters, with either side the longer one, at widths with tiles of their own and without."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [  # heads (148 SMs), B, M, D, T
    (74, 17, 17, 64, 1), (75, 17, 17, 64, 1), (75, 17, 17, 64, 3), (90, 24, 24, 72, 2), (91, 24, 24, 72, 2), (80, 18, 23, 32, 1), (85, 24, 17, 80, 2), (80, 24, 17, 40, 3),
    (75, 20, 5, 40, 2), (75, 25, 20, 64, 1), (1, 32, 32, 64, 1), (32, 32, 32, 80, 1), (33, 25, 25, 72, 1), (12, 17, 31, 40, 1), (32, 3, 32, 64, 1), (7, 16, 25, 24, 1),
    (7, 16, 25, 72, 1), (7, 30, 28, 64, 2)]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("H,B,M,D,T", SHAPES)
def test_forms_give_the_same_bits(H, B, M, D, T, masked, dtype):
    import monarch_attention_b200 as ma
    g = torch.Generator(device="cuda").manual_seed(H * B + D)
    many, N = 300, B * M - (M > 3)  # one CTA a head
    q, k, v = (torch.randn(1, N, many, D, generator=g, device="cuda").to(dtype).permute(0, 2, 1, 3) for _ in range(3))
    m = (torch.rand(1, N, generator=g, device="cuda") > 0.3) if masked else None
    mod = ma.MonarchAttention(B, T, "pre", impl="b200-head-resident")
    want = mod(q, k, v, m)
    some = [t[:, 50:50 + H] for t in (q, k, v)]
    for _ in range(2):
        assert torch.equal(mod(*some, m), want[:, 50:50 + H])


@pytest.mark.parametrize("D", range(8, 81, 8))
def test_every_shape_has_a_kernel(D):
    """Sides and numbers of heads around all lines of the choice; with every row of v equal to c, every row of the result is c."""
    import monarch_attention_b200 as ma
    g = torch.Generator(device="cuda").manual_seed(D)
    q, k = (torch.randn(1, 160, 32 * 32, D, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    c = torch.linspace(-2, 2, D, device="cuda").to(torch.bfloat16)
    v = c.expand(1, 160, 32 * 32, D).contiguous()
    for B in (1, 16, 17, 24, 25, 32):
        for M in (1, 16, 17, 24, 25, 32):
            for H in (1, 33, 40, 75, 91, 148, 160):
                for T in (1, 2):
                    out = ma.MonarchAttention(B, T, "post", impl="b200-head-resident")(*(t[:, :H, :B * M] for t in (q, k, v)))
                    # (factors and y are rounded to 8 bits of mantissa: up to 2 ulp of 2 in the sum)
                    assert (out.float() - c.float()).abs().max().item() < 3e-2, (B, M, H, T)


@pytest.mark.parametrize("H,B,M,D,T", [(80, 17, 19, 64, 2), (12, 32, 32, 64, 1)])
def test_clusters_in_a_captured_graph(H, B, M, D, T):
    import monarch_attention_b200 as ma
    g = torch.Generator(device="cuda").manual_seed(5)
    q, k, v, q2 = (torch.randn(1, H, B * M, D, generator=g, device="cuda").to(torch.bfloat16) for _ in range(4))
    mod = ma.MonarchAttention(B, T, "post")
    want, want2 = mod(mod(q, k, v), k, v), mod(mod(q2, k, v), k, v)
    x = q.clone()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = mod(mod(x, k, v), k, v)
    for a, b in ((q, want), (q2, want2), (q, want)):
        x.copy_(a)
        graph.replay()
        assert torch.equal(out, b)
