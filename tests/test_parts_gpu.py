"""A call cut into parts returns the bits of the undivided call: chunks of the host entry point, and shards that take the
kernel family of the whole call.  The shapes are ones where a part alone would take another family than the whole."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [  # E, H, N, D, B, T, heads per chunk, mask
    (1, 16, 16384, 64, 128, 2, 8, False),   # tile kernels; eight heads or fewer: fused kernel
    (1, 48, 4096, 64, 64, 1, 16, False),    # tile kernels; fewer heads: fused kernel
    (4, 50, 300, 80, 10, 2, 25, True),      # warp-level kernels; fewer heads: head-resident kernel
    (5, 16, 40 * 38, 64, 40, 1, 16, False)]  # tile kernels; fewer heads: warp-level kernels


def _inputs(E, H, N, D, mask):
    g = torch.Generator().manual_seed(N)
    q, k, v = (torch.randn(E, H, N, D, generator=g).to(torch.bfloat16) for _ in range(3))
    return q, k, v, (torch.rand(E, N, generator=g) > 0.2 if mask else None)


def _family(t, mask, T, B):
    from monarch_attention_b200 import _cabi
    from monarch_attention_b200.monarch_attention import make_problem
    L = _cabi.WorkspaceLayout()
    prob = make_problem(t, t, t, t, mask, T, B, False)
    _cabi.raise_for_status(_cabi.load().ma_b200_workspace_layout_of(C.byref(prob), C.byref(L)))
    return L.kernel


@pytest.mark.parametrize("E,H,N,D,B,T,hc,mask", SHAPES)
def test_host_chunks_return_the_bits_of_one_device_call(E, H, N, D, B, T, hc, mask):
    import monarch_attention_b200 as ma
    dev = torch.device("cuda:0")
    q, k, v, m = _inputs(E, H, N, D, mask)
    want = ma.MonarchAttention(B, T, "post")(q.to(dev), k.to(dev), v.to(dev), None if m is None else m.to(dev)).cpu()
    got = ma.monarch_attention_b200_host(q.pin_memory(), k.pin_memory(), v.pin_memory(), m, T, B, False, heads_per_chunk=hc)
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))


@pytest.mark.parametrize("E,H,N,D,B,T,hc,mask", SHAPES)
def test_shards_return_the_bits_of_the_unsharded_call(E, H, N, D, B, T, hc, mask):
    import monarch_attention_b200 as ma
    from monarch_attention_b200.sharding import kernel_of_part
    dev = torch.device("cuda:0")
    q, k, v, m = _inputs(E, H, N, D, mask)
    q, k, v = (t.to(dev) for t in (q, k, v))
    m = None if m is None else m.to(dev)
    want = ma.MonarchAttention(B, T, "post")(q, k, v, m)
    part = [t[:1, :3] for t in (q, k, v)]
    mp = None if m is None else m[:1]
    assert _family(part[0], mp, T, B) != _family(q, m, T, B)  # (or the shape shows nothing)
    kernel = kernel_of_part(*part, mp, T, B, False, heads=E * H)
    got = ma.monarch_attention_b200(*part, mp, T, B, False, kernel=kernel)
    assert torch.equal(got.view(torch.int16), want[:1, :3].view(torch.int16))


@pytest.mark.parametrize("N,B,H,T,name", [(4096, 64, 25, 2, "tcgen05-fused"), (4096, 64, 26, 2, "tile"), (16384, 128, 6, 3, "tcgen05-fused"),
                                          (16384, 128, 7, 3, "tile"), (4096, 64, 9, 1, "tcgen05-fused"), (4096, 64, 12, 1, "tile")])
def test_both_sides_of_the_line_between_fused_and_tile_kernels(N, B, H, T, name):
    """5.5 tiles of 128 rows per SM and stage (148 SMs: 814), two with one iteration (296); either side matches the generic kernels."""
    import monarch_attention_b200 as ma
    from monarch_attention_b200 import _cabi
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the head counts are those around the line of 148 SMs")
    dev = torch.device("cuda:0")
    q, k, v, _ = _inputs(1, H, N, 64, False)
    q, k, v = (t.to(dev) for t in (q, k, v))
    assert _cabi.KERNEL_NAMES[_family(q, None, T, B)] == name
    out = ma.MonarchAttention(B, T, "post")(q, k, v).float()
    ref = ma.MonarchAttention(B, T, "post", impl="b200-generic")(q, k, v).float()
    # (16-bit results of the same rounding points summed in different orders: the parity bound of the library)
    assert ((out - ref).norm() / ref.norm()).item() <= 1e-2
