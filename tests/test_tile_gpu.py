"""tcgen05 tile kernels at the edges of their tiles (two units per tile with an odd last one, row and column remainders,
the row behind the last whole block, both padding sides, masks that empty blocks, narrow heads, several tiles per CTA),
against the CPU oracle."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [  # E, H, N, D, B, T, pad, mask
    (1, 1, 64 * 64, 64, 64, 1, "post", "none"), (1, 2, 64 * 64, 64, 64, 2, "post", "none"),
    (2, 2, 64 * 61 - 7, 64, 64, 2, "post", "tail"), (1, 3, 45 * 47 - 11, 64, 45, 3, "pre", "rand"),
    (1, 1, 33 * 64, 64, 33, 2, "post", "none"), (1, 2, 128 * 128, 64, 128, 2, "post", "none"),
    (1, 1, 65 * 128 - 64, 64, 65, 2, "pre", "none"), (2, 1, 97 * 100 - 3, 64, 97, 2, "post", "block"),
    (1, 1, 129 * 40, 64, 129, 2, "post", "none"), (1, 1, 40 * 129 - 39, 64, 40, 2, "pre", "rand"),
    (1, 1, 256 * 256, 64, 256, 2, "post", "none"), (1, 1, 200 * 170 - 100, 64, 200, 1, "pre", "rand"),
    (1, 2, 60 * 70 - 1, 40, 60, 2, "post", "none"), (1, 2, 70 * 60, 32, 70, 3, "pre", "tail"), (1, 1, 150 * 66 - 20, 8, 150, 2, "post", "none"),
    (1, 1, 36 * 2 - 1, 64, 36, 2, "post", "none"), (1, 1, 20 * 3, 16, 20, 2, "pre", "none"),
    (8, 12, 40 * 38 - 3, 64, 40, 2, "post", "tail"), (2, 6, 100 * 90 - 13, 64, 100, 2, "pre", "none")]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("E,H,N,D,B,T,pad,mask", SHAPES)
def test_tile_kernels_match_the_oracle(E, H, N, D, B, T, pad, mask, dtype):
    import monarch_attention_b200 as ma
    from oracle.monarch_oracle import monarch_attention_oracle
    g = torch.Generator().manual_seed(N * 3 + D)
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
    md = None if m is None else m.to(dev)
    args = [t.to(dev) for t in (q, k, v)]
    mod = ma.MonarchAttention(B, T, pad, impl="b200-tile")
    out = mod(*args, md)
    ref = monarch_attention_oracle(q, k, v, m, T, B, pad == "pre").float()
    err = ((out.cpu().float() - ref).norm() / ref.norm()).item()
    assert torch.isfinite(out.float()).all() and err <= (1e-2 if dtype == torch.bfloat16 else 2e-3), err
    strided = [t.permute(0, 2, 1, 3).contiguous().permute(0, 2, 1, 3) for t in args]
    assert torch.equal(mod(*strided, md), out)


@pytest.mark.parametrize("H,B,M,T", [(1, 64, 64, 6), (2, 64, 60, 5), (1, 128, 128, 4), (3, 40, 100, 5)])
def test_single_launch_stages_read_what_the_stage_before_wrote(H, B, M, T):
    """Few heads and many iterations: in the single launch every tile waits for the stage before, and its row vectors (cl, cr)
    are read by all lanes of a warp of which one did the waiting.  Two alternating inputs leave different vectors in the same
    workspace, so a value read too early shows as a difference between calls."""
    import monarch_attention_b200 as ma
    g = torch.Generator().manual_seed(B + T)
    dev = torch.device("cuda:0")
    mod = ma.MonarchAttention(B, T, "post", impl="b200-tile")
    inputs = [[torch.randn(1, H, B * M, 64, generator=g).to(torch.bfloat16).to(dev) for _ in range(3)] for _ in range(2)]
    want = [mod(*x) for x in inputs]
    assert all(torch.isfinite(w.float()).all() for w in want)
    for _ in range(10):
        for x, w in zip(inputs, want):
            assert torch.equal(mod(*x), w)


@pytest.mark.parametrize("E,H,N,B,T", [(1, 2, 4096, 64, 2), (2, 12, 4096, 64, 1), (1, 3, 128 * 100 - 5, 128, 3),
                                       (1, 2, 40 * 100, 40, 2), (1, 2, 200 * 40, 200, 2), (1, 1, 256 * 256, 256, 1),
                                       (1, 2, 40 * 200, 40, 2), (1, 2, 100 * 150, 100, 1)])
def test_expired_wait_ends_the_launch_and_is_reported(E, H, N, B, T):
    """Single launch: the first stage is left out, so the waits for it run out; one launch per stage (blocks above 128): an
    operand is never asked for.  Every CTA gives up by itself, the status words say so, the next call raises, and the one
    after is an ordinary call."""
    import monarch_attention_b200 as ma
    from monarch_attention_b200 import _cabi
    from monarch_attention_b200.monarch_attention import make_problem
    lib, dev = _cabi.load(), torch.device("cuda:0")
    g = torch.Generator().manual_seed(N)
    q, k, v = (torch.randn(E, H, N, 64, generator=g).to(torch.bfloat16).to(dev) for _ in range(3))
    mod = ma.MonarchAttention(B, T, "post", impl="b200-tile")
    good = mod(q, k, v)
    stream = torch.cuda.current_stream().cuda_stream
    prob = make_problem(q, k, v, torch.empty_like(v), None, T, B, False, _cabi.KERNEL_TILE)
    ws = torch.zeros(lib.ma_b200_workspace_bytes(C.byref(prob)), dtype=torch.uint8, device=dev)
    assert lib.ma_b200_poll_device_status(0) == _cabi.OK
    start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    start.record()
    _cabi.raise_for_status(lib.ma_b200_selftest_wait_expiry(C.byref(prob), ws.data_ptr(), ws.numel(), stream))
    end.record()
    torch.cuda.synchronize()
    # the waits that run out are of 4096 tries; what a CTA still waits for on its way out has been asked for and is there
    # (a wait for something else would be one of millions of tries)
    assert start.elapsed_time(end) < 500
    assert lib.ma_b200_device_status(ws.data_ptr(), stream) == _cabi.DEVICE_WAIT_EXPIRED
    with pytest.raises(RuntimeError, match="gave up"):
        mod(q, k, v)
    assert lib.ma_b200_poll_device_status(0) == _cabi.OK
    assert torch.equal(mod(q, k, v), good)


def test_full_size_tile_kernels():
    """The headline size (16 heads of 16384 tokens): constant rows of V come back (the matrix is row-stochastic), heads may
    change places without changing a bit, calls repeat, and two heads agree with the CPU oracle."""
    import monarch_attention_b200 as ma
    from oracle.monarch_oracle import monarch_attention_oracle
    g = torch.Generator().manual_seed(1234)
    dev = torch.device("cuda:0")
    q, k, v = (torch.randn(1, 16, 16384, 64, generator=g).to(torch.bfloat16).to(dev) for _ in range(3))
    mod = ma.MonarchAttention(128, 2, "post", impl="b200-tile")
    c = torch.linspace(-2, 2, 64, device=dev).to(torch.bfloat16)
    assert (mod(q, k, c.expand_as(v).contiguous()).float() - c.float()).abs().max().item() < 3e-2
    out = mod(q, k, v)
    for _ in range(3):
        assert torch.equal(mod(q, k, v), out)
    perm = torch.randperm(16, generator=g).to(dev)
    assert torch.equal(mod(q[:, perm], k[:, perm], v[:, perm]), out[:, perm])
    for h in (0, 11):
        ref = monarch_attention_oracle(*(t[:, h:h + 1].cpu() for t in (q, k, v)), None, 2, 128, False).float()
        assert ((out[:, h:h + 1].cpu().float() - ref).norm() / ref.norm()).item() <= 1e-2
