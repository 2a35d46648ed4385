"""What bounds the device scratch of the host entry point: heads_per_chunk, and chunk_bytes where heads are small."""
import ctypes as C

import pytest
import torch


def test_no_grouping_with_chunk_bytes_of_zero():
    from monarch_attention_b200.host_pipeline import group_chunks
    assert group_chunks(9, 4, 64, 2, 0) == (2, 1, 1) and group_chunks(9, 4, 64, 7, 0) == (4, 1, 1)
    assert group_chunks(9, 4, 64, 2, 64 * 12) == (4, 3, 6)


@pytest.mark.parametrize("shape,T,B,heads,error", [((1, 2, 8, 0), 1, 4, 8, ValueError), ((2, 3, 8, 16), 0, 4, 8, ValueError),
                                                   ((2, 3, 8, 16), 1, 0, 8, ValueError), ((2, 3, 8, 16), 1, 4, 0, ValueError),
                                                   ((2, 3, 8, 16), 1, 4, 8.0, C.ArgumentError)])
def test_refused_before_a_gpu_is_touched(shape, T, B, heads, error):
    from monarch_attention_b200 import monarch_attention_b200_host
    t = torch.zeros(shape)
    with pytest.raises(error):
        monarch_attention_b200_host(t, t, t, None, T, B, False, out=torch.zeros(shape), device="cuda:0", heads_per_chunk=heads)


@pytest.mark.gpu
@pytest.mark.parametrize("asked,per_chunk,elements", [({"heads_per_chunk": 1}, 1, 1), ({"heads_per_chunk": 5}, 5, 1), ({}, 12, 6),
                                                      ({"chunk_bytes": 0}, 8, 1), ({"heads_per_chunk": 2, "chunk_bytes": 30 * 1000}, 5, 1)])
def test_scratch_is_what_was_asked_for(monkeypatch, asked, per_chunk, elements):
    import monarch_attention_b200 as ma
    from monarch_attention_b200 import _cabi, host_pipeline
    from monarch_attention_b200.monarch_attention import make_problem
    monkeypatch.setattr(host_pipeline, "_scratch", {})
    g = torch.Generator().manual_seed(3)
    q, k, v = (torch.randn(6, 12, 50, 64, generator=g).to(torch.bfloat16).pin_memory() for _ in range(3))
    dev = torch.device("cuda:0")
    out = ma.monarch_attention_b200_host(q, k, v, None, 2, 8, False, **asked)
    assert torch.equal(out, ma.MonarchAttention(8, 2, "post")(q.to(dev), k.to(dev), v.to(dev)).cpu())
    need = _cabi.load().ma_b200_host_scratch_bytes_grouped(C.byref(make_problem(q, k, v, out, None, 2, 8, False)), per_chunk, elements)
    assert host_pipeline._scratch[0].numel() == need


@pytest.mark.gpu
@pytest.mark.parametrize("chunk", [1, 3 * 4 * 50 * 64 * 2, 4 << 20])  # of one head, of three elements (the last ragged), all at once
@pytest.mark.parametrize("layout", ["heads", "tokens", "gaps"])
@pytest.mark.parametrize("masked", [False, True])
def test_chunks_over_elements_return_the_bits_of_one_device_call(chunk, layout, masked):
    import monarch_attention_b200 as ma
    E, H, N, D, B, T = 8, 4, 50, 64, 8, 2
    g = torch.Generator().manual_seed(chunk % 89)

    def host():
        t = torch.randn(E, H, N, D, generator=g).to(torch.bfloat16)
        if layout == "tokens":
            return t.permute(0, 2, 1, 3).contiguous().pin_memory().permute(0, 2, 1, 3)
        if layout == "gaps":  # elements that do not follow one another
            whole = torch.zeros(E, H + 1, N, D, dtype=t.dtype).pin_memory()
            whole[:, :H] = t
            return whole[:, :H]
        return t.pin_memory()

    q, k, v = host(), host(), host()
    m = torch.rand(E, N, generator=g) > 0.3 if masked else None
    dev = torch.device("cuda:0")
    want = ma.MonarchAttention(B, T, "pre")(q.to(dev), k.to(dev), v.to(dev), None if m is None else m.to(dev)).cpu()
    out = host()
    for streamed in (False, True, True):
        out.zero_()
        ma.monarch_attention_b200_host(q, k, v, m, T, B, True, out=out, heads_per_chunk=1, chunk_bytes=chunk, streamed=streamed)
        assert torch.equal(out.contiguous().view(torch.int16), want.contiguous().view(torch.int16))


@pytest.mark.gpu
def test_streamed_calls_with_slots_of_one_size_and_other_tensors_in_them():
    """Widths of 32 and 96 exchanged between q, k and v: the slots have one size, the results lie elsewhere in them."""
    import monarch_attention_b200 as ma
    dev = torch.device("cuda:0")
    g = torch.Generator().manual_seed(11)
    calls = []
    for i in range(10):
        D, Dv = (32, 96) if i % 2 else (96, 32)
        q, k, v = (torch.randn(1, 8, 600, w, generator=g).to(torch.bfloat16).pin_memory() for w in (D, D, Dv))
        calls.append((q, k, v, torch.empty_like(v).pin_memory()))
    for q, k, v, out in calls:
        ma.monarch_attention_b200_host(q, k, v, None, 1, 25, False, out=out, wait=False, streamed=True, heads_per_chunk=2)
    torch.cuda.synchronize()
    for q, k, v, out in calls:
        assert torch.equal(out, ma.monarch_attention_b200(q.to(dev), k.to(dev), v.to(dev), None, 1, 25, False).cpu())


@pytest.mark.gpu
def test_more_heads_than_a_grid_takes():
    """In chunks each family runs any number of heads: here one that is asked for by name, of one token each."""
    import monarch_attention_b200 as ma
    from monarch_attention_b200 import _cabi
    E, H = 9000, 8
    g = torch.Generator().manual_seed(1)
    q, k, v = (torch.randn(E, H, 1, 8, generator=g).to(torch.bfloat16).pin_memory() for _ in range(3))
    out = ma.monarch_attention_b200_host(q, k, v, None, 1, 1, False, kernel=_cabi.KERNEL_WARP_MMA)
    assert torch.equal(out, v)  # (one token attends to itself)
