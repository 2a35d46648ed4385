"""Chunks of the host entry point over several batch elements: how they are cut, and that their results are those of one call."""
import ctypes as C

import pytest
import torch


def test_small_heads_are_grouped():
    from monarch_attention_b200.host_pipeline import CHUNK_BYTES, group_chunks
    assert group_chunks(1, 16, CHUNK_BYTES, 8) == (8, 1, 1)           # a chunk is large enough as it is
    assert group_chunks(3, 20, CHUNK_BYTES // 16, 8) == (16, 1, 8)    # more heads, not all of an element
    assert group_chunks(3, 16, CHUNK_BYTES // 16, 8) == (16, 1, 8)
    assert group_chunks(9, 4, CHUNK_BYTES // 16, 2) == (4, 4, 8)      # whole elements
    assert group_chunks(2, 4, 64, 2) == (4, 2, CHUNK_BYTES // 128)    # no more than there are


def test_grouped_scratch_holds_whole_elements():
    from monarch_attention_b200 import _cabi
    from monarch_attention_b200.monarch_attention import make_problem
    lib = _cabi.load()
    t = torch.zeros(5, 3, 40, 16)
    p = make_problem(t, t, t, t, None, 1, 8, False)
    size = lambda heads, elements: lib.ma_b200_host_scratch_bytes_grouped(C.byref(p), heads, elements)  # noqa: E731
    assert size(3, 1) == lib.ma_b200_host_scratch_bytes(C.byref(p), 3) < size(3, 2) < size(3, 5) == size(9, 7)
    assert size(2, 5) == size(2, 1)                                   # elements only with all their heads
    assert size(3, 0) == 0 and b"elements_per_chunk" in lib.ma_b200_host_last_error()
    assert lib.ma_b200_forward_host_grouped(C.byref(p), 3, 2, 0, 0, None, 0, None) != 0


@pytest.mark.gpu
@pytest.mark.parametrize("chunk", [1, 3 * 4 * 50 * 64 * 2, 4 << 20])  # of one head, of three elements (the last ragged), all at once
@pytest.mark.parametrize("layout", ["heads", "tokens", "gaps"])
@pytest.mark.parametrize("masked", [False, True])
def test_grouped_chunks_return_the_bits_of_one_device_call(monkeypatch, chunk, layout, masked):
    import monarch_attention_b200 as ma
    from monarch_attention_b200 import host_pipeline
    E, H, N, D, B, T = 8, 4, 50, 64, 8, 2
    monkeypatch.setattr(host_pipeline, "CHUNK_BYTES", chunk)
    g = torch.Generator().manual_seed(chunk % 97)

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
        ma.monarch_attention_b200_host(q, k, v, m, T, B, True, out=out, heads_per_chunk=1, streamed=streamed)
        assert torch.equal(out.contiguous().view(torch.int16), want.contiguous().view(torch.int16))
