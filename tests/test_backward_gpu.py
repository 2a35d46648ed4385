"""Backward kernels at the edges of their tiles, against autograd through the same computation in float64."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [  # E, H, N, D, B, T, pad, mask, layout
    (1, 1, 1, 16, 1, 1, "post", "none", "heads"), (2, 3, 15 * 15, 64, 15, 1, "pre", "none", "tokens"),
    (1, 2, 250, 72, 16, 2, "pre", "rand", "heads"), (2, 2, 33 * 17 - 9, 32, 17, 3, "post", "block", "tokens"),
    (1, 2, 1024, 64, 32, 3, "post", "tail", "tokens"), (1, 1, 64 * 64, 64, 64, 2, "post", "none", "heads"),
    (2, 1, 48 * 64 - 1, 80, 64, 2, "pre", "rand", "heads"), (1, 1, 65 * 30, 40, 65, 1, "post", "none", "heads"),
    (1, 2, 128 * 128, 64, 128, 2, "post", "none", "heads"), (1, 1, 16 * 128 - 3, 80, 16, 2, "pre", "none", "heads")]


def _exact(q, k, v, mask, T, B, pre):
    """The computation without any rounding, differentiable (the library's own tensor-operation restatement casts
    the logits to fp32)."""
    E, H, N, D = q.shape
    M = -(-N // B)
    gap = M * B - N
    s = 1 / math.sqrt(D)
    pad = (lambda x: torch.nn.functional.pad(x, (0, 0, gap, 0) if pre else (0, 0, 0, gap)).reshape(E, H, M, B, -1))
    qb, kb, vb = pad(q), pad(k), pad(v)
    ok = torch.ones(E, N, dtype=torch.bool, device=q.device) if mask is None else mask
    ok = torch.nn.functional.pad(ok, (gap, 0) if pre else (0, gap)).reshape(E, 1, M, B)
    ar, cr, qc = qb, torch.ones(E, H, M, B, dtype=q.dtype, device=q.device), qb.transpose(-2, -3)
    for t in range(T):
        x = s * (ar @ kb.mT) / (cr[..., None] + 1e-12)
        x = x.masked_fill(~ok[..., None, :], -math.inf)
        e = torch.exp(x - x.amax(-1, keepdim=True).clamp(min=1e-12))
        r = (e / (e.sum(-1, keepdim=True) + 1e-12)).clamp(min=torch.finfo(torch.float32).tiny)
        cl = torch.special.xlogy(r, r).sum(-1).mT
        al = s * (r @ kb).transpose(-2, -3)
        if t < T - 1:
            lw = ok.mT.unsqueeze(-2) * torch.softmax(al @ qc.mT - cl[..., None], dim=-2)
            cr, ar = lw.sum(-1).mT, (lw @ qc).transpose(-2, -3)
    y = (r @ vb).transpose(-2, -3)
    z = torch.softmax(qc @ al.mT - cl[..., None, :], dim=-1) @ y
    z = z.transpose(-2, -3).reshape(E, H, M * B, -1)
    return z[..., gap:, :] if pre else z[..., :N, :]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("E,H,N,D,B,T,pad,mask,layout", SHAPES)
def test_backward_kernels_match_float64_gradients(E, H, N, D, B, T, pad, mask, layout, dtype):
    import monarch_attention_b200 as ma
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(N + D)

    def draw():
        shape = (E, H, N, D) if layout == "heads" else (E, N, H, D)
        t = torch.randn(shape, generator=g, device=dev).to(dtype)
        return t if layout == "heads" else t.permute(0, 2, 1, 3)

    q, k, v, w = (draw() for _ in range(4))
    m = None
    if mask != "none":
        m = torch.rand(E, N, generator=g, device=dev) > (0.3 if mask == "rand" else 0.0)
        if mask == "block":
            m[:, B:3 * B] = False
        if mask == "tail":
            m[0, N // 3:] = False
        m[:, 0] = True
    exact = [t.double().requires_grad_(True) for t in (q, k, v)]
    z = _exact(*exact, m, T, B, pad == "pre")
    want = torch.autograd.grad(z, exact, w.double())
    for t in (q, k, v):
        t.requires_grad_(True)
    out = ma.MonarchAttention(B, T, pad)(q, k, v, m)
    got = torch.autograd.grad(out, (q, k, v), w)
    tol = {torch.float32: 1e-5, torch.bfloat16: 1.5e-2, torch.float16: 2e-3}[dtype]
    for name, a, b in zip(("out", "dq", "dk", "dv"), (out, *got), (z, *want)):
        assert a.dtype == dtype and torch.isfinite(a.float()).all()
        err = ((a.double() - b).norm() / b.norm().clamp_min(1e-9)).item()
        assert err <= tol, (name, err)
    again = torch.autograd.grad(ma.MonarchAttention(B, T, pad)(q, k, v, m), (q, k, v), w)
    assert all(torch.equal(a, b) for a, b in zip(got, again))
