"""Host-side mirror of the reference's attention module for the B200 library.

Same constructor arguments, block size / iteration count meaning and the same
``forward(query, key, value[, attention_mask])`` shapes as the reference module
(reference: ma/monarch_attention.py:37-66), so the experiment models can construct
``MonarchAttention(config.block_size, config.num_steps, config.pad_type)`` and call
it unchanged (call sites: experiments/vit/model.py:97, experiments/roberta/model.py:104-106,
experiments/dit/attention_processor.py:143).

All arithmetic happens in the CUDA library behind the C ABI; PyTorch supplies device
memory and the current stream.  Inputs must live on a CUDA device: there is no CPU
path here.
"""
from __future__ import annotations

from collections.abc import Callable
from enum import StrEnum

import torch
import torch.nn as nn

from . import _cabi

Tensor = torch.Tensor
MonarchAttentionFn = Callable[[Tensor, Tensor, Tensor, "Tensor | None", int, int, bool], Tensor]

_DTYPE_CODE = {torch.float32: _cabi.F32, torch.bfloat16: _cabi.BF16, torch.float16: _cabi.F16}


class PadType(StrEnum):
    """Where the token axis is zero-padded to a multiple of the block size
    (reference: ma/monarch_attention.py:32-34)."""

    pre = "pre"
    post = "post"


def _tensor4(t: Tensor) -> _cabi.Tensor4:
    return _cabi.Tensor4(t.data_ptr(), t.stride(0), t.stride(1), t.stride(2))


def make_problem(q: Tensor, k: Tensor, v: Tensor, out: Tensor, mask: Tensor | None, T: int, B: int, pre_pad: bool,
                 kernel: int = _cabi.KERNEL_AUTO) -> _cabi.Problem:
    E, H, N, D = q.shape
    p = _cabi.Problem()
    p.abi_version = _cabi.ABI_VERSION
    p.E, p.H, p.N, p.D, p.Dv = E, H, N, D, v.shape[-1]
    p.block_size, p.num_steps, p.pre_pad = int(B), int(T), int(bool(pre_pad))
    p.qk_dtype, p.v_dtype = _DTYPE_CODE[q.dtype], _DTYPE_CODE[v.dtype]
    p.kernel = kernel
    p.q, p.k, p.v, p.out = _tensor4(q), _tensor4(k), _tensor4(v), _tensor4(out)
    if mask is not None:
        p.mask, p.mask_stride_e = mask.data_ptr(), mask.stride(0)
    else:
        p.mask, p.mask_stride_e = None, 0
    return p


def _check_device_free_inputs(q: Tensor, k: Tensor, v: Tensor, attn_mask: Tensor | None):
    """Shape and dtype rules of the host entry point (those of the device entry point are in the native binding)."""
    if q.dim() != 4 or k.dim() != 4 or v.dim() != 4:
        raise ValueError("query, key and value must have shape (batch, heads, tokens, width)")
    if k.shape != q.shape:
        raise ValueError(f"key shape {tuple(k.shape)} differs from query shape {tuple(q.shape)}")
    if v.shape[:3] != q.shape[:3]:
        raise ValueError(f"value shape {tuple(v.shape)} does not match query shape {tuple(q.shape)}")
    if q.dtype not in _DTYPE_CODE or v.dtype not in _DTYPE_CODE:
        raise ValueError(f"unsupported dtype {q.dtype} / {v.dtype}")
    if k.dtype != q.dtype:
        raise ValueError("query and key must have the same dtype")
    if attn_mask is not None and tuple(attn_mask.shape) != (q.shape[0], q.shape[2]):
        raise ValueError(f"attention_mask must have shape (batch, tokens) = {(q.shape[0], q.shape[2])}")


_native_forward = None


def _load_native():
    """The native entry point (monarch_attention_b200/_native.so); raises RuntimeError when it has not been built."""
    global _native_forward
    _cabi.load()
    try:
        from . import _native
    except ImportError as err:
        raise RuntimeError("monarch_attention_b200/_native.so is missing or does not match this PyTorch: build it with "
                           "`python -m monarch_attention_b200.build`. There is no fallback implementation.") from err
    _native_forward = _native.forward
    return _native_forward


def monarch_attention_b200(q: Tensor, k: Tensor, v: Tensor, attn_mask: Tensor | None, T: int, B: int, pre_pad: bool,
                           *, kernel: int = _cabi.KERNEL_AUTO, out: Tensor | None = None,
                           token_major_output: bool = False) -> Tensor:
    """Implementation function with the reference's registry signature
    (reference: ma/monarch_attention.py:11-19; computes what ma/ma_torch.py:65-108 computes).

    Returns a new (E, H, N, Dv) tensor of value's dtype on value's device.  With
    ``token_major_output`` the result is a (E, H, N, Dv) *view* of a (E, N, H, Dv) buffer, i.e. already
    in the layout the model adapters produce with ``permute(0, 2, 1, 3).contiguous()`` after the call
    (reference: experiments/vit/model.py:99-101), which then costs nothing.
    """
    fn = _native_forward or _load_native()
    result = fn(q, k, v, attn_mask, T, B, pre_pad, kernel, out, token_major_output)
    if result is None:   # a gradient is wanted that the backward kernels do not give
        from .backward import MonarchAttentionFunction
        result = MonarchAttentionFunction.apply(
            q, k, v, attn_mask, T, B, pre_pad,
            lambda a, b, c: fn(a, b, c, attn_mask, T, B, pre_pad, kernel, None, token_major_output))
    return result


def _generic(q, k, v, m, T, B, pre_pad):
    return monarch_attention_b200(q, k, v, m, T, B, pre_pad, kernel=_cabi.KERNEL_GENERIC)


def _tcgen05(q, k, v, m, T, B, pre_pad):
    return monarch_attention_b200(q, k, v, m, T, B, pre_pad, kernel=_cabi.KERNEL_TCGEN05)


_IMPLEMENTATIONS: dict[str, MonarchAttentionFn] = {}


def register_impl(name: str, fn: MonarchAttentionFn) -> None:
    """Same registry hook as the reference (reference: ma/monarch_attention.py:15-19)."""
    _IMPLEMENTATIONS[name] = fn


register_impl("b200", monarch_attention_b200)
register_impl("b200-generic", _generic)
register_impl("b200-tcgen05", _tcgen05)
register_impl("b200-tcgen05-staged",
              lambda q, k, v, m, T, B, pp: monarch_attention_b200(q, k, v, m, T, B, pp, kernel=_cabi.KERNEL_TCGEN05_STAGED))
register_impl("b200-warp-mma",
              lambda q, k, v, m, T, B, pp: monarch_attention_b200(q, k, v, m, T, B, pp, kernel=_cabi.KERNEL_WARP_MMA))
register_impl("b200-head-fused",
              lambda q, k, v, m, T, B, pp: monarch_attention_b200(q, k, v, m, T, B, pp, kernel=_cabi.KERNEL_HEAD_FUSED))
register_impl("b200-tf32x3",
              lambda q, k, v, m, T, B, pp: monarch_attention_b200(q, k, v, m, T, B, pp, kernel=_cabi.KERNEL_TF32X3))
register_impl("b200-head-resident",
              lambda q, k, v, m, T, B, pp: monarch_attention_b200(q, k, v, m, T, B, pp, kernel=_cabi.KERNEL_HEAD_RESIDENT))
register_impl("b200-tile",
              lambda q, k, v, m, T, B, pp: monarch_attention_b200(q, k, v, m, T, B, pp, kernel=_cabi.KERNEL_TILE))


class MonarchAttention(nn.Module):
    """Drop-in for the reference module (reference: ma/monarch_attention.py:37-66).

    ``impl`` selects the kernel family: "b200" (default: the library picks by shape, type and number of
    heads), "b200-tcgen05" (fused, one launch), "b200-tcgen05-staged" (same kernel, one launch per stage),
    "b200-tile" (tcgen05 tile kernels, one launch up to blocks of 128), "b200-head-resident" (small blocks: one
    CTA or a few per head, all stages), "b200-head-fused" (the same, one iteration only), "b200-warp-mma"
    (warp-level tensor-core kernels), "b200-tf32x3" (the same on fp32 tensors) or "b200-generic".  The reference's
    "torch" and "triton" implementations are not part of this library; asking for an
    unknown name raises ``ValueError`` exactly as the reference does.
    """

    def __init__(self, block_size, num_steps, pad_type, impl="b200"):
        super().__init__()
        self.block_size = block_size
        self.num_steps = num_steps
        self.pad_type = pad_type
        if impl not in _IMPLEMENTATIONS:
            available = ", ".join(sorted(_IMPLEMENTATIONS))
            raise ValueError(f"Unknown impl {impl!r}. Available: {available}")
        self._impl_fn = _IMPLEMENTATIONS[impl]
        # Set to True to get the result as a view of a (batch, tokens, heads, width) buffer (see
        # monarch_attention_b200); only the default implementation honours it.
        self.token_major_output = False

    def forward(self, query, key, value, attention_mask=None):
        if self.token_major_output and self._impl_fn is monarch_attention_b200:
            return monarch_attention_b200(query, key, value, attention_mask, self.num_steps, self.block_size,
                                          self.pad_type == PadType.pre, token_major_output=True)
        return self._impl_fn(query, key, value, attention_mask, self.num_steps, self.block_size,
                             self.pad_type == PadType.pre)

    def get_matrix(self, query, key, attention_mask=None):
        """Explicit (E, H, N, N) attention matrix: forward with V = identity
        (reference: ma/monarch_attention.py:61-66; fp32 identity, so an fp32 result)."""
        batch_size, num_heads, seq_len, _ = query.shape
        value = torch.eye(seq_len, device=query.device).expand(batch_size, num_heads, seq_len, seq_len)
        return self.forward(query, key, value, attention_mask)

    def extra_repr(self) -> str:
        return f"block_size={self.block_size}, num_steps={self.num_steps}, pad_type={str(self.pad_type)!r}"
