"""Forward pass on HOST tensors, with the PCIe copies overlapped with the kernels.

The reference module is handed device tensors by its callers (reference:
ma/monarch_attention.py:50-59); a caller whose q, k, v live in host memory pays
host-to-device and device-to-host copies around the call, and for the long-sequence
workloads those copies, not the kernels, are the time.  ``monarch_attention_b200_host``
binds the library's ``ma_b200_forward_host``, which cuts the (batch, head) pairs into chunks
of a few heads and pipelines H2D, kernels and D2H over three streams (see
``csrc/ma_host.cu``); this module only provides the device scratch and the pointers.
"""
from __future__ import annotations

import ctypes as C

import torch
from torch import Tensor

from . import _cabi
from .monarch_attention import _check_device_free_inputs, make_problem

_scratch: dict[int, Tensor] = {}

# Least bytes of one tensor in a chunk.  A chunk of a few heads whatever their size was bound by what it costs the host and the
# copy engines to start.  Measured (us, 8 heads a chunk / chunks of at least 1, 2, 4, 8 MB): 52 x 12 heads of 93 x 64 in fp32
# 2940 / 1284, 1105, 1092, 1084 (copying in alone 810); 5 x 12 of 769 x 64 650 / 591, 517, 466, 497; 16 x 16 of 512 x 64 1621 /
# 1426, 1274, 1176, 1170; 8 of 8192 x 64, whose chunks are larger anyway, 699 / 679, 684, 667, 684.
CHUNK_BYTES = 4 << 20
HEADS_PER_CHUNK = 8
# Most heads that the tensor-core kernels take in a launch (their grids' second dimension).
GRID_HEADS = 65535


def group_chunks(E: int, H: int, head_bytes: int, heads_per_chunk: int, chunk_bytes: int | None = None) -> tuple[int, int, int]:
    """(heads per chunk, batch elements per chunk, least heads of a chunk at the end): a chunk of less than ``chunk_bytes``
    (default CHUNK_BYTES) of one tensor grows to that, over whole batch elements where it has all their heads, and is not cut to
    fewer than half of it at the end.  With 0 it is ``heads_per_chunk`` heads of one batch element."""
    room = -(-(CHUNK_BYTES if chunk_bytes is None else chunk_bytes) // head_bytes)
    heads = min(H, max(heads_per_chunk, min(room, GRID_HEADS)))
    elements = min(E, max(1, min(room, GRID_HEADS) // H)) if heads == H else 1
    return heads, elements, max(1, room // 2)


def plan_chunks(E: int, H: int, heads_per_chunk: int, elements_per_chunk: int = 1, least_heads: int = 1) -> list[tuple[int, int, int]]:
    """(batch index, first head, number of heads, over whole elements where there are more than that element has left) of every
    chunk, in the order the library runs them; the arguments are what ``group_chunks`` returns."""
    if E < 0 or H < 0:
        raise ValueError("E and H must be non-negative")
    if min(heads_per_chunk, elements_per_chunk, least_heads) < 1:
        raise ValueError("heads_per_chunk, elements_per_chunk and least_heads must be at least 1")
    plan = _cabi.load().ma_b200_host_chunk_plan
    n = plan(E, H, heads_per_chunk, elements_per_chunk, least_heads, None, 0)
    flat = (C.c_int32 * (3 * n))()
    plan(E, H, heads_per_chunk, elements_per_chunk, least_heads, flat, n)
    return [tuple(flat[3 * i:3 * i + 3]) for i in range(n)]


def monarch_attention_b200_host(q: Tensor, k: Tensor, v: Tensor, attn_mask: Tensor | None, T: int, B: int,
                                pre_pad: bool, *, out: Tensor | None = None, device=None,
                                heads_per_chunk: int = HEADS_PER_CHUNK, wait: bool = True, streamed: bool = False,
                                kernel: int = _cabi.KERNEL_AUTO, chunk_bytes: int | None = None) -> Tensor:
    """Same computation as ``monarch_attention_b200`` for q, k, v (and the result) in host memory.

    q, k, v: CPU tensors (E, H, N, D) / (E, H, N, Dv) with unit inner stride; pinned for overlap.
    out:     optional CPU tensor (E, H, N, Dv) to receive the result (pinned for overlap).
    device:  CUDA device to run on (default: the current one).
    heads_per_chunk: most heads in a pipeline chunk (the last chunks are smaller: each at most half of what is left), and with that
             the device scratch: three chunks and the workspace of one; 8 measured best for 16 heads of N = 16384 (2.20 ms per call
             against 2.60 ms unpipelined; 4 gives 2.23 ms, 2 loses again to per-chunk start-up).  Small heads are
             grouped beyond the default 8, see ``chunk_bytes``.
    chunk_bytes: chunks of less than this of a tensor grow to it, over batch elements too (``group_chunks``).  Default: ``CHUNK_BYTES``
             with the default heads_per_chunk, 0 (never) with any other.
    wait:    block until the result is in ``out``; with ``wait=False`` the current stream has been made
             to wait for the last copy instead, and the caller synchronises it before reading ``out``
             (and keeps q, k, v, the mask and ``out`` alive until then).
    streamed: for a sequence of calls with ``wait=False`` whose host inputs are already valid when each call
             is made: the copy-in of a call starts while the kernels and the copy-out of the previous call
             are still running (``ma_b200_forward_host_streamed``), so that the host-to-device link never
             idles between calls.
    """
    _check_device_free_inputs(q, k, v, attn_mask)
    if q.is_cuda or k.is_cuda or v.is_cuda or (attn_mask is not None and attn_mask.is_cuda):
        raise ValueError("monarch_attention_b200_host takes host tensors; use monarch_attention_b200 for device ones")
    if heads_per_chunk < 1:
        raise ValueError("heads_per_chunk must be at least 1")
    if chunk_bytes is None:
        chunk_bytes = CHUNK_BYTES if heads_per_chunk == HEADS_PER_CHUNK else 0
    elif chunk_bytes < 0:
        raise ValueError("chunk_bytes must not be negative")
    E, H, N, _ = q.shape
    Dv = v.shape[-1]
    if out is None:
        out = torch.empty((E, H, N, Dv), dtype=v.dtype, pin_memory=True)
    elif out.is_cuda or tuple(out.shape) != (E, H, N, Dv) or out.dtype != v.dtype or out.stride(-1) != 1:
        raise ValueError("out must be a host tensor of shape (E, H, N, Dv), value's dtype and unit inner stride")
    if E == 0 or H == 0 or N == 0:
        return out
    lib = _cabi.load()
    q, k, v = (t if t.stride(-1) == 1 else t.contiguous() for t in (q, k, v))
    mask = None
    if attn_mask is not None:
        mask = attn_mask.view(torch.uint8) if attn_mask.dtype == torch.bool else (attn_mask != 0).view(torch.uint8)
        mask = mask if mask.stride(-1) == 1 else mask.contiguous()
    prob = make_problem(q, k, v, out, mask, T, B, pre_pad, kernel)
    if lib.ma_b200_host_scratch_bytes(C.byref(prob), heads_per_chunk) == 0:  # (says what is wrong with the problem, if anything is)
        raise ValueError(lib.ma_b200_host_last_error().decode())
    device = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    with torch.cuda.device(device):
        heads, elements, least = group_chunks(E, H, N * max(q.shape[-1], Dv) * q.element_size(), heads_per_chunk, chunk_bytes)
        need = lib.ma_b200_host_scratch_bytes_grouped(C.byref(prob), heads, elements)
        if need == 0:
            raise ValueError(lib.ma_b200_host_last_error().decode())
        idx = device.index if device.index is not None else torch.cuda.current_device()
        scratch = _scratch.get(idx)
        if scratch is None or scratch.numel() < need:
            torch.cuda.synchronize(device)  # an earlier call may still be using the old scratch
            scratch = _scratch[idx] = torch.empty(need, dtype=torch.uint8, device=device)
        stream = torch.cuda.current_stream(device)
        rc = lib.ma_b200_forward_host_grouped(C.byref(prob), heads, elements, least, int(streamed), scratch.data_ptr(),
                                              scratch.numel(), stream.cuda_stream)
        if rc != 0:
            _cabi.raise_for_status(rc, lib.ma_b200_host_last_error().decode())
        if wait:
            stream.synchronize()
    return out
