"""ma_b200_forward_timed launches the kernels of ma_b200_forward: same family, same bits, and a family of one launch has
its whole time in the first entry."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E,H,N,D,B,T,dtype,launches", [
    (1, 8, 128 * 128, 64, 128, 2, torch.bfloat16, 1),   # tile kernels, one launch
    (4, 12, 61 * 63 - 5, 64, 61, 2, torch.float16, 1),  # ... ragged
    (1, 2, 200 * 40, 64, 200, 2, torch.bfloat16, 4),    # tile kernels, a launch per stage
    (1, 2, 4096, 64, 64, 2, torch.bfloat16, 1),         # fused kernel
    (8, 12, 197, 64, 15, 2, torch.bfloat16, 1),         # head-resident kernel
    (2, 3, 250, 64, 16, 2, torch.float32, 1),           # fp32 tensor path, one launch
    (50, 6, 250, 64, 16, 2, torch.float32, 4),          # ... a launch per stage
    # ... while the GPU holds the clusters of all heads at once, whatever their blocks
    (17, 8, 250, 64, 16, 2, torch.float32, 1), (20, 8, 100, 64, 10, 2, torch.float32, 4), (40, 8, 36, 64, 6, 1, torch.float32, 2),
    # ... and blocks above 24 while each cluster has its SMs to itself
    (1, 14, 1024, 64, 32, 2, torch.float32, 1), (2, 8, 625, 64, 25, 2, torch.float32, 4), (2, 13, 576, 64, 24, 2, torch.float32, 1)])
def test_timed_forward_runs_the_kernels_of_the_forward(E, H, N, D, B, T, dtype, launches):
    from monarch_attention_b200 import _cabi
    from monarch_attention_b200.monarch_attention import make_problem
    lib, dev = _cabi.load(), torch.device("cuda:0")
    g = torch.Generator().manual_seed(N)
    q, k, v = (torch.randn(E, H, N, D, generator=g).to(dtype).to(dev) for _ in range(3))
    out, timed = torch.empty_like(v), torch.empty_like(v)
    stream = torch.cuda.current_stream().cuda_stream
    prob = make_problem(q, k, v, out, None, T, B, False)
    ws = torch.empty(lib.ma_b200_workspace_bytes(C.byref(prob)), dtype=torch.uint8, device=dev)
    _cabi.raise_for_status(lib.ma_b200_forward(C.byref(prob), ws.data_ptr(), ws.numel(), stream))
    prob = make_problem(q, k, v, timed, None, T, B, False)
    ms = (C.c_float * (2 * T))(*[-1.0] * (2 * T))
    _cabi.raise_for_status(lib.ma_b200_forward_timed(C.byref(prob), ws.data_ptr(), ws.numel(), stream, ms, 2 * T))
    assert torch.equal(out.view(torch.uint8), timed.view(torch.uint8))
    assert all(x > 0 for x in ms[:launches]) and all(x == 0 for x in ms[launches:])
