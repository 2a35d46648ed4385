"""The choice between the warp-level and the tile kernels where one is faster by an eighth or more on 148 SMs; the microseconds are warp-level /
tile."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu

CALLS = [  # B, M, D, T, heads, family
    (72, 72, 64, 1, 4, "warp-mma"),    # 12.4 / 18.5
    (65, 65, 64, 2, 4, "warp-mma"),    # 25.3 / 36.2
    (33, 75, 32, 1, 96, "warp-mma"),   # 57 / 73
    (96, 33, 32, 1, 16, "warp-mma"),   # 18.6 / 25.0
    (128, 16, 64, 1, 128, "tile"),     # 122 / 89
    (128, 16, 64, 1, 256, "tile"),     # 237 / 169
    (16, 128, 64, 1, 192, "warp-mma"),  # 126 / 146
    (64, 121, 64, 2, 48, "tile")]      # long documents


@pytest.mark.parametrize("B,M,D,T,heads,family", CALLS)
def test_the_faster_family_is_taken(B, M, D, T, heads, family):
    from monarch_attention_b200 import _cabi
    from monarch_attention_b200.monarch_attention import make_problem
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the times are those of 148 SMs")
    t = torch.zeros(1, 1, B * M - 1, D, dtype=torch.bfloat16, device="cuda")
    got = _cabi.load().ma_b200_kernel_of_part(C.byref(make_problem(t, t, t, t, None, T, B, False)), heads)
    assert _cabi.KERNEL_NAMES[got] == family
