"""The chunks that the host entry point runs: every head once, in order, none larger than the scratch holds, none needlessly small."""
import random

import pytest

from monarch_attention_b200.host_pipeline import group_chunks, plan_chunks

MB = 1 << 20


@pytest.mark.parametrize("E,H,head_bytes,want", [
    (3, 16, 2300 * 128, [(0, 0, 8), (0, 8, 8), (1, 0, 8), (1, 8, 8), (2, 0, 8), (2, 8, 7), (2, 15, 1)]),  # 15 fit a chunk
    (1, 12, 3000 * 128, [(0, 0, 6), (0, 6, 5), (0, 11, 1)]),  # 11
    (9, 4, MB // 4, [(0, 0, 16), (4, 0, 16), (8, 0, 4)]),     # four elements
    (5, 2, MB, [(0, 0, 4), (2, 0, 4), (4, 0, 2)]),            # a remainder of one element
    (2, 20, MB // 4, [(0, 0, 10), (0, 10, 10), (1, 0, 10), (1, 10, 8), (1, 18, 2)]),
    (1, 16, 2 * MB, [(0, 0, 8), (0, 8, 4), (0, 12, 2), (0, 14, 1), (0, 15, 1)])])  # large heads: down to one
def test_chunks_of_a_call(E, H, head_bytes, want):
    assert plan_chunks(E, H, *group_chunks(E, H, head_bytes, 8)) == want


def test_every_head_is_in_one_chunk():
    rng = random.Random(5)
    for _ in range(3000):
        E, H, head_bytes, asked = rng.randint(1, 40), rng.randint(1, 40), int(2 ** rng.uniform(5, 24)), rng.choice([1, 3, 8, 8, 8, 30])
        heads, elements, least = group_chunks(E, H, head_bytes, asked, rng.choice([0, MB, 4 * MB]))
        at = 0
        plan = plan_chunks(E, H, heads, elements, least)
        for e, h0, n in plan:
            assert e * H + h0 == at and (n <= min(heads, H - h0) or (h0 == 0 and n % H == 0 and n <= elements * H))
            at += n
        assert at == E * H
        ends = [n for e, _, n in plan if e == E - 1]
        assert all(n >= min(least, heads) for n in ends[:-1])
        if least > 1 and elements == 1:  # an element before the last is cut evenly
            for at in range(E - 1):
                cut = [n for e, _, n in plan if e == at]
                assert max(cut) - min(cut) <= 1
        # as many chunks as it takes, and the few at the end of the last element
        per_element = -(-H // heads)
        full = -(-E // elements) if elements > 1 else E * per_element
        assert len(plan) <= full + H.bit_length()


def test_a_chunk_is_no_larger_than_a_grid():
    for E, H in ((200000, 1), (3, 70000), (9000, 30)):
        heads, elements, _ = group_chunks(E, H, 16, 8)
        assert heads * elements <= 65535
