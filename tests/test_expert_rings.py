"""How many blocks of the experts' products share an SM in a decode step (host rule, no GPU)."""
import pytest

from gpt_fast_b200.ops.cuda import expert_blocks_per_sm


@pytest.mark.parametrize("T,top,E,N,want", [(8, 4, 17, 3584, 3), (16, 4, 17, 3584, 2), (1, 4, 17, 3584, 2), (1, 16, 64, 3584, 2), (17, 4, 17, 3584, 2),
                                            (1, 17, 64, 3328, 3), (8, 4, 17, 2048, 2), (4, 20, 10, 5120, 3)])
def test_three_where_two_would_need_a_second_round(T, top, E, N, want):
    assert expert_blocks_per_sm(T, top, E, N, 148) == want
    live = E * (1 - (1 - min(1, top / E)) ** T) * -(-N // 128)
    assert want == 2 or 2 * 148 < live <= 3 * 148
