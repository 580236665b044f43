"""The rules of the experts' kernels: blocks per SM of a decode step's products, launches of the router and of the plan (host only, no GPU)."""
import pytest

from gpt_fast_b200.ops.cuda import expert_blocks_per_sm, plan_with_rows, router_in_one_launch


@pytest.mark.parametrize("T,top,E,N,want", [(8, 4, 17, 3584, 3), (16, 4, 17, 3584, 2), (1, 4, 17, 3584, 2), (1, 16, 64, 3584, 2), (17, 4, 17, 3584, 2),
                                            (1, 17, 64, 3328, 3), (8, 4, 17, 2048, 2), (4, 20, 10, 5120, 3)])
def test_three_where_two_would_need_a_second_round(T, top, E, N, want):
    assert expert_blocks_per_sm(T, top, E, N, 148) == want
    live = E * (1 - (1 - min(1, top / E)) ** T) * -(-N // 128)
    assert want == 2 or 2 * 148 < live <= 3 * 148


@pytest.mark.parametrize("T,rows,D,wide,want", [(64, 128, 4096, False, True), (65, 16, 1024, False, True), (65, 17, 1024, False, False), (3072, 16, 1024, False, True),
                                                (4096, 16, 1024, False, False), (256, 16, 2048, False, True), (1024, 16, 2048, False, True), (512, 16, 4096, False, False),
                                                (2048, 8, 4096, False, True), (4096, 8, 4096, False, False), (256, 64, 2048, False, False),
                                                (256, 32, 2048, True, True), (256, 64, 1024, True, True), (256, 64, 2048, True, False), (2048, 16, 4096, True, False)])
def test_the_router_in_one_launch_where_that_is_faster(T, rows, D, wide, want):
    assert router_in_one_launch(T, rows, D, wide) is want


@pytest.mark.parametrize("pairs,E,D,want", [(24, 17, 2048, True), (256, 16, 2048, True), (512, 16, 2048, False), (512, 64, 2048, True), (64, 8, 1024, False),
                                            (32, 8, 1024, True), (256, 16, 1024, False), (512, 32, 1024, True), (1024, 32, 1024, False), (1024, 32, 2048, True),
                                            (1025, 64, 2048, False), (8, 1025, 2048, False), (1, 1, 8, False)])
def test_plan_and_rows_in_one_launch_where_that_is_faster(pairs, E, D, want):
    assert plan_with_rows(pairs, E, D) is want
