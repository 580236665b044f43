"""Which steps take the chunked recurrences: by the work of their chunks, not by the longest sequence alone (host rule, no GPU)."""
import pytest

from gpt_fast_b200.ops.cuda import CudaKernels, delta_in_chunks, fewest_chunks, ssd_in_chunks

DELTA_LINE, SSD_LINE = CudaKernels.DELTA_CHUNK_TOKENS, CudaKernels.SSD_CHUNK_TOKENS


@pytest.mark.parametrize("lens", [[1], [64], [65], [63, 1], [64] * 8, [200, 1, 3, 9, 27, 81], [512] + [1] * 63, [48] * 9, [130, 130, 130]])
def test_fewest_chunks(lens):
    real = sum(-(-n // 64) for n in lens)
    assert real - (len(lens) - 1) <= fewest_chunks(sum(lens), len(lens), max(lens)) <= real


# measured at 16 heads of 128 x 128 and at 64 heads of 128 x 64: which form was faster (by more than the runs differ)
@pytest.mark.parametrize("lens,delta,ssd", [([48], False, None), ([128], False, True), ([256], True, True), ([2048], True, True), ([32] * 8, None, None),
                                            ([48] * 8, True, True), ([64] * 8, True, True), ([16] * 32, False, False), ([8] * 64, False, False),
                                            ([512] + [1] * 7, True, True), ([64] + [1] * 15, False, False), ([64] + [1] * 255, False, False),
                                            ([160] + [1] * 63, False, False), ([512] + [1] * 63, False, False), ([512] + [1] * 255, False, False),
                                            ([48] + [1] * 432, False, False), ([32] * 64, False, None), ([64] * 64, False, None), ([1000] * 4 + [1] * 12, None, True), ([256] * 2 + [1] * 30, False, False), ([1, 3, 9, 27, 81, 200], True, True)])
def test_the_faster_form_is_taken(lens, delta, ssd):
    step = sum(lens), len(lens), max(lens)
    assert delta in (None, delta_in_chunks(*step, 16, 128, 128, DELTA_LINE))
    assert ssd in (None, ssd_in_chunks(*step, 64, 64, 128, SSD_LINE))


@pytest.mark.parametrize("n", [1, 2, 8, 64, 256, 1024])
@pytest.mark.parametrize("heads,dim", [(1, 64), (4, 64), (16, 128), (64, 128)])
def test_a_decode_step_is_never_in_chunks(n, heads, dim):
    assert not delta_in_chunks(n, n, 1, heads, dim, dim, DELTA_LINE)
    assert not ssd_in_chunks(n, n, 1, heads, dim, 128, SSD_LINE)
