"""The 32-bit product in bfloat16 pieces at the edges of its tiles, stages and portions of K, against 64-bit sums: no further from them than
the product on CUDA cores, the same bits in every batch, and what is not finite as 32-bit sums have it."""
from ctypes import c_int, c_long, c_void_p

import pytest
import torch

from gpt_fast_b200 import ops
from gpt_fast_b200.csrc import build
from test_kernels_gpu import DEV, rnd


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["store", "add", "swiglu", "gelu", "gelu_tanh", "silu", "relu2"])
@pytest.mark.parametrize("M,N,K", [(1, 2, 384), (16, 128, 416), (17, 130, 388), (33, 66, 2052), (64, 6, 412), (65, 258, 1000), (129, 4, 500), (256, 126, 448),
                                   (257, 3072, 512), (520, 20000, 384), (40, 64, 380), (40, 64, 4)])
def test_edges(mode, M, N, K):
    a, w = rnd(M, K, seed=1), rnd(N, K, scale=K ** -0.5, seed=2)
    got = rnd(M, N // 2 if mode == "swiglu" else N, seed=3)
    z = a.double() @ w.double().t()
    f = torch.nn.functional
    want = {"store": lambda: z, "add": lambda: got.double() + z, "swiglu": lambda: f.silu(z[:, 0::2]) * z[:, 1::2], "gelu": lambda: f.gelu(z),
            "gelu_tanh": lambda: f.gelu(z, approximate="tanh"), "silu": lambda: f.silu(z), "relu2": lambda: f.relu(z) ** 2}[mode]()
    ops.linear(a, w, got, mode)
    # sums of unit scale, each of at most 64 accumulators of which every one loses at most 3 units of 2^-23 of its size, and squared or
    # multiplied with one another
    torch.testing.assert_close(got.double(), want, rtol=2e-5, atol=2e-5)


@pytest.mark.gpu
@pytest.mark.parametrize("spread", [0.0, 1.0, 4.0])
@pytest.mark.parametrize("M,N,K", [(1, 1024, 512), (40, 5120, 3072), (240, 3072, 8192), (300, 20000, 1024)])
def test_nearer_to_64_bits_than_on_cuda_cores(M, N, K, spread):
    """Numbers of one scale, and numbers whose scales spread over e^(+-3) and e^(+-12).  In the last a sum is little more than its largest
    product, which is rounded once on CUDA cores (2.8e-8) and cut off once on tensor cores (5.5e-8): one unit of 2^-24 at most."""
    a, w = rnd(M, K, seed=4), rnd(N, K, seed=5)
    if spread:
        a, w = a * torch.exp(spread * rnd(M, K, seed=6)), w * torch.exp(spread * rnd(N, K, seed=7))
    want = a.double() @ w.double().t()
    ours, cores = torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
    ops.linear(a, w, ours)
    lib = build.library("gemm_simt")
    lib.gfb_gemm_simt_scratch_floats.restype = c_long
    room = torch.empty(max(1, lib.gfb_gemm_simt_scratch_floats(M, N, K)), device=DEV)
    ptr = lambda t: c_void_p(t.data_ptr())  # noqa: E731
    assert lib.gfb_gemm_simt(ptr(a), ptr(w), ptr(cores), 0, 0, c_int(M), c_int(N), c_int(K), 0, ptr(room), c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    error = [((x.double() - want).norm() / want.norm()).item() for x in (ours, cores)]
    assert error[0] <= (error[1] if spread < 4.0 else max(error[1], 2.0 ** -24)), error


@pytest.mark.gpu
@pytest.mark.parametrize("N,K", [(96, 2100), (20000, 1000)])          # portions of K in blocks of their own; one block per tile
def test_a_row_has_the_same_bits_in_every_batch(N, K):
    a, w = rnd(600, K, seed=8), rnd(N, K, seed=9)
    whole = torch.empty(600, N, device=DEV)
    ops.linear(a, w, whole)
    for lo, hi in ((0, 1), (0, 16), (3, 36), (250, 450), (100, 400), (599, 600)):
        part = torch.empty(hi - lo, N, device=DEV)
        ops.linear(a[lo:hi].contiguous(), w, part)
        assert torch.equal(part, whole[lo:hi]), (lo, hi)


@pytest.mark.gpu
@pytest.mark.parametrize("N,K", [(96, 2100), (20000, 388)])
def test_not_finite_and_extreme_numbers(N, K):
    """An infinity against a bfloat16 number and against its own sign, NaNs, numbers that truncation keeps finite, sums that overflow."""
    a, w = rnd(40, K, seed=10), rnd(N, K, seed=11)
    a[3, 5] = float("inf")
    w[:, 5] = 1.0
    a[4, 7], a[4, 8] = float("inf"), float("inf")
    a[5, 9] = float("nan")
    a[6, 10] = torch.tensor(0x7F800001, dtype=torch.int32).view(torch.float32)       # a NaN whose upper half is an infinity's
    w[50, 11] = float("-inf")
    a[7] = 0.0
    a[7, 12] = torch.finfo(torch.float32).max
    a[8] = 2e38
    a[9] = 1e-30
    want = (a.double() @ w.double().t()).float()
    got = torch.empty(40, N, device=DEV)
    ops.linear(a, w, got)
    assert torch.equal(got.isnan(), want.isnan())
    assert torch.equal(got.isinf(), want.isinf())
    assert torch.equal(got[3], torch.full_like(got[3], float("inf")).where(torch.arange(N, device=DEV) != 50, want[3]))
    fine = want.isfinite() & got.isfinite()
    scale = a.abs().nan_to_num(0.0, 0.0, 0.0).double() @ w.abs().nan_to_num(0.0, 0.0, 0.0).double().t()
    assert bool(((got.double() - want.double()).abs() <= 1e-6 * scale + 1e-37)[fine].all())


@pytest.mark.gpu
@pytest.mark.parametrize("N,K", [(2, 28672), (256, 14340), (300, 14336), (130, 8196)])
def test_few_columns_of_long_rows_take_more_portions(N, K):
    """More than 16 portions of K, the last of them shorter: as near to 64 bits as elsewhere, and the same bits in every batch."""
    a, w = rnd(70, K, seed=16), rnd(N, K, seed=17)
    want = a.double() @ w.double().t()
    whole, one = torch.empty(70, N, device=DEV), torch.empty(1, N, device=DEV)
    ops.linear(a, w, whole)
    assert float((whole.double() - want).norm() / want.norm()) < 2.5e-7
    ops.linear(a[69:].contiguous(), w, one)
    assert torch.equal(one[0], whole[69])
    lib = build.library("gemm_split")
    assert lib.gfb_gemm_split_scratch_bytes(70, N, K) > 6 * 70 * K + 16 * 4 * 70 * N


@pytest.mark.gpu
@pytest.mark.parametrize("N,K", [(98, 2100), (18946, 388), (131, 1000)])      # (the last columns are no group of eight)
def test_sums_that_all_need_the_32_bit_numbers(N, K):
    """Every sum of a tile, and every other one, worked out from the 32-bit numbers: infinities at the end of every row, NaNs from the start, small rows
    beside ordinary ones."""
    a, w = rnd(37, K, seed=14), rnd(N, K, seed=15)
    a[:20, K - 1] = float("inf")
    a[20:25] = float("nan")
    a[25:36] *= 1e-33
    w[::2, K - 1] = 0.0                                               # infinity times zero
    want = (a.double() @ w.double().t()).float()
    got = torch.empty(37, N, device=DEV)
    ops.linear(a, w, got)
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got[:20].nan_to_num(), want[:20].nan_to_num())
    torch.testing.assert_close(got[25:36], want[25:36], rtol=2.0 ** -22, atol=0.0)       # (rounded once each, but for sums in another order of 64 bits)
    torch.testing.assert_close(got[36], want[36], rtol=0.0, atol=1e-5 * K ** 0.5)


@pytest.mark.gpu
@pytest.mark.parametrize("N,K", [(96, 2100), (20000, 388)])          # portions of K in blocks of their own; one block per tile
@pytest.mark.parametrize("rows,weights", [(1.0, 1e-24), (1.0, 1e-27), (1.0, 1e-33), (1.0, 1e-36), (1e12, 1e-36), (1e-24, 1.0), (1e-28, 1.0), (1e-30, 1.0),
                                          (1e-34, 1.0), (1e-36, 1.0), (1e-15, 1e-15), (1e-20, 1e-16), (1e30, 1e-36), (1e-36, 1e30)])
def test_small_numbers_keep_their_bits(N, K, rows, weights):
    """Numbers whose third and second pieces bfloat16 does not reach, on either side: each row is as near to 64 bits, by its own size, as sums
    on CUDA cores.  A row of zeros, a zero weight and a lone small number among ordinary ones stay what they are."""
    a, w = rnd(24, K, seed=12) * rows, rnd(N, K, seed=13) * weights
    a[5] = 0.0
    w[7] = 0.0
    a[6, 1:] = 0.0
    want = a.double() @ w.double().t()
    got, cores = torch.empty(24, N, device=DEV), torch.empty(24, N, device=DEV)
    ops.linear(a, w, got)
    lib = build.library("gemm_simt")
    room = torch.empty(max(1, lib.gfb_gemm_simt_scratch_floats(24, N, K)), device=DEV)
    assert lib.gfb_gemm_simt(a.data_ptr(), w.data_ptr(), cores.data_ptr(), 0, 0, 24, N, K, 0, room.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    ours, theirs = ((x.double() - want).norm(dim=1) / want.norm(dim=1) for x in (got, cores))
    some = torch.arange(24, device=DEV) != 5
    assert float(ours[some].max()) <= max(2.0 ** -24, float(theirs[some].max())), (ours, theirs)
    assert not got[5].any() and not got[:, 7].any()


def test_scratch_is_bounded():
    lib = build.library("gemm_split")
    lib.gfb_gemm_split_scratch_bytes.restype = c_long
    for N in (1, 70, 3072, 4096, 28672, 151936, 3000000):
        for K in (4, 512, 3072, 14336, 500000):
            one = lib.gfb_gemm_split_scratch_bytes(c_int(256), c_int(N), c_int(K))
            for M in (1, 17, 198, 600, 8192, 70000):
                got = lib.gfb_gemm_split_scratch_bytes(c_int(M), c_int(N), c_int(K))
                assert 6 * min(M, 256) * K <= got <= max((256 << 20) + 256, one), (M, N, K)
