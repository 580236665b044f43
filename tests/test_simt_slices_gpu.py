"""The 32-bit product at the edges of its tiles and of its slices of 512 numbers of k, against 64-bit sums, and the promise that a
row's bits do not depend on the batch: tiles of 16, 32 and 64 rows, slices in blocks of their own or in one block."""
import pytest
import torch

from gpt_fast_b200 import ops
from test_kernels_gpu import DEV, rnd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["store", "add", "swiglu", "gelu"])
@pytest.mark.parametrize("M,N,K", [(1, 70, 511), (16, 64, 512), (17, 130, 513), (33, 66, 2050), (198, 3072, 2048), (65, 12, 3000), (300, 40000, 1040)])
def test_edges_of_tiles_and_slices(mode, M, N, K):
    a, w = rnd(M, K, seed=1), rnd(N, K, scale=K ** -0.5, seed=2)
    out = rnd(M, N // 2 if mode == "swiglu" else N, seed=3)
    want = out.double()
    got = out.clone()
    ops.linear(a, w, got, mode)
    z = a.double() @ w.double().t()
    if mode == "store":
        want = z
    elif mode == "add":
        want = want + z
    elif mode == "swiglu":
        want = torch.nn.functional.silu(z[:, 0::2]) * z[:, 1::2]
    else:
        want = torch.nn.functional.gelu(z)
    # sums of K products of unit scale: K^0.5 2^-24 of random rounding is below 4e-6; the factor covers the largest of 6e6 sums
    torch.testing.assert_close(got.double(), want, rtol=2e-5, atol=2e-5)


@pytest.mark.parametrize("N,K", [(96, 2100), (60000, 1100)])
def test_a_row_has_the_same_bits_in_every_batch(N, K):
    a, w = rnd(260, K, seed=4), rnd(N, K, seed=5)
    whole = torch.empty(260, N, device=DEV)
    ops.linear(a, w, whole)
    for rows in (1, 16, 17, 40, 64, 130, 259):
        part = torch.empty(rows, N, device=DEV)
        ops.linear(a[:rows].contiguous(), w, part)
        assert torch.equal(part, whole[:rows]), rows


@pytest.mark.parametrize("mode", ["store", "add", "swiglu"])
@pytest.mark.parametrize("M,N,K", [(600, 4096, 14336), (1100, 70000, 520)])      # 28 slices in blocks of their own; totals of slices in one block
def test_portions_of_rows_have_the_same_bits(M, N, K, mode):
    a, w = rnd(M, K, seed=6), rnd(N, K, seed=7)
    cols = N // 2 if mode == "swiglu" else N
    start = rnd(M, cols, seed=8)
    whole = torch.cat([start, torch.full((1, cols), 7.0, device=DEV)])
    ops.linear(a, w, whole[:M], mode)
    assert bool((whole[M] == 7.0).all())
    for lo, hi in ((0, 33), (M // 2 - 20, M // 2 + 60), (M - 17, M)):
        part = start[lo:hi].clone()
        ops.linear(a[lo:hi].contiguous(), w, part, mode)
        assert torch.equal(part, whole[lo:hi]), lo
