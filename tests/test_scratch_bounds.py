"""What a call takes beside its operands: the scratch of the 32-bit products and of the chunked recurrences stays below 256 MB, or is the
smallest portion's (host arithmetic of the libraries, no GPU)."""
from ctypes import c_int, c_long

import pytest

from gpt_fast_b200.csrc import build

LIMIT = 256 << 20


def floats(lib, name, *args):
    fn = getattr(build.library(lib), name)
    fn.restype = c_long
    return fn(*map(c_int, args))


@pytest.mark.parametrize("K", [512, 513, 3072, 14336, 28672, 500000])
@pytest.mark.parametrize("N", [1, 70, 3072, 4096, 28672, 151936, 3000000])
def test_slices_of_a_product(N, K):
    for M in (1, 16, 17, 33, 198, 512, 600, 1728, 8192, 70000):
        got = floats("gemm_simt", "gfb_gemm_simt_scratch_floats", M, N, K)
        rows = min(M, 64 if M > 32 else 32 if M > 16 else 16)
        assert 0 <= 4 * got <= max(LIMIT, 4 * rows * N), (M, N, K)
        assert (got == 0) == (K <= 512) and got % N == 0


def test_chunks_of_the_recurrences():
    for T, n in ((64, 1), (2048, 1), (100000, 3), (5000, 4000)):
        for H, d, dv in ((1, 64, 64), (16, 128, 128), (64, 128, 256)):
            for lib, name, args, one in (("delta_chunk", "gfb_delta_chunks_scratch_floats", (H, d, dv), H * (64 * 64 + 64 * d * 3 + (d + 64) * dv + d)),
                                         ("ssd_chunk", "gfb_ssd_chunks_scratch_floats", (H, dv, d, 1), 64 * 64 + 64 * d + H * (68 + d * dv))):
                assert 0 < 4 * floats(lib, name, T, n, *args) <= max(LIMIT, 4 * one)
