"""The reciprocal of the gated epilogue against the division it stands for: every 32-bit number from 1 to infinity."""
from ctypes import c_long

import pytest
import torch

from gpt_fast_b200 import ops
from gpt_fast_b200.ops.cuda import _ptr, _stream
from test_kernels_gpu import DEV

pytestmark = pytest.mark.gpu


def reciprocal(d):
    out = torch.empty_like(d)
    ops.kernels()._call("gemm_tc", "gfb_reciprocal", _ptr(d), _ptr(out), c_long(d.numel()), _stream())
    return out


def test_every_number_from_one_to_infinity():
    lo, hi, step = 0x3F800000, 0x7F800000, 1 << 26
    differ = 0
    for first in range(lo, hi + 1, step):
        bits = torch.arange(first, min(first + step, hi + 1), dtype=torch.int32, device=DEV)
        d = bits.view(torch.float32)
        off = (reciprocal(d).view(torch.int32) - (1.0 / d).view(torch.int32)).abs()
        assert int(off.max()) <= 1
        differ += int((off != 0).sum())
    assert differ == 5


def test_not_a_number_stays_that():
    d = torch.tensor([float("nan"), float("inf"), 1.0, 2.0], device=DEV)
    r = reciprocal(d)
    assert bool(torch.isnan(r[0])) and r[1:].tolist() == [0.0, 1.0, 0.5]
