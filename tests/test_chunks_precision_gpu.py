"""How far the chunked recurrences are from 64 bits beside the token-by-token kernels: with decays as models start from (steps of 0.001 to
0.1, A of 1 to 16), with fast ones, and with keys that are alike."""
import math

import pytest
import torch

import test_delta_chunks_gpu as delta
import test_ssd_chunks_gpu as ssd
from test_kernels_gpu import DEV

pytestmark = pytest.mark.gpu
LENS, H, D = [700, 333], 4, 128


def model_decays(x, n):
    g = torch.Generator().manual_seed(5)
    dt = torch.exp(torch.rand(n, generator=g) * math.log(100.0) + math.log(1e-3))
    x["dt_bias"] = (dt + torch.log(-torch.expm1(-dt))).to(DEV)
    x["a_log"] = torch.log(torch.rand(H, generator=g) * 15 + 1).to(DEV)
    return x


def errors(which, x, dim, **kw):
    """outputs' distance from 64 bits, token by token and in chunks"""
    S0 = torch.zeros(len(LENS) + 2, 4 + H * D * dim, device=DEV).double()
    outs = []
    for chunks in (False, True):
        if which is delta:
            outs.append(which.run(x, LENS, H, H, D, dim, kw.get("head_decay", False), S0.float(), chunks))
        else:
            outs.append(which.run(x, LENS, H, dim, D, 1, S0.float(), chunks))
    args = (x, LENS, H, H, D, dim, kw.get("head_decay", False)) if which is delta else (x, LENS, H, dim, D, 1)
    want = which.exact(*args, S0, outs[0][1].slots.tolist())
    return [float((o.double() - want).norm() / want.norm()) for o, _ in outs]


# independent keys: sums of other pieces, so within a tenth of the token-by-token kernel's rounding at worst
@pytest.mark.parametrize("rate", [None, 4.0, 0.0, -6.0])
def test_delta_rule(rate):
    x = delta.inputs(LENS, H, H, D, D, False, rate or 0.0)
    by_token, in_chunks = errors(delta, model_decays(x, H * D) if rate is None else x, D)
    assert in_chunks <= 1.1 * by_token


@pytest.mark.parametrize("rate", [None, 4.0, 0.0, -6.0])
def test_state_space(rate):
    x = ssd.inputs(LENS, H, 64, D, 1, rate or 0.0)
    by_token, in_chunks = errors(ssd, model_decays(x, H) if rate is None else x, 64)
    assert in_chunks <= 1.1 * by_token


# Keys that are alike make the chunk's triangular system far from the identity, and the rounding of its 32-bit entries counts with it: the
# entries' sums are made in 64 bits from pieces of 16 terms (chains of 64 terms left the outputs 2.7 times as far as token by token)
@pytest.mark.parametrize("alike,most", [(0.5, 1.15), (0.9, 1.6), (0.99, 2.1)])
@pytest.mark.parametrize("rate", [-6.0, -3.0])
@pytest.mark.parametrize("head_decay", [False, True])
def test_delta_rule_with_keys_that_are_alike(alike, most, rate, head_decay):
    x = delta.inputs(LENS, H, H, D, D, head_decay, rate)
    k = x["qkv"][:, 2 + H * D:2 + 2 * H * D]
    one = torch.randn(1, H * D, generator=torch.Generator().manual_seed(7)).to(DEV)
    k.copy_(alike ** 0.5 * one + (1 - alike) ** 0.5 * k)
    x["beta"] += 4.0
    by_token, in_chunks = errors(delta, x, D, head_decay=head_decay)
    assert in_chunks <= most * by_token
