"""Attention of prompts in 32-bit, whose rows share their keys and values, has the bits of the kernel that takes a row per block (which the same call
runs for a batch that is said to bring one token per sequence): heads per group that fill a block's rows, straddle tokens or blocks, small and
whole heads, every option of mask and score, and numbers that are not finite where a row does not look."""
import dataclasses
import math

import pytest
import torch

from gpt_fast_b200 import ops
from gpt_fast_b200.ops.cuda import rows_share_keys
from gpt_fast_b200.ops.types import PagedKV
from test_kernels_gpu import DEV, make_batch, rnd



@pytest.fixture
def sharing(monkeypatch):
    monkeypatch.setattr(type(ops.kernels()), "SHARING_ROWS", 1)


def both(batch, kv, q, H, G, d, dv, **kw):
    outs = []
    for most in (batch.max_q_len, 1):
        guard = torch.full((batch.n_tokens + 1, H * dv), 7.0, device=DEV)
        ops.attention(q, kv, dataclasses.replace(batch, max_q_len=most), guard[:-1], H, G, d, 1 / math.sqrt(d), v_head_dim=dv, **kw)
        assert bool((guard[-1] == 7.0).all())
        outs.append(guard[:-1])
    ops.check_status(batch.status)
    return outs


@pytest.mark.gpu
@pytest.mark.parametrize("q_lens,starts", [([2], [0]), ([137, 61], [0, 0]), ([1, 33, 128], [200, 127, 0]), ([5, 300], [1000, 3])])
@pytest.mark.parametrize("H,G,d,dv,page", [(24, 8, 128, 128, 64), (4, 4, 64, 32, 64), (7, 1, 20, 124, 16), (40, 2, 4, 4, 64), (16, 1, 128, 64, 128)])
def test_the_same_bits(sharing, q_lens, starts, H, G, d, dv, page):
    batch, table, n_pages = make_batch(q_lens, starts, 6, page, -(-1400 // page), seed=1)
    kv = PagedKV(rnd(n_pages, G, page, d, seed=2), rnd(n_pages, G, page, dv, seed=3), table, page)
    q = rnd(batch.n_tokens, H, d, seed=4)
    for kw in ({}, dict(window=50), dict(window=1), dict(chunk=48), dict(sink=rnd(H, seed=5)), dict(window=130, bias=rnd(40, H, seed=6)),
               dict(slopes=rnd(H, seed=7).abs()), dict(softcap=2.0)):
        new, row_by_row = both(batch, kv, q, H, G, d, dv, **kw)
        assert torch.equal(new, row_by_row), kw


@pytest.mark.gpu
def test_values_in_keys_and_what_a_row_does_not_see(sharing):
    batch, table, n_pages = make_batch([100, 40], [30, 0], 3, 64, 8, seed=8)
    pool = rnd(n_pages, 1, 64, 96, seed=9)
    kv = PagedKV(pool, torch.zeros(n_pages, 1, 64, 0, device=DEV), table, 64)
    q = rnd(140, 3, 96, seed=10)
    clean, row_by_row = both(batch, kv, q, 3, 1, 96, 64, values_in_keys=True)
    assert torch.equal(clean, row_by_row)
    slot = int(batch.slots[0])
    pool[int(table[slot, 1]), 0, 40] = float("nan")                     # key 104: new token 74 of the first sequence
    for got in both(batch, kv, q, 3, 1, 96, 64, values_in_keys=True):
        assert torch.equal(got[:74], clean[:74]) and torch.equal(got[100:], clean[100:]) and bool(got[74:100].isnan().all())


def test_the_rule():
    assert rows_share_keys(198 * 24, 137, 137, 1536) and rows_share_keys(256, 16, 2016, 1536)
    assert not rows_share_keys(198 * 24, 1, 137, 1536) and not rows_share_keys(1024, 64, 64, 1536) and not rows_share_keys(80, 2, 800, 1536)


def test_the_rule_counts_blocks_that_are_not_full():
    few_live = [(64 * 4 * 8, 4, 4, 1536, 8 * 64), (64 * 2 * 32, 2, 2, 1536, 32 * 64), (16 * 8 * 24, 8, 8, 1536, 8 * 24)]       # a block per row is the faster form
    full = [(64 * 8 * 24, 8, 108, 1536, 8 * 96), (16 * 32 * 32, 32, 32, 1536, 8 * 128), (64 * 4 * 32, 4, 604, 1536, 8 * 64), (200 * 16, 200, 200, 1536, 200)]
    assert not any(rows_share_keys(*c) for c in few_live) and all(rows_share_keys(*c) for c in full)
    assert rows_share_keys(198 * 24, 137, 137, 1536, 8 * 38) and rows_share_keys(8, 2, 2, 1, 4)
