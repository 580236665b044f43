"""Prompts against a shared latent on tcgen05: every rank the kernel takes, heads that fill a tile of 128 (token, head) rows or straddle it,
one to many pages, windows and sinks, sequences that go on behind cached tokens, against 64-bit softmax attention."""
import dataclasses
from ctypes import c_float, c_int

import pytest
import torch

from gpt_fast_b200 import ops
from gpt_fast_b200.ops.cuda import _ptr, _stream
from gpt_fast_b200.ops.types import PagedKV
from test_kernels_gpu import DEV, REF, make_batch, rnd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R", [128, 256, 384, 512])
@pytest.mark.parametrize("H,q_lens,starts,window,sinks", [
    (1, [2], [0], None, False),                          # two rows
    (16, [8, 9], [0, 56], None, False),                  # one whole tile, one and a bit, up to a page's edge
    (7, [130, 3, 65], [0, 63, 640], None, True),         # tiles that end inside a token
    (48, [20, 40], [1, 700], 64, True),                  # windows that begin inside a page
    (16, [300], [0], 1, False),
    (16, [200, 1, 64], [0, 5, 64], 500, False),
])
def test_latent_prompts(R, H, q_lens, starts, window, sinks):
    dtype = torch.bfloat16
    batch, table, n_pages = make_batch(q_lens, starts, 6, 64, 16, seed=3)
    kv = PagedKV(rnd(n_pages, 1, 64, R + 64, dtype=dtype, scale=0.5, seed=1), torch.zeros(n_pages, 1, 64, 0, dtype=dtype, device=DEV), table, 64)
    q, sink = rnd(batch.n_tokens, H, R + 64, dtype=dtype, scale=0.5, seed=2), rnd(H, seed=4, scale=2.0) if sinks else None
    guard = torch.full((batch.n_tokens + 1, H * R), 7.0, dtype=dtype, device=DEV)
    out = guard[:-1]
    ops.attention(q, kv, batch, out, H, 1, R + 64, 0.25, window, sink=sink, v_head_dim=R, values_in_keys=True)
    ops.check_status(batch.status)
    assert bool((guard[-1] == 7.0).all())
    cpu = dataclasses.replace(batch, **{f: getattr(batch, f).cpu() for f in ("cu_seqlens", "tok_seq", "slots", "lengths", "status")})
    want = torch.empty(batch.n_tokens, H * R, dtype=torch.float64)
    REF.attention(q.cpu(), PagedKV(kv.k_pool.cpu(), kv.v_pool.cpu(), table.cpu(), 64), cpu, want, H, 1, R + 64, 0.25, window,
                  sink=sink.cpu() if sinks else None, v_head_dim=R, values_in_keys=True)
    # P and the output are rounded to bfloat16 once each (2^-9), values are of size 0.5 to 2
    torch.testing.assert_close(out.double().cpu(), want, rtol=2e-2, atol=1e-2)
    assert float((out.double().cpu() - want).norm() / want.norm()) < 5e-3


def test_one_warp_that_rescales_every_page():
    """Rows whose maxima rise by more than 2^8 from page to page, in one of the four softmax warps: that warp is late for every page, and
    the others' weights of the next page are not counted for it.  The same bits in every run."""
    dtype, H, R, n = torch.bfloat16, 16, 256, 640
    batch, table, n_pages = make_batch([n], [0], 1, 64, 16, seed=5)
    pool = rnd(n_pages, 1, 64, R + 64, dtype=dtype, scale=0.5, seed=1)
    for i in range(n // 64):
        pool[table[0, i].item(), 0, :, R] = float(i)
    q = rnd(n, H, R + 64, dtype=dtype, scale=0.5, seed=2)
    q[:, :, R] = 0.0
    late = torch.arange(n, device=DEV) % 8 // 2 == 1                  # tokens 2 and 3 of eight: rows 32 to 63 of every tile
    q[late, :, R] = 32.0
    kv = PagedKV(pool, torch.zeros(n_pages, 1, 64, 0, dtype=dtype, device=DEV), table, 64)
    runs = []
    for _ in range(20):
        out = torch.empty(n, H * R, dtype=dtype, device=DEV)
        ops.attention(q, kv, batch, out, H, 1, R + 64, 0.25, v_head_dim=R, values_in_keys=True)
        runs.append(out)
    ops.check_status(batch.status)
    assert all(torch.equal(r.view(torch.int16), runs[0].view(torch.int16)) for r in runs)
    cpu = dataclasses.replace(batch, **{f: getattr(batch, f).cpu() for f in ("cu_seqlens", "tok_seq", "slots", "lengths", "status")})
    want = torch.empty(n, H * R, dtype=torch.float64)
    REF.attention(q.cpu(), PagedKV(kv.k_pool.cpu(), kv.v_pool.cpu(), table.cpu(), 64), cpu, want, H, 1, R + 64, 0.25, v_head_dim=R, values_in_keys=True)
    assert float((runs[0].double().cpu() - want).norm() / want.norm()) < 5e-3


@pytest.mark.parametrize("size", [0.5, 1.0, 2.0, 4.0])
def test_no_further_from_64_bits_than_the_kernel_of_decode_steps(size):
    """Rows with many weights of one size, and rows with few large ones."""
    dtype, H, R, n, scale = torch.bfloat16, 8, 512, 600, 0.0722
    batch, table, n_pages = make_batch([n], [0], 1, 64, 16, seed=6)
    kv = PagedKV(rnd(n_pages, 1, 64, R + 64, dtype=dtype, seed=1), torch.zeros(n_pages, 1, 64, 0, dtype=dtype, device=DEV), table, 64)
    q = rnd(n, H, R + 64, dtype=dtype, scale=size, seed=2)
    rows = kv.k_pool[table[0, :-(-n // 64)].long(), 0].reshape(-1, R + 64)[:n].double()
    s = torch.einsum("thd,kd->htk", q.double(), rows) * scale
    s = s.masked_fill(torch.ones(n, n, dtype=torch.bool, device=DEV).triu(1), -torch.inf)
    want = torch.einsum("htk,kr->thr", s.softmax(-1), rows[:, :R]).reshape(n, H * R)
    tc, other = (torch.empty(n, H * R, dtype=dtype, device=DEV) for _ in range(2))
    ops.attention(q, kv, batch, tc, H, 1, R + 64, scale, v_head_dim=R, values_in_keys=True)
    k = ops.kernels()
    k._call("latent", "gfb_latent_attention", _ptr(q), _ptr(other), _ptr(kv.k_pool), _ptr(table), c_int(table.shape[1]), c_int(64), c_int(n_pages),
            *k._batch_args(batch), c_int(n), c_int(H), c_int(R + 64), c_int(R), c_float(scale), c_int(0), _ptr(None), c_int(1), _ptr(None),
            _ptr(batch.status), _stream())
    ops.check_status(batch.status)
    err = lambda got: float((got.double() - want).norm() / want.norm())  # noqa: E731
    # the norm of 2.5e6 roundings of 2^-9: half a percent is far more than two draws of them differ
    assert err(tc) <= 1.005 * err(other)
