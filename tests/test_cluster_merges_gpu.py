"""What slices of a sum leave, merged within a cluster of blocks: the split over K of a product with few tokens, whose bits are those of its
partial sums added in ascending order, and the slices of a decode step's attention, up to the largest cluster and one beyond."""
import math

import pytest
import torch

from gpt_fast_b200 import ops
from gpt_fast_b200.ops.cuda import split_parts
from test_kernels_gpu import DEV, make_batch, rnd
from gpt_fast_b200.ops.types import PagedKV

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("splits", [2, 3, 8, 9])
@pytest.mark.parametrize("bn,M,N", [(16, 1, 128), (16, 16, 136), (32, 17, 264), (64, 33, 128), (128, 100, 392), (128, 300, 264)])
def test_split_products(bn, M, N, splits):
    K = 64 * splits * 2 - 40                              # a ragged last slice
    a, w = rnd(M, K, dtype=torch.bfloat16, seed=1), rnd(N, K, dtype=torch.bfloat16, scale=K ** -0.5, seed=2)
    k, plan = ops.kernels(), (1, bn, splits, 3)
    parts = k._linear_tc(a, w, torch.empty(M, N, device=DEV), "store", plan=plan, defer=True)
    total = parts[0].clone()
    for p in parts[1:]:
        total += p
    for dtype in (torch.float32, torch.bfloat16):
        guard = torch.full((M + 1, N), 7.0, dtype=dtype, device=DEV)
        k._linear_tc(a, w, guard[:M], "store", plan=plan)
        assert torch.equal(guard[:M], total.to(dtype)) and bool((guard[M] == 7.0).all())
    x = rnd(M, N, seed=3)
    got = x.clone()
    k._linear_tc(a, w, got, "add", plan=plan)
    assert torch.equal(got, x + total)
    f = torch.nn.functional
    for mode, want in (("gelu", f.gelu(total)), ("gelu_tanh", f.gelu(total, approximate="tanh")), ("relu2", f.relu(total) ** 2)):
        out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
        k._linear_tc(a, w, out, mode, plan=plan)
        torch.testing.assert_close(out.float(), want, rtol=2.0 ** -7, atol=1e-5)         # (one rounding to bfloat16, the activation's own error)
    if N % 16 == 0:
        out = torch.empty(M, N // 2, dtype=torch.bfloat16, device=DEV)
        k._linear_tc(a, w, out, "swiglu", plan=plan)
        torch.testing.assert_close(out.float(), f.silu(total[:, 0::2]) * total[:, 1::2], rtol=2.0 ** -7, atol=1e-5)


@pytest.mark.parametrize("splits", [2, 7, 8, 9])
@pytest.mark.parametrize("H,G,d,sinks", [(6, 2, 128, False), (8, 1, 64, True), (4, 4, 128, True)])
def test_slices_of_attention(splits, H, G, d, sinks):
    batch, table, n_pages = make_batch([1, 1, 1], [1100, 0, 64], 4, 64, 20, seed=2)      # eighteen pages, one, two: slices without keys too
    k, v = (rnd(n_pages, G, 64, d, dtype=torch.bfloat16, seed=s) for s in (1, 2))
    kv, q = PagedKV(k, v, table, 64), rnd(3, H, d, dtype=torch.bfloat16, seed=3)
    sink = rnd(H, seed=4) if sinks else None
    outs = []
    for n in (1, splits):
        guard = torch.full((4, H * d), 7.0, dtype=torch.bfloat16, device=DEV)
        ops.kernels()._attention_bf16(q, kv, batch, guard[:3], H, G, d, 1 / math.sqrt(d), None, splits=n, sink=sink)
        assert bool((guard[3] == 7.0).all())
        outs.append(guard[:3].float())
    ops.check_status(batch.status)
    # sums in another order, rounded to bfloat16 once; the weights are rounded against another maximum
    torch.testing.assert_close(outs[1], outs[0], rtol=2.0 ** -6, atol=4e-3)


@pytest.mark.parametrize("splits", [2, 5, 8])
@pytest.mark.parametrize("bn,M,N", [(16, 3, 144), (32, 31, 272), (128, 130, 400)])
def test_products_have_the_bits_of_parts_in_memory(bn, M, N, splits):
    K = 64 * splits * 2 - 40
    a, w = rnd(M, K, dtype=torch.bfloat16, seed=1), rnd(N, K, dtype=torch.bfloat16, scale=2 * K ** -0.5, seed=2)
    for mode, width, dtype in (("store", N, torch.float32), ("store", N, torch.bfloat16), ("add", N, torch.float32), ("swiglu", N // 2, torch.bfloat16),
                               ("gelu", N, torch.bfloat16), ("gelu_tanh", N, torch.bfloat16), ("relu2", N, torch.bfloat16)):
        outs = [rnd(M, width, seed=3).to(dtype) for _ in range(2)]
        for out, merge in zip(outs, (True, False)):
            ops.kernels()._linear_tc(a, w, out, mode, plan=(1, bn, splits, 3), merge=merge)
        assert torch.equal(*outs), mode


@pytest.mark.parametrize("splits", [2, 3, 8])
@pytest.mark.parametrize("H,G,d,sinks,window,keep", [(6, 2, 128, False, None, 0), (8, 1, 64, True, None, 0), (24, 8, 128, True, 200, 0),
                                                     (8, 8, 128, False, 130, 70), (16, 4, 64, False, 1000, 0)])
def test_attention_has_the_bits_of_slices_in_memory(H, G, d, sinks, window, keep, splits):
    starts = [1100, 0, 64, 700, 511, 37]                                                 # slices without keys too
    batch, table, n_pages = make_batch([1] * 6, starts, 7, 64, 20, seed=2)
    k, v = (rnd(n_pages, G, 64, d, dtype=torch.bfloat16, seed=s) for s in (1, 2))
    kv, q, sink = PagedKV(k, v, table, 64), rnd(6, H, d, dtype=torch.bfloat16, seed=3), rnd(H, seed=4) if sinks else None
    outs = [torch.empty(6, H * d, dtype=torch.bfloat16, device=DEV) for _ in range(2)]
    for out, merge in zip(outs, (True, False)):
        ops.kernels()._attention_bf16(q, kv, batch, out, H, G, d, 1 / math.sqrt(d), window, splits=splits, sink=sink, keep_first=keep, merge=merge)
    ops.check_status(batch.status)
    assert torch.equal(*outs)


@pytest.mark.parametrize("H,G,d,window", [(24, 8, 128, None), (8, 2, 64, 300)])
def test_rotary_attention_has_the_bits_of_slices_in_memory(H, G, d, window):
    starts, outs = [1100, 0, 64], []
    table = torch.empty(20 * 64, d // 2, 2, device=DEV)
    ops.rope_table((1.0 / (10000 ** (torch.arange(d // 2).float() * 2 / d))).to(DEV), table)
    for merge in (True, False):
        batch, pages, n_pages = make_batch([1] * 3, starts, 4, 64, 20, seed=2)
        assert 1 < ops.kernels().decode_slices(batch.max_kv_len, 64, 3 * G) <= 8
        kv = PagedKV(rnd(n_pages, G, 64, d, dtype=torch.bfloat16, seed=1), rnd(n_pages, G, 64, d, dtype=torch.bfloat16, seed=2), pages, 64)
        outs.append(torch.empty(3, H * d, dtype=torch.bfloat16, device=DEV))
        assert ops.kernels().rope_append_attention(None, rnd(3, 3, (H + 2 * G) * d, seed=5), kv, batch, table, outs[-1], H, G, d, "interleaved", True,
                                                   1 / math.sqrt(d), window, merge=merge)
        ops.check_status(batch.status)
    assert torch.equal(*outs)


def test_parts_of_a_split():
    assert [split_parts(K, s) for K, s in ((64, 4), (640, 4), (640, 9), (600, 9), (3072, 16), (1, 1))] == [1, 4, 5, 5, 16, 1]
