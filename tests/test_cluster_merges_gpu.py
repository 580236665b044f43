"""What slices of a sum leave, merged within a cluster of blocks: the split over K of a product with few tokens, whose bits are those of its
partial sums added in ascending order, and the slices of a decode step's attention, up to the largest cluster and one beyond."""
import math

import pytest
import torch

from gpt_fast_b200 import ops
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
