"""The experts of a prompt where the rows of their tiles change: tiles of 64 rows with several per expert, 256 from 128 pairs per expert on."""
import pytest
import torch

from gpt_fast_b200 import ops
from test_kernels_gpu import DEV, rnd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [65, 129, 255, 256, 600])
@pytest.mark.parametrize("act", ["glu", "relu2"])
def test_experts_around_the_line(T, act):
    E, top, D, F = 4, 2, 136, 72                                       # 128 pairs per expert: T = 256
    N1 = F if act == "relu2" else 2 * F
    h, w13 = rnd(T, D, dtype=torch.bfloat16, seed=1), rnd(E, N1, D, dtype=torch.bfloat16, scale=D ** -0.5, seed=2)
    w2, w = rnd(E, D, F, dtype=torch.bfloat16, scale=F ** -0.5, seed=3), rnd(T, top, seed=4).abs()
    g = torch.Generator().manual_seed(T)
    idx = (torch.rand(T, top, generator=g) ** 2 * E).int().clamp(max=E - 1).to(DEV)
    x = rnd(T, D, seed=5)
    want = x.double()
    for e in range(E):
        a = h.double() @ w13[e].double().t()
        if act == "relu2":
            a = a.clamp(min=0) ** 2
        else:
            gate, up = a[:, ::2].clamp(max=3.0), a[:, 1::2].clamp(-3.0, 3.0)
            a = gate * torch.sigmoid(1.7 * gate) * (up + 1.0)
        y = a.to(torch.bfloat16).double() @ w2[e].double().t()
        want = want + ((idx == e) * w).sum(1, keepdim=True).double() * y
    ops.moe_experts(h, idx, w, w13, w2, x, 3.0, 1.7, 1.0, act=act)
    ops.check_status(ops.kernels().status)
    # the activations are rounded to bfloat16 once, here from 64 bits and there from 32: a few of them fall to the other neighbour (2^-8)
    assert float((x.double() - want).norm() / want.norm()) < 2e-4
