"""The router over a prompt at the edges of its blocks of tokens and pairs of rows: a token's choice is the same bits as in a small call."""
import pytest
import torch

from gpt_fast_b200 import ops
from test_kernels_gpu import DEV, DTYPES, rnd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("T,E,top,n_extra,D,score,shared", [(65, 1, 1, 0, 16, "sigmoid", False), (72, 17, 3, 1, 264, "softmax", True),
                                                            (129, 32, 4, 0, 1024, "sigmoid", False), (300, 33, 8, 0, 2048, "softmax_top", False),
                                                            (67, 127, 8, 1, 520, "sigmoid_plain", True)])
def test_router_over_a_prompt(T, E, top, n_extra, D, score, shared, dtype):
    h, router = rnd(T, D, dtype=dtype, seed=1), rnd(E + n_extra, D, dtype=dtype, scale=D ** -0.5, seed=2)
    corr = rnd(E, seed=3, scale=0.1)

    def route(x):
        n = x.shape[0]
        idx = torch.full((n + 1, top + shared), -7, dtype=torch.int32, device=DEV)
        w = torch.full((n + 1, top + shared), 7.0, device=DEV)
        extra = torch.full((n + 1, n_extra), 7.0, device=DEV) if n_extra else None
        assert ops.kernels().moe_router(x, router, corr, top, 1.5, idx[:-1], w[:-1], score=score, extra=extra[:-1] if n_extra else None, shared=shared)
        assert bool((idx[-1] == -7).all()) and bool((w[-1] == 7.0).all()) and (not n_extra or bool((extra[-1] == 7.0).all()))
        return idx[:-1], w[:-1], extra[:-1] if n_extra else w[:-1]

    whole = route(h)
    parts = [route(p) for p in h.split(64)]
    for i in range(3):
        assert torch.equal(whole[i], torch.cat([p[i] for p in parts]))
