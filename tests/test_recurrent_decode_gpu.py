"""One token per sequence in one launch (delta rule, state space) against the token-by-token kernel, which rows of an odd length take: the
same bits, at heads around a lane's rows and a block's columns, few and many sequences, fewer key heads, one decay per head."""
import pytest
import torch

from gpt_fast_b200 import ops
from test_kernels_gpu import DEV, DTYPES, make_batch, rnd

pytestmark = pytest.mark.gpu


def states(n_seqs, size):
    wide = rnd(n_seqs + 2, 4 + size + 1, seed=6)                       # an odd row length: the general kernel
    return wide[:, :-1].contiguous(), wide


def same(a, b):
    assert torch.equal(a.view(torch.int32), b.view(torch.int32))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("n,H,J,d,dv,head_decay", [(1, 1, 1, 8, 4, False), (3, 2, 1, 64, 64, False), (8, 16, 16, 128, 128, False), (5, 4, 2, 65, 132, True),
                                                   (2, 2, 2, 256, 36, True), (40, 16, 8, 128, 64, True), (64, 8, 8, 64, 128, False)])
def test_delta_rule(n, H, J, d, dv, head_decay, dtype):
    batch, _, _ = make_batch([1] * n, [3] * n, n + 2, 64, 200, seed=9)
    per = H if head_decay else H * d
    qkv, beta, a = rnd(n, 2 * J * d + H * dv + 3, seed=1), rnd(n, H + 1, dtype=dtype, seed=2), rnd(n, per + 3, seed=3)
    dt_bias, a_log = rnd(per, seed=4), rnd(H, scale=0.5, seed=5)
    outs = []
    rows = states(n, H * d * dv)
    for st in rows:
        out = torch.full((n + 1, H, dv), 7.0, device=DEV)
        ops.delta_rule(qkv.clone(), (1, 1 + J * d, 1 + 2 * J * d), beta, 1, a.clone(), 2, dt_bias, a_log, st, 4, out[:-1], batch, H, J, d, dv,
                       d ** -0.5, **({"head_decay": True} if head_decay else {}))
        assert bool((out[-1] == 7.0).all())
        outs.append(out)
    same(outs[0], outs[1])
    same(rows[0], rows[1][:, :-1].contiguous())


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("n,H,P,N,G,skip", [(1, 1, 4, 8, 1, True), (3, 4, 64, 128, 2, True), (8, 64, 64, 128, 1, False), (5, 3, 132, 65, 3, True),
                                            (2, 2, 36, 512, 1, True), (40, 16, 64, 64, 1, True)])
def test_state_space(n, H, P, N, G, skip, dtype):
    batch, _, _ = make_batch([1] * n, [3] * n, n + 2, 64, 200, seed=9)
    x, dt = rnd(n, H * P + 2 * G * N + 5, seed=1), rnd(n, H + 1, dtype=dtype, seed=2)
    dt_bias, a_log, sk = rnd(H, seed=3), rnd(H, scale=0.5, seed=4), rnd(H, seed=5)
    outs = []
    rows = states(n, H * P * N)
    for st in rows:
        out = torch.full((n + 1, H, P), 7.0, device=DEV)
        ops.ssd_scan(x, H * P + 5, H * P + 5 + G * N, dt, 1, dt_bias, a_log, sk if skip else None, st, 4, out[:-1], batch, H, P, N, G)
        assert bool((out[-1] == 7.0).all())
        outs.append(out)
    same(outs[0], outs[1])
    same(rows[0], rows[1][:, :-1].contiguous())
