"""The delta rule in chunks of 64 tokens (and its choice by length) against the token-by-token kernel and against 64-bit sums: lengths
around whole chunks, several sequences, fewer key heads than heads, one decay per head, decays that forget at once, states that go on."""
import pytest
import torch

from gpt_fast_b200 import ops
from test_kernels_gpu import DEV, make_batch, rnd

pytestmark = pytest.mark.gpu


def inputs(lens, H, J, d, dv, head_decay, rate, dtype=torch.float32):
    n = sum(lens)
    qkv = rnd(n, 2 * J * d + H * dv + 4, seed=1)
    per = H if head_decay else H * d
    return dict(qkv=qkv, beta=rnd(n, H + 1, dtype=dtype, seed=2), a=rnd(n, per + 3, seed=3), dt_bias=rnd(per, seed=4) - rate,
                a_log=rnd(H, scale=0.5, seed=5) + rate)


def run(x, lens, H, J, d, dv, head_decay, state, chunks):
    batch, _, _ = make_batch(lens, [3] * len(lens), len(lens) + 2, 64, 200, seed=9)
    out = torch.full((sum(lens) + 1, H, dv), 7.0, device=DEV)
    k = ops.kernels()
    old = k.DELTA_CHUNK_TOKENS
    try:
        type(k).DELTA_CHUNK_TOKENS = 1 if chunks else 1 << 30
        ops.delta_rule(x["qkv"].clone(), (2, 2 + J * d, 2 + 2 * J * d), x["beta"], 1, x["a"].clone(), 2, x["dt_bias"], x["a_log"], state, 4,
                       out[:-1], batch, H, J, d, dv, d ** -0.5, **({"head_decay": True} if head_decay else {}))
    finally:
        type(k).DELTA_CHUNK_TOKENS = old
    assert bool((out[-1] == 7.0).all())
    return out[:-1], batch


def exact(x, lens, H, J, d, dv, head_decay, state, slots):
    n = sum(lens)
    f = x["qkv"].double()
    q, k = (f[:, 2 + i * J * d:2 + (i + 1) * J * d].reshape(n, J, d).repeat_interleave(H // J, 1) for i in (0, 1))
    v = f[:, 2 + 2 * J * d:2 + 2 * J * d + H * dv].reshape(n, H, dv)
    q, k = (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
    beta = torch.sigmoid(x["beta"].double()[:, 1:1 + H])
    a = torch.nn.functional.softplus(x["a"].double()[:, 2:2 + x["dt_bias"].numel()] + x["dt_bias"].double(), threshold=60)
    a = a[:, :, None].expand(n, H, d) if head_decay else a.view(n, H, d)
    g = torch.exp(-torch.exp(x["a_log"].double())[:, None] * a)
    out, t = [], 0
    for slot, ln in zip(slots, lens):
        S = state[slot, 4:].double().view(H, d, dv)
        for _ in range(ln):
            S = g[t][:, :, None] * S
            u = beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
            S = S + k[t][:, :, None] * u[:, None, :]
            out.append(torch.einsum("hdv,hd->hv", S, q[t]) * d ** -0.5)
            t += 1
        state[slot, 4:] = S.flatten()
    return torch.stack(out)


@pytest.mark.parametrize("rate", [0.0, 4.0, -6.0])
@pytest.mark.parametrize("lens,H,J,d,dv,head_decay", [([1], 1, 1, 64, 64, False), ([64], 2, 2, 128, 128, False), ([65, 15, 128], 2, 1, 128, 64, False),
                                                      ([130, 63], 2, 2, 64, 192, True), ([16, 17, 48, 200], 4, 2, 128, 128, True), ([333], 3, 3, 64, 128, False)])
def test_chunks_against_64_bit_and_token_by_token(lens, H, J, d, dv, head_decay, rate):
    x = inputs(lens, H, J, d, dv, head_decay, rate)
    S0 = rnd(len(lens) + 2, 4 + H * d * dv, seed=6).double()
    states = [S0.float().clone() for _ in range(2)]
    by_token, batch = run(x, lens, H, J, d, dv, head_decay, states[0], False)
    in_chunks, _ = run(x, lens, H, J, d, dv, head_decay, states[1], True)
    want = exact(x, lens, H, J, d, dv, head_decay, S0, batch.slots.tolist())
    err = lambda got, ref: float((got.double() - ref).norm() / ref.norm())  # noqa: E731
    # both are 32-bit sums of the same products in another order: as near to 64 bits as the token-by-token kernel, or within a few 2^-24
    assert err(in_chunks, want) <= max(1.5 * err(by_token, want), 1e-6)
    assert err(states[1], S0) <= max(1.5 * err(states[0], S0), 1e-6)
    torch.testing.assert_close(in_chunks.double(), want, rtol=2e-5, atol=2e-5)
    assert torch.equal(states[1][:, :4], states[0][:, :4])


def test_more_chunks_than_are_in_flight_together():
    lens, H, d = [2600, 2700], 16, 128                # 84 chunks of 16 heads: two rounds of the scratch
    x = inputs(lens, H, H, d, d, False, 2.0)
    states = [torch.zeros(4, 4 + H * d * d, device=DEV) for _ in range(2)]
    by_token, _ = run(x, lens, H, H, d, d, False, states[0], False)
    in_chunks, _ = run(x, lens, H, H, d, d, False, states[1], True)
    torch.testing.assert_close(in_chunks, by_token, rtol=1e-4, atol=1e-5)
    torch.testing.assert_close(states[1], states[0], rtol=1e-4, atol=1e-5)
