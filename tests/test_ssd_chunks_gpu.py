"""The state space in chunks of 64 tokens (and its choice by length) against the token-by-token kernel and against 64-bit sums: lengths
around whole chunks, several sequences and groups, with and without the skip, decays from almost none to all at once."""
import pytest
import torch

from gpt_fast_b200 import ops
from test_kernels_gpu import DEV, make_batch, rnd

pytestmark = pytest.mark.gpu


def inputs(lens, H, P, N, G, rate, dtype=torch.float32):
    n = sum(lens)
    return dict(x=rnd(n, H * P + 2 * G * N + 4, seed=1), dt=rnd(n, H + 1, dtype=dtype, seed=2), dt_bias=rnd(H, seed=3) - rate,
                a_log=rnd(H, scale=0.5, seed=4) + rate, skip=rnd(H, seed=5))


def run(x, lens, H, P, N, G, state, chunks, skip=True):
    batch, _, _ = make_batch(lens, [3] * len(lens), len(lens) + 2, 64, 200, seed=9)
    out = torch.full((sum(lens) + 1, H, P), 7.0, device=DEV)
    k = ops.kernels()
    old = k.SSD_CHUNK_TOKENS
    try:
        type(k).SSD_CHUNK_TOKENS = 1 if chunks else 1 << 30
        ops.ssd_scan(x["x"], H * P + 4, H * P + 4 + G * N, x["dt"], 1, x["dt_bias"], x["a_log"], x["skip"] if skip else None, state, 4, out[:-1],
                     batch, H, P, N, G)
    finally:
        type(k).SSD_CHUNK_TOKENS = old
    assert bool((out[-1] == 7.0).all())
    return out[:-1], batch


def exact(x, lens, H, P, N, G, state, slots, skip=True):
    n = sum(lens)
    f = x["x"].double()
    v = f[:, :H * P].reshape(n, H, P)
    B, C = (f[:, H * P + 4 + i * G * N:H * P + 4 + (i + 1) * G * N].reshape(n, G, N).repeat_interleave(H // G, 1) for i in (0, 1))
    dt = torch.nn.functional.softplus(x["dt"].double()[:, 1:1 + H] + x["dt_bias"].double(), threshold=60)
    decay = torch.exp(-torch.exp(x["a_log"].double()) * dt)
    out, t = [], 0
    for slot, ln in zip(slots, lens):
        S = state[slot, 4:].double().view(H, N, P)
        for _ in range(ln):
            S = decay[t][:, None, None] * S + B[t][:, :, None] * (dt[t][:, None] * v[t])[:, None, :]
            out.append(torch.einsum("hnp,hn->hp", S, C[t]) + (x["skip"].double()[:, None] * v[t] if skip else 0.0))
            t += 1
        state[slot, 4:] = S.flatten()
    return torch.stack(out)


@pytest.mark.parametrize("rate", [0.0, 3.0, -6.0])
@pytest.mark.parametrize("lens,H,P,N,G,skip", [([1], 1, 64, 64, 1, True), ([64], 4, 64, 128, 2, True), ([65, 15, 128], 2, 64, 128, 1, False),
                                               ([130, 63], 3, 128, 64, 3, True), ([16, 17, 48, 200], 4, 64, 128, 1, True)])
def test_chunks_against_64_bit_and_token_by_token(lens, H, P, N, G, skip, rate):
    x = inputs(lens, H, P, N, G, rate)
    S0 = rnd(len(lens) + 2, 4 + H * N * P, seed=6).double()
    states = [S0.float().clone() for _ in range(2)]
    by_token, batch = run(x, lens, H, P, N, G, states[0], False, skip)
    in_chunks, _ = run(x, lens, H, P, N, G, states[1], True, skip)
    sizes = exact(dict(x, x=x["x"].abs(), skip=x["skip"].abs()), lens, H, P, N, G, S0.abs(), batch.slots.tolist(), skip)
    want = exact(x, lens, H, P, N, G, S0, batch.slots.tolist(), skip)
    err = lambda got, ref: float((got.double() - ref).norm() / ref.norm())  # noqa: E731
    # 32-bit sums of the same products in another order: as near to 64 bits as the token-by-token kernel, or within a few 2^-24
    assert err(in_chunks, want) <= max(1.5 * err(by_token, want), 1e-6)
    assert err(states[1], S0) <= max(1.5 * err(states[0], S0), 1e-6)
    # a number is at most 32 + 12 roundings of partial sums and a dozen of its factors away: 56 times 2^-24 of the sum of its terms' sizes
    assert bool(((in_chunks.double() - want).abs() <= 56 * 2.0 ** -24 * sizes).all())
    assert torch.equal(states[1][:, :4], states[0][:, :4])


def test_more_chunks_than_are_in_flight_together():
    lens, H, P, N = [4400, 4100], 64, 64, 128         # 134 chunks of 64 heads: two rounds of the scratch
    x = inputs(lens, H, P, N, 1, 1.0)
    states = [torch.zeros(4, 4 + H * N * P, device=DEV) for _ in range(2)]
    by_token, _ = run(x, lens, H, P, N, 1, states[0], False)
    in_chunks, _ = run(x, lens, H, P, N, 1, states[1], True)
    torch.testing.assert_close(in_chunks, by_token, rtol=1e-4, atol=5e-4)
    torch.testing.assert_close(states[1], states[0], rtol=1e-4, atol=5e-4)
