"""Numbers that are not finite in the chunked recurrences: a decay that is infinite forgets and nothing else, and a token that is spoiled
spoils itself and what comes behind it, as in the token-by-token kernels."""
import pytest
import torch

import test_delta_chunks_gpu as delta
import test_ssd_chunks_gpu as ssd
from test_kernels_gpu import DEV

pytestmark = pytest.mark.gpu
LENS, H, D = [100, 70], 2, 128
INF, NAN = float("inf"), float("nan")


def both(which, x, dim=D, **kw):
    """(outputs, state) token by token and in chunks"""
    pairs = []
    for chunks in (False, True):
        state = torch.zeros(len(LENS) + 2, 4 + H * D * dim, device=DEV)
        if which is delta:
            out, _ = which.run(x, LENS, H, H, D, dim, kw.get("head_decay", False), state, chunks)
        else:
            out, _ = which.run(x, LENS, H, dim, D, 1, state, chunks)
        pairs.append((out, state))
    return pairs


def close(a, b):
    torch.testing.assert_close(a[0], b[0], rtol=1e-4, atol=1e-5)
    torch.testing.assert_close(a[1], b[1], rtol=1e-4, atol=1e-5)
    assert bool(torch.isfinite(a[0]).all())


@pytest.mark.parametrize("head_decay", [False, True])
def test_delta_rule_forgets(head_decay):
    x = delta.inputs(LENS, H, H, D, D, head_decay, 0.0)
    per = 1 if head_decay else D
    x["a"][20, 2] = INF                                   # one channel (or the head) forgets at tokens 20, 50 and 120
    x["a"][50, 2:2 + per] = 3e38
    x["a"][120, 2 + per:2 + 2 * per] = INF
    x["a"][66, 2] = -INF                                  # and one keeps everything
    close(*both(delta, x, head_decay=head_decay))
    x["a_log"][1] = 95.0                                  # a head that forgets at every token
    close(*both(delta, x, head_decay=head_decay))


def test_state_space_forgets():
    x = ssd.inputs(LENS, H, 64, D, 1, 0.0)
    x["a_log"][0] = 95.0
    close(*both(ssd, x, 64))
    x["a_log"][1] = 60.0
    close(*both(ssd, x, 64))


J = H * D
SPOILED = [(delta, "qkv", 2 + 5, D), (delta, "qkv", 2 + J + 5, D), (delta, "qkv", 2 + 2 * J + 5, D), (delta, "beta", 1, D), (delta, "a", 2 + 5, D),
           (ssd, "x", 5, 64), (ssd, "x", H * 64 + 4 + 7, 64), (ssd, "x", H * 64 + 4 + D + 7, 64), (ssd, "dt", 1, 64)]


@pytest.mark.parametrize("value", [NAN, INF])
@pytest.mark.parametrize("t", [5, 37, 63, 64, 90, 100])
@pytest.mark.parametrize("which,name,column,dim", SPOILED, ids=["q", "k", "v", "beta", "a", "x", "B", "C", "dt"])
def test_a_spoiled_token_spoils_nothing_ahead_of_it(which, name, column, dim, t, value):
    x = which.inputs(LENS, H, H, D, D, False, 0.0) if which is delta else which.inputs(LENS, H, dim, D, 1, 0.0)
    clean = both(which, x, dim)[1][0]
    x[name] = x[name].clone()
    x[name][t, column] = value
    (by_token, token_state), (in_chunks, chunk_state) = both(which, x, dim)
    first, last = (0, LENS[0]) if t < LENS[0] else (LENS[0], sum(LENS))
    ahead = torch.ones(sum(LENS), dtype=torch.bool, device=DEV)
    ahead[t:last] = False                                # the other sequence's tokens too
    assert torch.equal(in_chunks[ahead], clean[ahead])
    if not (value == INF and name in ("beta", "a")):     # (an infinite gate or decay input is a number: one, or a decay that forgets)
        assert bool(torch.isnan(in_chunks[t, 0]).any() or torch.isinf(in_chunks[t, 0]).any())
    assert torch.equal(torch.isfinite(in_chunks), torch.isfinite(by_token))
    assert torch.equal(torch.isfinite(chunk_state), torch.isfinite(token_state))
