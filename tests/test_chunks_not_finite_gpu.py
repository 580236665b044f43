"""Numbers that are not finite in the chunked recurrences: a decay that is infinite forgets and nothing else, as token by token."""
import pytest
import torch

import test_delta_chunks_gpu as delta
import test_ssd_chunks_gpu as ssd
from test_kernels_gpu import DEV

pytestmark = pytest.mark.gpu
LENS, H, D = [100, 70], 2, 128
INF = float("inf")


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

