"""Latent attention's per-token work in 16-byte accesses against the general kernel, which the same numbers take in rows that are no multiple of
16 bytes: the same turned numbers, and latents whose norm is summed in another order."""
import pytest
import torch

from gpt_fast_b200 import ops
from gpt_fast_b200.config.spec import PartSpec
from gpt_fast_b200.ops.types import PagedKV
from gpt_fast_b200.parts import POSITIONS, build_part
from test_kernels_gpu import DEV, make_batch, rnd

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.mark.parametrize("norm_dtype", [torch.float32, BF])
@pytest.mark.parametrize("H,d,rot,R", [(1, 8, 8, 8), (16, 128, 64, 512), (40, 64, 32, 1032), (3, 24, 16, 120)])
def test_wide_rows(H, d, rot, R, norm_dtype):
    batch, table, n_pages = make_batch([3, 1, 70], [62, 130, 0], 5, 64, 4, seed=2)
    T, kv_off = batch.n_tokens, 8 + H * (d + rot)
    wide = rnd(T, kv_off + R + rot + 8, dtype=BF, seed=3)
    position = build_part(POSITIONS, PartSpec("rope", dict(head_dim=rot, base=100.0, pairing="interleaved")))
    position.prepare(256, DEV)
    norm = (rnd(R, seed=4) + 1).to(norm_dtype)
    got = []
    for src in (wide, torch.cat([wide, wide[:, :1]], 1).contiguous()):
        kv = PagedKV(torch.full((n_pages, 1, 64, R + rot), 7.0, dtype=BF, device=DEV), torch.zeros(n_pages, 1, 64, 0, dtype=BF, device=DEV), table, 64)
        q = torch.full((T, H, R + rot), 7.0, dtype=BF, device=DEV)
        ops.latent_prepare(src, 8, kv_off, q, kv, batch, H, d, rot, R, norm, 1e-5, position.table, "interleaved", False)
        assert bool((kv.k_pool == 7.0).all())
        ops.latent_prepare(src, 8, kv_off, q, kv, batch, H, d, rot, R, norm, 1e-5, position.table, "interleaved", True)
        ops.check_status(batch.status)
        got.append((q, kv.k_pool))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1][..., R:], got[1][1][..., R:])
    # one unit of bfloat16 where the two norms round to either side
    torch.testing.assert_close(got[0][1].float(), got[1][1].float(), rtol=2.0 ** -7, atol=0.0)
