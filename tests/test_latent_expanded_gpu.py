"""Prompts of latent attention with keys and values expanded per head: tiles of 128 and pairs of 256 tokens, blocks of 128 keys, sequences that go on
behind cached tokens, windows (also over pages that are gone), sinks and both kinds of gates, against 64-bit attention over the same
cached rows, and no further from it than attention on the latent itself."""
import pytest
import torch

from gpt_fast_b200 import ops
from gpt_fast_b200.ops.cuda import expand_latents
from gpt_fast_b200.ops.types import PagedKV
from gpt_fast_b200.parts import POSITIONS, build_part
from gpt_fast_b200.config.spec import PartSpec
from test_kernels_gpu import DEV, make_batch, rnd

BF = torch.bfloat16


def case(H, R, q_lens, starts, window, sinks, per_head, size=1.0, seed=0):
    batch, table, n_pages = make_batch(q_lens, starts, 20, 64, 40, seed=3 + seed)
    T, gates = batch.n_tokens, H if per_head else H * 128
    kv_off, g_off = H * 192, H * 192 + R + 64
    W = -(-(g_off + gates) // 8) * 8
    proj = rnd(T, W, dtype=BF, seed=1 + seed)
    proj[:, :kv_off] *= size
    pool = rnd(n_pages, 1, 64, R + 64, dtype=BF, seed=2 + seed)
    kv = PagedKV(pool, torch.zeros(n_pages, 1, 64, 0, dtype=BF, device=DEV), table, 64)
    position = build_part(POSITIONS, PartSpec("rope", dict(head_dim=64, base=10000.0, pairing="interleaved")))
    position.prepare(40 * 64, DEV)
    return dict(batch=batch, proj=proj, kv=kv, position=position, H=H, R=R, kv_off=kv_off, g_off=g_off, per_head=per_head, window=window,
                sink=rnd(H, seed=4, scale=2.0) if sinks else None, norm=1.0 + rnd(R, seed=5, scale=0.1), wuk=rnd(H, 128, R, dtype=BF, scale=R ** -0.5, seed=6),
                wuv=rnd(H, R, 128, dtype=BF, scale=R ** -0.5, seed=7), scale=0.0722)


def expanded(c):
    T, H = c["batch"].n_tokens, c["H"]
    guard = torch.full((T + 1, H * 128), 7.0, dtype=BF, device=DEV)
    assert ops.latent_expanded(c["proj"], 0, c["kv_off"], c["g_off"], c["per_head"], guard[:-1], c["kv"], c["batch"], H, 128, 64, 128, c["R"], c["norm"], 1e-5,
                               c["position"].table, "interleaved", True, c["wuk"], c["wuv"],
                               ops.value_scales(c["wuv"], c["norm"]), c["scale"], c["window"], c["sink"])
    ops.check_status(c["batch"].status)
    assert bool((guard[-1] == 7.0).all())
    return guard[:-1]


def on_the_latent(c):
    T, H, R = c["batch"].n_tokens, c["H"], c["R"]
    q = torch.empty(T, H, R + 64, dtype=BF, device=DEV)
    ops.latent_prepare(c["proj"], 0, c["kv_off"], q, c["kv"], c["batch"], H, 128, 64, R, c["norm"], 1e-5, c["position"].table, "interleaved", True)
    ops.headwise_linear(c["proj"], c["wuk"], q.view(T, -1), H, 128, R, a_off=0, a_stride=192, out_stride=R + 64)
    o, y = torch.empty(T, H * R, dtype=BF, device=DEV), torch.empty(T, H * 128, dtype=BF, device=DEV)
    ops.attention(q, c["kv"], c["batch"], o, H, 1, R + 64, c["scale"], c["window"], sink=c["sink"], v_head_dim=R, values_in_keys=True)
    ops.headwise_linear(o, c["wuv"], y, H, R, 128, gate=c["proj"], gate_off=c["g_off"], gate_per_head=c["per_head"])
    return y


def want(c):
    """In 64 bits, over the rows that the cache holds."""
    b, H, R, kv = c["batch"], c["H"], c["R"], c["kv"]
    cu, out = b.cu_seqlens.tolist(), []
    for i in range(b.n_seqs):
        slot, n = int(b.slots[i]), cu[i + 1] - cu[i]
        start = int(b.lengths[slot])
        pos = torch.arange(start, start + n, device=DEV)
        first = max(0, start - c["window"] + 1) if c["window"] else 0
        at = torch.arange(first, start + n, device=DEV)
        rows = kv.k_pool[kv.page_table[slot, at // 64].long(), 0, at % 64].double()
        p = c["proj"][cu[i]:cu[i + 1]].double()
        q = p[:, :H * 192].view(n, H, 192)
        cs = c["position"].table[pos].double()
        u, v = q[..., 128::2], q[..., 129::2]
        turned = torch.stack([u * cs[:, None, :, 0] - v * cs[:, None, :, 1], v * cs[:, None, :, 0] + u * cs[:, None, :, 1]], -1).flatten(-2)
        k = torch.einsum("jr,hdr->jhd", rows[:, :R], c["wuk"].double())
        s = (torch.einsum("thd,jhd->htj", q[..., :128], k) + torch.einsum("thd,jd->htj", turned, rows[:, R:])) * c["scale"]
        dist = pos[:, None] - at[None]
        s = s.masked_fill((dist < 0) | ((dist >= c["window"]) if c["window"] else (dist < 0)), -torch.inf)
        if c["sink"] is not None:
            s = torch.cat([s, c["sink"].double()[:, None, None].expand(H, n, 1)], 2)
        w = s.softmax(-1)[..., :len(at)]
        y = torch.einsum("htj,jhd->thd", w, torch.einsum("jr,hrd->jhd", rows[:, :R], c["wuv"].double()))
        g = torch.sigmoid(p[:, c["g_off"]:c["g_off"] + (H if c["per_head"] else H * 128)])
        out.append((y * g.view(n, H, -1)).reshape(n, H * 128))
    return torch.cat(out)


@pytest.mark.gpu
@pytest.mark.parametrize("H,R,q_lens,starts,window,sinks,per_head", [
    (1, 64, [2], [0], None, False, False),
    (16, 512, [128], [0], None, False, False),                           # a whole tile
    (4, 512, [129, 127], [0, 0], None, True, True),
    (3, 128, [256, 257, 255], [0, 0, 0], None, False, False),            # a whole pair of tiles, one and a bit, nearly one
    (2, 512, [1, 700, 64], [0, 0, 100], None, True, False),              # a lone token beside a prompt; one that goes on
    (2, 192, [300, 280], [63, 129], None, False, True),
    (2, 512, [400], [0], 1, False, True),
    (4, 256, [600, 40], [0, 0], 64, True, True),                         # windows inside a block; tiles that are active in turn
    (2, 512, [500], [333], 200, False, False),
    (2, 320, [1200], [0], 500, True, False),
])
def test_against_64_bits(H, R, q_lens, starts, window, sinks, per_head):
    c = case(H, R, q_lens, starts, window, sinks, per_head)
    got = expanded(c).double()
    ref = want(c)
    # keys, values, weights and outputs are rounded to bfloat16 once each
    assert float((got - ref).norm() / ref.norm()) < 6e-3
    torch.testing.assert_close(got, ref, rtol=4e-2, atol=4e-2 * float(ref.square().mean().sqrt()))


@pytest.mark.gpu
@pytest.mark.parametrize("size", [0.25, 1.0, 4.0])
@pytest.mark.parametrize("window", [None, 256])
def test_no_further_from_64_bits_than_on_the_latent(size, window):
    c = case(8, 512, [900, 300], [0, 0], window, False, False, size)
    err = [float((f(c).double() - want(c)).norm() / want(c).norm()) for f in (expanded, on_the_latent)]
    assert err[0] <= 1.005 * err[1], err                                 # (1.2e6 roundings: half a percent is far more than two draws differ)


@pytest.mark.gpu
def test_value_columns_of_every_scale():
    """Columns of values from 1e-20 to 1e20: each is as near to 64 bits as the others."""
    c = case(2, 512, [300], [0], None, False, False)
    spread = torch.logspace(-20, 20, 128, device=DEV)
    c["wuv"] = (c["wuv"].float() * spread).to(BF)
    got, ref = expanded(c).double().view(300, 2, 128), want(c).view(300, 2, 128)
    err = (got - ref).norm(dim=(0, 1)) / ref.norm(dim=(0, 1))
    assert float(err.max()) < 6e-3, err


@pytest.mark.gpu
@pytest.mark.parametrize("depth", [8.0, 14.5, 20.0, 25.5, 30.0, 34.0])
@pytest.mark.parametrize("peak", [0, 400, 699])
def test_a_flat_tail_far_below_a_peak(depth, peak):
    """One key whose weight is 2^depth times every other one's, ahead of the others, among them and behind them.  Half of the value columns hold nothing
    of the peak: what they get is the tail's share, as far below the row as that is, and no worse than on the latent."""
    c = case(2, 128, [700], [0], None, False, True)
    R, kv_off = 128, c["kv_off"]
    c["position"].table[..., 0], c["position"].table[..., 1] = 1.0, 0.0                    # no rotation: a score is set by one number of the key
    c["norm"] = torch.ones(R, device=DEV)
    c["proj"][:, :c["g_off"]] = 0.0
    q = c["proj"][:, :kv_off].view(700, 2, 192)
    q[:, :, 128] = 64.0
    others = torch.arange(700, device=DEV) != peak
    c["proj"][others, kv_off:kv_off + 64] = rnd(1, 64, dtype=BF, seed=9)                   # the tail's latent, the same for all: its errors add up
    c["proj"][peak, kv_off + 64:kv_off + 128] = rnd(64, dtype=BF, seed=10)
    c["proj"][others, kv_off + R] = -depth / (1.4426950408889634 * 64.0 * c["scale"])
    c["wuv"][:, 64:, :64] = 0.0
    c["wuv"][:, :64, 64:] = 0.0
    y = [f(c).double().view(700, 2, 128)[1:] for f in (expanded, on_the_latent)]
    ref = want(c).view(700, 2, 128)[1:]
    sees = torch.arange(1, 700, device=DEV) >= peak
    for cols, rows in ((slice(0, 64), slice(None)), (slice(64, 128), sees)):
        err = [float(((v - ref)[rows][..., cols]).norm() / ref[rows][..., cols].norm()) for v in y]
        # 2^-9 is the output's rounding, at most; weights are multiples of 2^-24 at least, half of that against 2^12 at the peak
        assert err[0] <= max(1.05 * err[1], 2.0 ** -8, 2.0 ** (depth - 37)), (depth, peak, err)


def test_scales_of_values():
    w = torch.randn(3, 64, 16) * torch.logspace(-30, 30, 16)
    w[0, :, 3] = 0.0
    w[1, 5, 4] = float("inf")
    norm = 1.0 + 0.1 * torch.randn(64)
    s, back = ops.value_scales(w, norm)
    bound = 8.0 * (w.abs() * norm.abs()[None, :, None]).sum(1).flatten()
    fine = (bound > 2.0 ** -100) & (bound < 2.0 ** 100)                    # (not the columns of zeros and of an infinity)
    assert bool((s * back == 1.0).all()) and bool((s.log2() == s.log2().round()).all())
    assert bool(((bound * s)[fine] < 2.0 ** 15).all()) and bool(((bound * s)[fine] >= 2.0 ** 14 * 0.999).all())
    assert bool(s.isfinite().all()) and float(s.min()) > 0.0


@pytest.mark.gpu
def test_the_cache_is_the_same_and_what_lies_beyond_is_not_read_into_results():
    """The same rows are appended; NaNs behind a sequence's end, and pages ahead of the window that are gone, change nothing."""
    a, b = case(4, 512, [200, 130], [0, 250], 100, True, True), case(4, 512, [200, 130], [0, 250], 100, True, True)
    first = expanded(a)
    table, slots = b["kv"].page_table, b["batch"].slots.tolist()
    b["kv"].page_table[slots[1], 0:2] = -1                               # keys 0 to 127; the window begins at 151
    for i, n in ((0, 200), (1, 380)):
        page = int(table[slots[i], n // 64])
        b["kv"].k_pool[page, 0, n % 64:] = float("nan")
    assert torch.equal(expanded(b).view(torch.int16), first.view(torch.int16))
    on_the_latent(a)
    for i, (lo, hi) in enumerate(((0, 200), (250, 380))):
        at = torch.arange(lo, hi, device=DEV)
        pages = table[slots[i], at // 64].long()
        assert torch.equal(a["kv"].k_pool[pages, 0, at % 64].view(torch.int16), b["kv"].k_pool[pages, 0, at % 64].view(torch.int16))


@pytest.mark.gpu
def test_what_it_does_not_take_runs_on_the_latent():
    few = case(2, 512, [20], [2000], None, False, False)                 # few new tokens behind many cached ones
    y = torch.empty(20, 256, dtype=BF, device=DEV)
    args = (0, few["kv_off"], few["g_off"], False, y, few["kv"], few["batch"], 2, 128, 64, 128, 512, few["norm"], 1e-5, few["position"].table, "interleaved",
            True, few["wuk"], few["wuv"], ops.value_scales(few["wuv"], few["norm"]), few["scale"])
    assert not ops.latent_expanded(few["proj"], *args)
    assert not ops.latent_expanded(few["proj"].float(), *args)


def test_the_rule():
    assert expand_latents(4096, 1, 4096, 4096) and expand_latents(20, 1, 20, 128) and expand_latents(2056, 16, 256, 256)
    assert not expand_latents(16, 16, 1, 128)                            # a decode step
    assert not expand_latents(100, 1, 100, 2176) and expand_latents(300, 1, 300, 1024)


def test_the_rule_refuses_many_short_continuations():
    slower = [(128, 64, 2, 128, 16), (512, 64, 8, 128, 16), (2240, 64, 35, 128, 16), (4096, 64, 64, 256, 16), (32, 16, 2, 128, 128)]
    faster = [(4096, 64, 64, 128, 16), (1024, 16, 64, 256, 16), (32, 16, 2, 128, 16), (3200, 16, 200, 512, 16), (4096, 1, 4096, 4096, 128), (100, 1, 100, 128, 128)]
    assert not any(expand_latents(*c) for c in slower) and all(expand_latents(*c) for c in faster)
