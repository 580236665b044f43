"""The vectorised row kernels of the mixers at the sizes where they can go wrong: the convolution at tiles of eight tokens that straddle
sequences and their carried inputs, the gated norm at every register form, the per-head product on tcgen05 at its tiles' edges."""
import pytest
import torch

from gpt_fast_b200 import ops
from test_kernels_gpu import DEV, DTYPES, make_batch, rnd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("taps", [2, 3, 4])
@pytest.mark.parametrize("lens", [[1], [1, 1, 1], [2, 2], [8], [9, 1, 2, 3, 30], [65, 7]])
def test_convolution_by_four_channels(dtype, taps, lens):
    T, C, off = sum(lens), 132, 4
    src, w, b, ib = rnd(T, C + 8, dtype=dtype, seed=1), rnd(C, taps, seed=2), rnd(C, seed=3), rnd(C, seed=4)
    batch, _, _ = make_batch(lens, [3] * len(lens), len(lens) + 1, 64, 4, seed=5)
    state = rnd(len(lens) + 1, 3 + (taps - 1) * C, seed=6)
    before, want_state, want = state.clone(), state.double(), []
    for i, s in enumerate(batch.slots.tolist()):
        lo, hi = int(batch.cu_seqlens[i]), int(batch.cu_seqlens[i + 1])
        full = torch.cat([before[s, 3:].double().view(taps - 1, C), src[lo:hi, off:off + C].double() + ib.double()])
        z = sum(full[j:j + hi - lo] * w[:, j].double() for j in range(taps)) + b.double()
        want.append(z * torch.sigmoid(z))
        want_state[s, 3:] = full[-(taps - 1):].flatten()
    guard = torch.full((T + 1, C), 7.0, device=DEV)
    ops.short_conv(src, off, C, w, b, state, 3, guard[:-1], batch, True, in_bias=ib)
    assert bool((guard[-1] == 7.0).all())
    torch.testing.assert_close(guard[:-1].double(), torch.cat(want), rtol=1e-5, atol=1e-5)
    torch.testing.assert_close(state.double(), want_state, rtol=1e-6, atol=1e-6)


@pytest.mark.parametrize("lens", [[1] * 40 + [30], [2] * 30 + [1] * 9, [1] * 255 + [257], [300] + [1] * 20])
def test_convolution_of_a_long_sequence_among_single_tokens(lens):
    test_convolution_by_four_channels(torch.bfloat16, 4, lens)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("first", [True, False])
@pytest.mark.parametrize("groups,gs", [(3, 4), (2, 128), (5, 132), (1, 512), (2, 516), (1, 4096), (1, 4100), (1, 8192)])
def test_gated_norm_in_registers(dtype, groups, gs, first):
    T, C = 5, groups * gs
    y, gate, w = rnd(T, C, seed=1) * 2, rnd(T, C + 8, dtype=dtype, seed=2), rnd(C, seed=3) + 1
    guard = torch.full((T + 1, C), 7.0, dtype=dtype, device=DEV)
    ops.gated_norm(y, gate, 4, w, guard[:-1], gs, 1e-5, act="silu", gate_first=first)
    z = gate[:, 4:4 + C].double()
    a = z * torch.sigmoid(z)
    v = y.double() * a if first else y.double()
    v = v.view(T, groups, gs)
    n = (v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-5)).reshape(T, C) * w.double()
    want = n if first else n * a
    assert bool((guard[-1] == 7.0).all())
    torch.testing.assert_close(guard[:-1].double(), want, **(dict(rtol=2e-5, atol=2e-5) if dtype == torch.float32 else dict(rtol=8e-3, atol=8e-3)))


@pytest.mark.parametrize("T", [65, 128, 129, 300])
@pytest.mark.parametrize("H,K,N,gates", [(1, 64, 128, 0), (3, 128, 512, 0), (2, 512, 128, 1), (5, 320, 256, 2)])
def test_per_head_products_on_tensor_cores(T, H, K, N, gates):
    dtype = torch.bfloat16
    a, w = rnd(T, H * (K + 8) + 16, dtype=dtype, seed=1), rnd(H, K, N, dtype=dtype, scale=K ** -0.5, seed=2)
    gate = rnd(T, 3 + H * (N if gates == 2 else 1), dtype=dtype, seed=3) if gates else None
    guard = torch.full((T + 1, 4 + H * (N + 4)), 7.0, dtype=dtype, device=DEV)
    ops.headwise_linear(a, w, guard[:-1], H, K, N, a_off=8, a_stride=K + 8, out_off=4, out_stride=N + 4, gate=gate, gate_off=3, gate_per_head=gates == 1)
    x = a[:, 8:8 + H * (K + 8)].reshape(T, H, K + 8)[:, :, :K].double()
    want = torch.einsum("thk,hkn->thn", x, w.double())
    if gates:
        g = torch.sigmoid(gate[:, 3:].double())
        want = want * (g.view(T, H, N) if gates == 2 else g.view(T, H, 1))
    got = guard[:-1, 4:].reshape(T, H, N + 4)
    # one rounding to bfloat16 (2^-9) of sums of unit size
    torch.testing.assert_close(got[:, :, :N].double(), want, rtol=4e-3, atol=4e-3)
    assert bool((guard[-1] == 7.0).all()) and bool((guard[:, :4] == 7.0).all()) and bool((got[:, :, N:] == 7.0).all())
