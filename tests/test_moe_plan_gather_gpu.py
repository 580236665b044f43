"""A decode step's plan and gathered rows in one launch, at the edges of its tiles, quarters and scans: every pair gets one row of its expert's
tiles, in the order of the pairs, with its token's numbers; a token that names an expert twice, and pairs of no expert."""
from ctypes import c_int

import pytest
import torch

from gpt_fast_b200 import ops
from gpt_fast_b200.ops.cuda import _ptr, _stream
from test_kernels_gpu import DEV, rnd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,top,E,rows,D,spread", [(1, 1, 1, 16, 8, 1.0), (8, 3, 16, 16, 2048, 1.0), (16, 4, 33, 16, 2040, 3.0), (32, 8, 64, 32, 4096, 1.0),
                                                   (64, 16, 1024, 64, 2056, 2.0), (64, 9, 8, 64, 72, 6.0), (33, 31, 5, 64, 264, 1.0)])
def test_plan_and_rows(T, top, E, rows, D, spread):
    n = T * top
    g = torch.Generator().manual_seed(n)
    idx = (torch.rand(n, generator=g) ** spread * (E + 0.5)).int()                 # E itself: no expert
    live = idx < E
    h = rnd(T, D, dtype=torch.bfloat16, seed=1)
    tiles = (n + min(E, n) * (rows - 1)) // rows
    row_pair, pair_row, tile_expert = (torch.full((k + 1,), -9, dtype=torch.int32, device=DEV) for k in (tiles * rows, n, tiles))
    used, hs, on = torch.zeros(1, dtype=torch.int32, device=DEV), torch.full((tiles * rows + 1, D), 7.0, dtype=torch.bfloat16, device=DEV), idx.to(DEV)
    ops.kernels()._call("moe", "gfb_moe_plan_gather", _ptr(on), c_int(n), c_int(E), c_int(rows), _ptr(h), _ptr(hs), c_int(top), c_int(D), _ptr(row_pair),
                        _ptr(pair_row), _ptr(tile_expert), c_int(tiles), _ptr(used), _stream())
    count = torch.bincount(idx[live].long(), minlength=E)
    per = (count + rows - 1) // rows
    start, ahead = (per.cumsum(0) - per) * rows, count.cumsum(0) - count
    order = torch.sort(torch.where(live, idx, E), stable=True).indices[:int(live.sum())]
    e = idx[order].long()
    want = torch.full((n,), -1)
    want[order] = (start - ahead)[e] + torch.arange(len(order))
    back = torch.full((tiles * rows,), -1)
    back[want[live]] = torch.arange(n)[live]
    n_used = int(per.sum())
    experts = torch.full((tiles,), -1)
    experts[:n_used] = torch.repeat_interleave(torch.arange(E), per)
    guard = torch.tensor([-9])
    assert int(used) == n_used
    assert torch.equal(pair_row.cpu().long(), torch.cat([want, guard]))
    assert torch.equal(row_pair.cpu().long(), torch.cat([back, guard]))
    assert torch.equal(tile_expert.cpu().long(), torch.cat([experts, guard]))
    src = torch.where(back >= 0, back // top, T)[:n_used * rows]
    rows_want = torch.cat([h.cpu(), torch.zeros(1, D, dtype=torch.bfloat16)])[src]
    assert torch.equal(hs.cpu()[:n_used * rows], rows_want) and bool((hs[-1] == 7.0).all())
