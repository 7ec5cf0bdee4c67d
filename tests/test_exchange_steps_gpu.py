"""Reverse exchange where a warp takes several steps through the listed rows, next to lists shorter than one step.

Three ranks in one process (all pushes first, then all waits).  Rows go to one peer, to both (two received rows) or to none;
the gradients are small whole numbers, so every sum is exact whatever its order and the result must equal ``index_add_``.
"""

import pytest
import torch

import dynamis_b200 as D

pytestmark = pytest.mark.gpu


def _ranks(n, F, dtype, dev):
    gen = torch.Generator().manual_seed(n + F)
    sends = []
    for r in range(3):
        both = torch.rand(n, generator=gen)
        sends.append({p: torch.nonzero((both < 0.6) if k == 0 else (both > 0.4) & (both < 0.9)).reshape(-1)
                      for k, p in enumerate(p for p in range(3) if p != r)})
    ex, metas = [], []
    for r in range(3):
        so, ro = [0], [0]
        for p in range(3):
            so.append(so[-1] + (sends[r][p].numel() if p != r else 0))
            ro.append(ro[-1] + (sends[p][r].numel() if p != r else 0))
        e = D.FeatureExchanger()
        metas.append(e.local_setup(torch.tensor(so), torch.cat([sends[r][p] for p in range(3) if p != r]), torch.tensor(ro), n, F, r, 3, dev, dtype))
        ex.append(e)
    for e in ex:
        e.connect(metas)
    return ex, sends


# 4 blocks of 8 warps and 2 rows a warp on each of 148 SMs are 9,472 rows a step: 1, 3, 7 rows, one step and a bit, three steps
# and a bit; widths on both sides of the 32 columns and of the four columns a lane takes where a row has no 16-byte pieces
@pytest.mark.parametrize("n", [1, 3, 7, 11000, 34001])
@pytest.mark.parametrize("F,dtype", [(3, torch.float32), (31, torch.float32), (33, torch.float32), (130, torch.float32), (128, torch.float32),
                                     (132, torch.float32), (32, torch.float64), (67, torch.float64)])
@pytest.mark.parametrize("listed_first", [True, False])
def test_reverse_sums_are_exact(cuda, n, F, dtype, listed_first):
    ex, sends = _ranks(n, F, dtype, cuda)
    if not listed_first:  # without the list of first received rows the kernel looks them up itself
        for e in ex:
            e.reverse.row_first = e.reverse.row_first.new_empty(0)
    gen = torch.Generator(device=cuda).manual_seed(1)
    for _ in range(2):
        grads = [torch.randint(-8, 9, (n + sum(sends[p][r].numel() for p in range(3) if p != r), F), generator=gen, device=cuda).to(dtype)
                 for r in range(3)]
        begun = [e.backward_begin(g) for e, g in zip(ex, grads)]
        got = [e.backward_end(*b) for e, b in zip(ex, begun)]
        for r in range(3):
            want = grads[r][:n].clone()
            for p in range(3):
                if p != r:
                    at = n + sum(sends[o][p].numel() for o in range(r) if o != p)
                    rows = sends[r][p].to(cuda)
                    want.index_add_(0, rows, grads[p][at:at + rows.numel()])
            assert torch.equal(got[r], want)
    for e in ex:
        e.check_status()
        e.teardown()
