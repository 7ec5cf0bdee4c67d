"""Halo marking from the list of groups: every shape of the list (no group, all groups, groups at the end of a warp's 32), one rank's
edges against all ranks' edges, and twice from one plan."""

import numpy as np
import pytest
import torch

from dynamis_b200 import _lib
from dynamis_b200.graph import BinnedAtoms
from oracle import cpu_oracle as O

pytestmark = pytest.mark.gpu


def _mark(bins, owner, W, rank):
    n = owner.numel()
    needed = torch.full((n, (W + 31) // 32), -1, dtype=torch.int32, device=owner.device)
    foreign = torch.full((n,), 9, dtype=torch.uint8, device=owner.device)
    _lib.check(_lib.lib().dynb_rg_halo_mark_rank(bins.ws.data_ptr(), bins.dtype_code, owner.data_ptr(), n, W, rank, needed.data_ptr(),
                                                 foreign.data_ptr(), None, torch.cuda.current_stream().cuda_stream), "rg_halo_mark")
    return needed.cpu().numpy().view(np.uint32), foreign.cpu().numpy()


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("owners", ["one", "two_slabs", "scattered", "sixty_four"])
@pytest.mark.parametrize("n,length", [(40, 9.0), (3000, 31.0)])
def test_marks(cuda, n, length, owners, dtype):
    rng = np.random.default_rng(n)
    pos = (rng.random((n, 3)) * length)
    W = {"one": 3, "two_slabs": 2, "scattered": 5, "sixty_four": 64}[owners]
    own = {"one": np.ones(n, int), "two_slabs": (pos[:, 2] > 0.4 * length).astype(int), "scattered": rng.integers(0, W, n), "sixty_four": rng.integers(0, W, n)}[owners]
    p = pos.astype(np.float64 if dtype == torch.float64 else np.float32)
    cell, r = (np.eye(3) * length).astype(p.dtype), 4.0
    g = O.radius_graph(p, cell, [True] * 3, r, None)
    a, b = own[g["src"]], own[g["dst"]]
    bins = BinnedAtoms(torch.as_tensor(p, device=cuda), torch.as_tensor(cell), torch.tensor([True] * 3), r)
    bins.launch()
    torch.cuda.synchronize()
    assert bins.done()
    owner = torch.as_tensor(own, device=cuda)
    for rank in (-1, 0, W - 1, -1):
        seen = (a != b) & ((rank < 0) | (a == rank) | (b == rank))
        want = np.zeros((n, (W + 31) // 32), dtype=np.uint32)
        np.bitwise_or.at(want, (g["src"][seen], b[seen] // 32), (np.uint32(1) << (b[seen] % 32).astype(np.uint32)))
        needed, foreign = _mark(bins, owner, W, rank)
        assert (needed == want).all()
        want_f = np.zeros(n, dtype=np.uint8)
        want_f[g["dst"][seen]] = 1
        mine = np.ones(n, bool) if rank < 0 else own == rank
        assert (foreign[mine] == want_f[mine]).all()
