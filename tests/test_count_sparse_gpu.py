"""The count pass of a thin gas: so many groups that a warp takes several in a row, lists of up to 64 places of many short runs."""

import numpy as np
import pytest
import torch

import dynamis_b200 as D
from _util import assert_same_edges, canon_o, canon_t
from dynamis_b200.graph import plan_radius_graph
from oracle import cpu_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("subset", [False, True])
def test_gas(cuda, subset, dtype):
    n, rho, r = 600_011, 0.004, 5.0
    rng = np.random.default_rng(4)
    length = (n / rho) ** (1.0 / 3.0)
    pos, cell, pbc = (rng.random((n, 3)) * length).astype(dtype), (np.eye(3) * length).astype(dtype), [True] * 3
    targets = rng.permutation(n)[:n - 7] if subset else None
    pos_t, cell_t, pbc_t = torch.as_tensor(pos, device=cuda), torch.as_tensor(cell), torch.tensor(pbc)
    targets_t = torch.as_tensor(targets, device=cuda) if subset else None
    sms = torch.cuda.get_device_properties(cuda).multi_processor_count
    assert plan_radius_graph(pos_t, cell_t, pbc_t, r, targets_t).num_groups >= 2 * 64 * 4 * 5 * sms   # two in a row
    g = O.radius_graph(pos, cell, pbc, r, targets)
    ei, cs, _, counts = D.radius_graph_pbc_ex(pos_t, cell_t, pbc_t, r, 0, False, targets_t)
    np.testing.assert_array_equal(counts.cpu().numpy(), g["counts"])
    assert_same_edges(canon_t(ei, cs), canon_o(g), f"{n} atoms")
