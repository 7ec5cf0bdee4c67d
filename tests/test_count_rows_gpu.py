"""The count pass looks for records within the self-distance limit in the targets' own cell rows only: pairs on both sides of that limit,
across the faces of cells, in dense clusters; degrees and edges against the oracle.  Cells of 0.015: one pair in fifty lies across a face."""

import numpy as np
import pytest
import torch

import dynamis_b200 as D
from _util import assert_same_edges, canon_o, canon_t
from oracle import cpu_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("subset", [False, True])
@pytest.mark.parametrize("n, box", [(3000, 0.25), (9000, 0.25), (14000, 0.2)])
def test_pairs_at_the_limit(cuda, n, box, subset, dtype):
    rng = np.random.default_rng(n)
    pos = rng.random((n, 3)) * box
    step = rng.normal(size=(n // 2, 3))
    pos[n // 2:2 * (n // 2)] = pos[:n // 2] + step / np.linalg.norm(step, axis=1, keepdims=True) * 1e-4 * rng.choice([0.0, 0.9, 0.999, 1.001, 1.1], (n // 2, 1))
    pos = (pos + 0.1).astype(dtype)
    cell, pbc, r = (np.eye(3) * 0.5).astype(dtype), [True] * 3, 0.03
    targets = rng.permutation(n)[: n // 3] if subset else None
    g = O.radius_graph(pos, cell, pbc, r, targets)
    ei, cs, _, counts = D.radius_graph_pbc_ex(torch.as_tensor(pos, device=cuda), torch.as_tensor(cell), torch.tensor(pbc), r, 0, False,
                                              torch.as_tensor(targets, device=cuda) if subset else None)
    np.testing.assert_array_equal(counts.cpu().numpy(), g["counts"])
    assert_same_edges(canon_t(ei, cs), canon_o(g), f"{n} atoms")
