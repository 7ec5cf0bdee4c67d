"""The count pass keeps the candidates of a group in registers, 64 to a block, with copies of its loop for 2, 4, 5, 6, 7 and 8 blocks:
candidate lists whose lengths lie at the edges of the blocks and of the 512 places that have hit bits, against the oracle."""

import numpy as np
import pytest
import torch

import dynamis_b200 as D
from _util import assert_same_edges, canon_o, canon_t
from oracle import cpu_oracle as O

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 31, 32, 33, 63, 64, 65, 127, 128, 129, 191, 192, 193, 255, 256, 257, 319, 320, 321, 384, 385, 448, 449, 511, 512, 513, 1024, 1025]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", LENGTHS)
def test_list_lengths(cuda, n, dtype):
    """All atoms in one neighbourhood of a box without periodic directions: every list has n candidates.  Some atoms coincide,
    and some lie within and just beyond the self-distance limit of 1e-4 of one another."""
    rng = np.random.default_rng(n)
    pos = rng.random((n, 3)) * 0.6
    k = n // 8
    if k:
        pos[:k] = pos[k:2 * k]
        step = rng.normal(size=(k, 3))
        pos[2 * k:3 * k] = pos[3 * k:4 * k] + step / np.linalg.norm(step, axis=1, keepdims=True) * 1e-4 * rng.choice([0.9, 1.1], (k, 1))
    pos = pos.astype(dtype)
    cell, pbc, r = (np.eye(3) * 50.0).astype(dtype), [False] * 3, 0.45
    g = O.radius_graph(pos, cell, pbc, r, None)
    ei, cs, nni, counts = D.radius_graph_pbc_ex(torch.as_tensor(pos, device=cuda), torch.as_tensor(cell), torch.tensor(pbc), r, 0, False)
    np.testing.assert_array_equal(counts.cpu().numpy(), g["counts"])
    assert int(nni) == g["E"] or g["E"] == 0
    assert_same_edges(canon_t(ei, cs), canon_o(g), f"{n} candidates")


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_radius_below_the_self_distance_limit(cuda, dtype):
    rng = np.random.default_rng(3)
    pos = (rng.random((200, 3)) * 2e-4).astype(dtype)
    for r in (5e-5, 1e-4, 2e-4):
        g = O.radius_graph(pos, (np.eye(3) * 9.0).astype(dtype), [False] * 3, r, None)
        counts = D.radius_graph_pbc_counts_ex(torch.as_tensor(pos, device=cuda), torch.eye(3, dtype=torch.as_tensor(pos).dtype) * 9.0,
                                              torch.tensor([False] * 3), r)
        np.testing.assert_array_equal(counts.cpu().numpy(), g["counts"])
