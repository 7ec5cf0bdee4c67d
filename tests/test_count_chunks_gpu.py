"""The count pass tests a chunk of a list with the smallest copy of its loop that holds it, with both tests everywhere where the records of
the targets' own cell rows lie in more than two blocks of 64 or in a list of several chunks: lists of one chunk whose records all lie in the
own rows (a thread of atoms), and last chunks at the edges of the copies, against the oracle."""

import numpy as np
import pytest
import torch

import dynamis_b200 as D
from _util import assert_same_edges, canon_o, canon_t
from oracle import cpu_oracle as O

pytestmark = pytest.mark.gpu


def check(cuda, pos, r, what):
    cell, pbc = (np.eye(3) * 50.0).astype(pos.dtype), [False] * 3
    g = O.radius_graph(pos, cell, pbc, r, None)
    ei, cs, _, counts = D.radius_graph_pbc_ex(torch.as_tensor(pos, device=cuda), torch.as_tensor(cell), torch.tensor(pbc), r, 0, False)
    np.testing.assert_array_equal(counts.cpu().numpy(), g["counts"])
    assert_same_edges(canon_t(ei, cs), canon_o(g), what)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [128, 129, 191, 193, 256, 257, 320, 321, 385, 449, 511, 512])
def test_all_records_in_the_own_row(cuda, n, dtype):
    rng = np.random.default_rng(n)
    pos = rng.random((n, 3)) * [0.6, 0.01, 0.01]
    pos[: n // 8] = pos[n // 8: 2 * (n // 8)]
    check(cuda, pos.astype(dtype), 0.45, f"{n} candidates")


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("tail", [64, 65, 128, 129, 192, 256, 257, 320, 321, 448, 449])
def test_last_chunk(cuda, tail, dtype):
    rng = np.random.default_rng(tail)
    check(cuda, (rng.random((512 + tail, 3)) * 0.6).astype(dtype), 0.45, f"512 + {tail} candidates")
