"""Targets that the count pass tests in full: those at the faces of their cell rows (a plane of atoms at the end of an open direction: all of
them), those with an undecided distance (an ideal crystal in double precision, the cutoff on a shell of neighbours: all of them)
and those of coordinates beyond the range of the float test."""

import numpy as np
import pytest
import torch

import dynamis_b200 as D
from _util import assert_same_edges, canon_o, canon_t
from oracle import cpu_oracle as O

pytestmark = pytest.mark.gpu

FCC = np.array([[0.0, 0.0, 0.0], [0.5, 0.5, 0.0], [0.5, 0.0, 0.5], [0.0, 0.5, 0.5]])
A = 3.615


def lattice(cells):
    corner = np.stack(np.meshgrid(*[np.arange(float(cells))] * 3, indexing="ij"), -1).reshape(-1, 1, 3)
    return (corner + FCC).reshape(-1, 3) * A, np.eye(3) * cells * A


def crystal():
    pos, cell = lattice(9)
    return pos, cell, [True] * 3, A * 1.5 ** 0.5


def mixed():
    """One half of the crystal out of place: whole batches of both kinds, and batches of some of each."""
    pos, cell = lattice(9)
    rng = np.random.default_rng(1)
    off = (pos[:, 0] > 4.5 * A) | (rng.random(len(pos)) < 0.3)
    return pos + off[:, None] * rng.normal(size=pos.shape) * 0.05, cell, [True] * 3, A * 1.5 ** 0.5


def plane():
    x, y = np.meshgrid(np.arange(45) * 1.2, np.arange(45) * 1.2, indexing="ij")
    return np.stack([x.ravel(), y.ravel(), np.full(x.size, 7.0)], 1), np.diag([54.0, 54.0, 20.0]), [True, True, False], 6.0


def far():
    rng = np.random.default_rng(2)
    pos = rng.integers(0, 16, (900, 3)) * 0.5
    pos[::2] += 3.0e15
    return pos, np.eye(3) * 1.0e17, [False] * 3, 4.0


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("system", [crystal, mixed, plane, far])
def test_degrees_and_edges(cuda, system, dtype):
    pos, cell, pbc, r = system()
    pos, cell = pos.astype(dtype), cell.astype(dtype)
    g = O.radius_graph(pos, cell, pbc, r, None)
    ei, cs, _, counts = D.radius_graph_pbc_ex(torch.as_tensor(pos, device=cuda), torch.as_tensor(cell), torch.tensor(pbc), r, 0, False)
    np.testing.assert_array_equal(counts.cpu().numpy(), g["counts"])
    assert_same_edges(canon_t(ei, cs), canon_o(g), system.__name__)


def test_time_of_a_crystal_with_the_cutoff_on_a_shell(cuda):
    """Both tests for every place are at most twice the work of the count pass, which is half of the call, and a few places of a list go
    through the double test: a call takes less than twice as long as with the cutoff off the shell (3.4 times when every place went
    through the double test)."""
    pos, cell = (torch.as_tensor(x) for x in lattice(50))
    pos, pbc = pos.to(cuda), torch.tensor([True] * 3)
    best = {}
    for _ in range(6):
        for r in (A * 1.5 ** 0.5, A * 1.5 ** 0.5 + 0.02):
            D.radius_graph_pbc_counts_ex(pos, cell, pbc, r)
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            start.record()
            for _ in range(5):
                D.radius_graph_pbc_counts_ex(pos, cell, pbc, r)
            end.record()
            torch.cuda.synchronize()
            best[r] = min(best.get(r, float("inf")), start.elapsed_time(end))
    on, off = best[A * 1.5 ** 0.5], best[A * 1.5 ** 0.5 + 0.02]
    assert on < 2.0 * off, f"{on / 5 * 1e3:.0f} us on the shell, {off / 5 * 1e3:.0f} us off it"
