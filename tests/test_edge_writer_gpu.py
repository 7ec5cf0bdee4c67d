"""The edge writer's forms: groups whose candidates have one shift code or several, more edges at a time than its buffer holds,
outputs at any address of their types, against the oracle."""

import numpy as np
import pytest
import torch

import dynamis_b200 as D
from _util import assert_same_edges, canon_o, canon_t
from dynamis_b200 import _lib
from dynamis_b200 import graph as G
from oracle import cpu_oracle as O

pytestmark = pytest.mark.gpu


def _system(kind, dtype):
    rng = np.random.default_rng(17)
    if kind == "dense":        # 449 neighbours each: the edges of four targets fill the buffer several times
        pos, length, pbc, r = rng.random((450, 3)) * 0.5, 40.0, [False] * 3, 1.0
    elif kind == "dense_codes":
        pos, length, pbc, r = rng.random((450, 3)) * 0.5, 40.0, [True] * 3, 1.0
        pos[::2] += 3.0 * length
    else:
        n = 3001
        length, pbc, r = (n / 0.1) ** (1.0 / 3.0), [True] * 3, 5.0
        pos = rng.random((n, 3)) * length
        if kind == "unwrapped":    # cells apart: shift codes differ from atom to atom
            pos += rng.integers(-3, 4, (n, 3)) * length
        elif kind == "moved":      # all atoms three cells away: one code, which is not that of a shift of zero
            pos += 3.0 * length
        elif kind == "halves":     # the edges of four targets often exceed the buffer, those of two never do
            r = 6.1
        elif kind == "few_long":   # some groups have lists without hit bits: warps share their targets
            pos[:700] = pos[0] + rng.random((700, 3)) * 2.5
        elif kind == "columns":    # few targets a row
            pos[:, 1:] *= 0.3
            r = 2.0
    return pos.astype(dtype), (np.eye(3) * length).astype(dtype), pbc, r


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("kind", ["dense", "dense_codes", "wrapped", "unwrapped", "moved", "columns", "halves", "few_long"])
def test_edges(cuda, kind, dtype):
    pos, cell, pbc, r = _system(kind, dtype)
    g = O.radius_graph(pos, cell, pbc, r, None)
    tp, tc, tb = torch.as_tensor(pos, device=cuda), torch.as_tensor(cell), torch.tensor(pbc)
    ei, cs, nni, counts = D.radius_graph_pbc_ex(tp, tc, tb, r, 0, False)
    assert_same_edges(canon_t(ei, cs), canon_o(g), kind)
    assert int(nni) == g["E"]
    # the targets' runs: as long as the degrees say, each target once
    runs = ei[1][torch.cat([torch.ones(1, dtype=torch.bool, device=cuda), ei[1][1:] != ei[1][:-1]])]
    assert runs.numel() == int((counts > 0).sum()) == runs.unique().numel()
    # the model-side form: the opposite sign and the Cartesian shift
    e2, unit, cart = D.owned_graph(tp, tc, tb, r, pos.shape[0])
    assert torch.equal(e2, ei) and torch.equal(unit, -cs) and torch.equal(cart, torch.matmul(unit, tc.to(cuda, torch.float32)))


@pytest.mark.parametrize("kind", ["wrapped", "unwrapped"])
@pytest.mark.parametrize("offset", [0, 1, 2, 3])
def test_outputs_at_any_address(cuda, kind, offset):
    pos, cell, pbc, r = _system(kind, np.float32)
    plan = G.plan_radius_graph(torch.as_tensor(pos, device=cuda), torch.as_tensor(cell), torch.tensor(pbc), r)
    ei, cs, _ = plan.fill()
    E = plan.E
    a = torch.full((2 * E + 8,), -7, dtype=torch.int64, device=cuda)
    b = torch.full((3 * E + 16,), -7.0, device=cuda)
    fo = 2 * offset + 1
    _lib.check(_lib.lib().dynb_rg_fill(plan.ws.data_ptr(), plan.dtype_code, a.data_ptr() + 8 * offset, b.data_ptr() + 4 * fo, None, E,
                                       torch.cuda.current_stream().cuda_stream), "rg_fill")
    assert torch.equal(a[offset:offset + 2 * E].view(2, E), ei) and torch.equal(b[fo:fo + 3 * E].view(E, 3), cs)
    assert (a[:offset] == -7).all() and (a[offset + 2 * E:] == -7).all() and (b[:fo] == -7).all() and (b[fo + 3 * E:] == -7).all()


def test_negative_zero_shifts(cuda):
    """A column of the cell that is all negative makes the Cartesian shift of a zero shift a negative zero."""
    cell = torch.tensor([[-30.0, -1.0, -2.0], [-3.0, -28.0, -1.0], [-1.0, -2.0, -33.0]])
    frac = torch.rand(2000, 3, generator=torch.Generator().manual_seed(4))
    pos = (frac @ cell).to(cuda)
    _, unit, cart = D.owned_graph(pos, cell, torch.tensor([True] * 3), 4.0, 2000)
    still = (unit == 0).all(dim=1)
    assert still.any() and torch.signbit(cart[still]).all()
