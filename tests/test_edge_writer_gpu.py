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
    runs, lengths = torch.unique_consecutive(ei[1], return_counts=True)
    assert runs.numel() == int((counts > 0).sum()) == runs.unique().numel()
    assert torch.equal(lengths, counts[runs].to(torch.int64))
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


class _Plan:
    """What a plan leaves in its workspace, read on the host: the grid, the records in the order of the cells, the hit bits."""

    POINTERS = ["h", "cstart", "tcstart", "spos", "sscan", "tpos", "tscan", "tmeta", "tcount", "toffset", "hitmask", "smeta"]

    def __init__(self, plan, n):
        base = plan.ws.data_ptr()
        raw = plan.ws.cpu().numpy()
        start = -base % 256
        at = {k: int(v) - base for k, v in zip(self.POINTERS, raw[start + 512:start + 512 + 8 * len(self.POINTERS)].view(np.uint64))}
        assert at["h"] == start

        def view(name, dtype, count):
            return raw[at[name]:at[name] + count * np.dtype(dtype).itemsize].view(dtype)

        self.nx, self.ny, self.nz, self.sx = (int(v) for v in raw[start + 24:start + 40].view(np.int32))
        self.pad, self.gx, self.sy = (int(v) for v in raw[start + 68:start + 80].view(np.int32))
        assert (self.nx, self.ny, self.nz) == plan.grid
        cells = self.nx * self.ny * self.nz
        self.cstart, self.tcstart = view("cstart", np.uint32, cells + 1).astype(int), view("tcstart", np.uint32, cells + 1).astype(int)
        self.smeta = view("smeta", np.uint32, 2 * plan.M).reshape(-1, 2).astype(int)
        self.tmeta = view("tmeta", np.int32, 4 * n).reshape(-1, 4).astype(int)
        self.toffset = view("toffset", np.int64, n + 1)
        self.hitmask = view("hitmask", np.uint16, 32 * n).reshape(-1, 32)

    def groups(self):
        """(targets, records of the candidate list) of every group with targets."""
        for cz in range(self.nz):
            for cy0 in range(0, self.ny, self.sy):
                cy1 = min(cy0 + self.sy, self.ny) - 1
                for cx0 in range(0, self.nx, self.sx):
                    cx1 = min(cx0 + self.sx, self.nx) - 1
                    targets = [t for cy in range(cy0, cy1 + 1)
                               for t in range(self.tcstart[(cz * self.ny + cy) * self.nx + cx0], self.tcstart[(cz * self.ny + cy) * self.nx + cx1 + 1])]
                    if not targets:
                        continue
                    records = []
                    for zz in range(max(cz - self.pad, 0), min(cz + self.pad, self.nz - 1) + 1):
                        for yy in range(max(cy0 - self.pad, 0), min(cy1 + self.pad, self.ny - 1) + 1):
                            row = (zz * self.ny + yy) * self.nx
                            records += range(self.cstart[row + max(cx0 - self.pad, 0)], self.cstart[row + min(cx1 + self.pad, self.nx - 1) + 1])
                    yield targets, np.array(records, dtype=int)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("kind", ["dense", "dense_codes", "wrapped", "unwrapped", "halves", "columns", "few_long"])
def test_order_of_the_edges(cuda, kind, dtype):
    """The order is part of the result.  Targets follow one another cell by cell.  The edges of a target come by (place mod 32,
    place / 32) of their candidates in the group's list where it has at most 512 places, and by place in longer lists and
    wherever distances are asked for."""
    pos, cell, pbc, r = _system(kind, dtype)
    n = len(pos)
    plan = G.plan_radius_graph(torch.as_tensor(pos, device=cuda), torch.as_tensor(cell), torch.tensor(pbc), r)
    p = _Plan(plan, n)
    edges = {d: [a.cpu().numpy() for a in plan.fill(d)[:2]] for d in (False, True)}
    degrees, lists = plan.counts.cpu().numpy(), set()
    assert plan.E == p.toffset[-1] == degrees.sum()
    seen = 0
    for targets, records in p.groups():
        short = len(records) <= 512
        lists.add(short)
        codes = p.smeta[records, 1]
        atoms, moved = p.smeta[records, 0], np.stack([(codes >> k & 1023) - 512 for k in (0, 10, 20)], axis=1)
        for t in targets:
            seen += 1
            at = slice(int(p.toffset[t]), int(p.toffset[t + 1]))
            atom, shifts = p.tmeta[t, 0], moved + p.tmeta[t, 1:]
            assert at.stop - at.start == degrees[atom]
            place_of = {(a, *s): k for k, (a, s) in enumerate(zip(atoms.tolist(), shifts.tolist()))}
            assert len(place_of) == len(records)
            for dist, (ei, cs) in edges.items():
                places = [place_of[(a, *s)] for a, s in zip(ei[0, at].tolist(), cs[at].astype(int).tolist())]
                assert (ei[1, at] == atom).all()
                if short and not dist:
                    bits = p.hitmask[t][:, None] >> np.arange(16) & 1
                    assert places == [32 * s + lane for lane, s in zip(*np.nonzero(bits))]
                else:
                    assert places == sorted(set(places)), "by place"
    assert seen == n
    assert True in lists and (kind != "few_long" or False in lists)


# boxes a few cells wide along two axes or one, so that a row or a column of groups is one, two, three, 63 to 65 or hundreds long
@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("length,other", [(L, 8.0) for L in (8.0, 12.0, 16.0, 25.0, *np.arange(240.0, 268.0, 4.0), *np.arange(480.0, 528.0, 4.0), 2500.0)] + [(260.0, 260.0)])
def test_look_up_of_a_group_in_thin_boxes(cuda, length, other, axis, periodic):
    """The kernels divide a group's number by the lengths of the rows and of the columns of groups."""
    box = np.array([length, other, 8.0] if axis == 0 else [other, length, 8.0])
    pos = (np.random.default_rng(int(length)).random((int(0.04 * box.prod()) + 2, 3)) * box).astype(np.float32)
    cell, pbc = np.diag(box).astype(np.float32), [periodic] * 3
    g = O.radius_graph(pos, cell, pbc, 4.0, None)
    ei, cs, nni, counts = D.radius_graph_pbc_ex(torch.as_tensor(pos, device=cuda), torch.as_tensor(cell), torch.tensor(pbc), 4.0, 0, False)
    np.testing.assert_array_equal(counts.cpu().numpy(), g["counts"])
    assert_same_edges(canon_t(ei, cs), canon_o(g), f"{box}")
