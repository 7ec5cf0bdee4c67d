"""The host buffers of the calls that wait for a count, whatever the modes and threads around them.  The wait lets go of the
interpreter: another thread may make a call on the same stream before the waiting one reads its count.  And the header of a binning
pass, which outlives a graph call."""

import threading

import numpy as np
import pytest
import torch

import dynamis_b200 as D
from dynamis_b200 import graph as G
from dynamis_b200.graph import BinnedAtoms
from dynamis_b200.partition import select_eq

pytestmark = pytest.mark.gpu


@pytest.fixture
def fresh_state(monkeypatch):
    """No buffers left by earlier calls."""
    monkeypatch.setattr(G, "_STATE", {})
    monkeypatch.setattr(G, "_HOST_WORDS", [])


class _Wait:
    """A stream behind whose first wait another thread makes a call on the same stream, before the waiting one goes on."""

    def __init__(self, stream, pending):
        self.stream, self.pending = stream, pending

    def __getattr__(self, name):
        return getattr(self.stream, name)

    def synchronize(self):
        self.stream.synchronize()
        if self.pending:
            t = threading.Thread(target=self.pending.pop())
            t.start()
            t.join()


@pytest.fixture
def behind_the_wait(monkeypatch):
    """behind_the_wait(call): ``call`` runs in another thread right behind the next wait of this one."""
    pending, me, real = [], threading.get_ident(), torch.cuda.current_stream
    monkeypatch.setattr(torch.cuda, "current_stream", lambda dev=None: _Wait(real(dev), pending) if threading.get_ident() == me else real(dev))
    yield pending.append
    assert not pending, "the call did not wait"


def _halo_edges(dev):
    """Edges of a ring of 600 atoms on two ranks, as rank 0 sees them: (edges, owners, its atoms)."""
    at = torch.arange(600, device=dev)
    owner = (at >= 300).to(torch.int64)
    mine = at[:300].contiguous()
    return torch.cat([torch.stack([(mine + s) % 600, mine]) for s in (1, -1)], dim=1).contiguous(), owner, mine


def _check_halo(dev):
    edges, owner, mine = _halo_edges(dev)
    send_offsets, send_local, recv_offsets, _, interior, recv_atom = D.extract_halo_info(edges, owner, mine, 0, 2, 600)
    assert send_offsets.tolist() == [0, 0, 2] and recv_offsets.tolist() == [0, 0, 2]
    assert send_local.tolist() == [0, 299] and recv_atom.tolist() == [300, 599] and int(interior.sum()) == 298


def test_counts_under_another_default_device(cuda, fresh_state):
    """The pinned words are the host's whatever device new tensors go to."""
    values = (torch.arange(5000, device=cuda) % 7).to(torch.int64)
    with torch.device(cuda):
        assert torch.equal(select_eq(values, 3), torch.nonzero(values == 3).reshape(-1))
        _check_halo(cuda)


def test_counts_first_read_in_inference_mode(cuda, fresh_state):
    """What the first call leaves for later ones can be written outside the mode it was made in."""
    with torch.inference_mode():
        _check_halo(cuda)
    _check_halo(cuda)
    with torch.inference_mode():
        _check_halo(cuda)


def test_count_of_a_selection(cuda, behind_the_wait):
    values = (torch.arange(5000, device=cuda) % 7).to(torch.int64)
    others = torch.ones(3000, dtype=torch.int64, device=cuda)
    got = []
    behind_the_wait(lambda: got.append(select_eq(others, 1)))
    mine = select_eq(values, 3)
    assert torch.equal(mine, torch.nonzero(values == 3).reshape(-1))
    assert torch.equal(got[0], torch.arange(3000, device=cuda))


def test_count_of_filtered_edges(cuda, behind_the_wait):
    pos = torch.zeros((400, 3), device=cuda)
    pos[:, 0] = torch.arange(400, device=cuda)
    src = torch.arange(399, device=cuda)
    edges = torch.cat([torch.stack([src, src + 1]), torch.stack([src[:-1], src[:-1] + 2])], dim=1).contiguous()
    shifts = torch.zeros((edges.size(1), 3), device=cuda)
    others = torch.ones(900, dtype=torch.int64, device=cuda)
    behind_the_wait(lambda: select_eq(others, 1))
    kept, kept_shifts = D.filter_edges_to_radius(edges, shifts, pos, torch.eye(3) * 500.0, 1.5)
    assert torch.equal(kept, edges[:, :399]) and kept_shifts.shape == (399, 3)


def test_sizes_of_halo_lists(cuda, behind_the_wait):
    others = torch.ones(900, dtype=torch.int64, device=cuda)
    behind_the_wait(lambda: [select_eq(others, 1) for _ in range(3)])
    _check_halo(cuda)


def test_words_are_one_calls_and_bounded(cuda, fresh_state):
    held = [G.take_host_words(n) for n in [1, G.HOST_WORDS, G.HOST_WORDS + 1] + [2] * (G.HOST_WORDS_KEPT + 3)]
    assert len({w.data_ptr() for w in held}) == len(held) and all(w.is_pinned() for w in held)
    assert held[2].numel() == G.HOST_WORDS + 1
    for w in held:
        G.give_host_words(w)
    assert len(G._HOST_WORDS) == G.HOST_WORDS_KEPT and all(w.numel() == G.HOST_WORDS for w in G._HOST_WORDS)
    assert G.take_host_words(3).data_ptr() in {w.data_ptr() for w in held}


@pytest.mark.parametrize("periodic", [True, False])
def test_header_of_a_binning_pass(cuda, periodic):
    """The status of a pass whose image capacity was too small outlives a graph call made before it is looked at."""
    rng = np.random.default_rng(8)
    pos = torch.as_tensor((rng.random((4000, 3)) * 30.0).astype(np.float32), device=cuda)
    cell, pbc = torch.eye(3) * 30.0, torch.tensor([True, True, periodic])
    bins = BinnedAtoms(pos, cell, pbc, 5.0)
    bins.src_capacity = 1000   # fewer slots than atoms: reported, nothing is written behind them
    bins.launch()
    D.radius_graph_pbc_ex(pos[:500].contiguous(), cell, pbc, 4.0, 0, False)
    torch.cuda.synchronize()
    assert bins.done() is False and bins.src_capacity > 4000
    bins.launch()
    torch.cuda.synchronize()
    assert bins.done() is True and int(bins.hdr.M) >= 4000
