"""The host buffers of the calls that wait for a count, whatever the modes and threads around them."""

import pytest
import torch

import dynamis_b200 as D
from dynamis_b200 import graph as G
from dynamis_b200.partition import select_eq

pytestmark = pytest.mark.gpu


@pytest.fixture
def fresh_state(monkeypatch):
    """No buffers left by earlier calls."""
    monkeypatch.setattr(G, "_STATE", {})


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
